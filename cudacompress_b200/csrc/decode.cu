// decode.cu - device entropy decoder: decodeRLHuff / decodeHuff
// (Encode.cpp:473-646, :792-917; Huffman.cu:189-279; HuffmanTable.cu:117-266;
// RunLength.cu:257-328).
//
// One call decodes a batch of streams of any sizes and of both kinds.  Two
// front ends fill the same descriptors:
//  * cc_decode (the reference's decode entry points, caller's host bit
//    streams): the host walks the stream headers - the reference's own
//    decode parses them on the host too and returns before the GPU work is
//    done - and stages the touched words once;
//  * decodePrepare / decodeLaunch (batched volume codec, device-resident bit
//    streams): one warp per bit stream walks its headers on the device, so
//    nothing goes through the host and the launches can be replayed.
// Back end, one launch per stage over the whole batch (coding blocks are
// numbered across the streams of a kind and found back by binary search):
//   symPlan -> tables -> huffman (Huff) | zero counts -> run scan -> symbols
// Every read of the bit stream is bounds-checked, and malformed tables or
// codes raise CC_ERR_CORRUPT_STREAM instead of reading or writing out of
// bounds.
#include <algorithm>
#include <cstring>

#include "capi_internal.cuh"

namespace ccb {

struct DecParams {
    u32 S, T, nSrc, nRl, nH;
    u32 rlBlocks, hBlocks;     // coding blocks (upper bounds) of the RLHuff / Huff streams
    u32 rlMaxN, maxN;          // largest output of an RLHuff stream, and of any
    u32 cb, cbLog, log2Max, symBytes, leavesMax;   // cb = 2^cbLog
    u64 capLeaves;
    DecStreamDesc* streams;
    DecTableDesc* tables;
    DecSource* sources;
    const u32* rlList;         // RLHuff stream indices (by blockFirst)
    const u32* hList;          // Huff stream indices (by blockFirst)
    const u32* wordsBase;      // indirect sources (device walk): base + wordOff[k], bitSize[k]
    const u64* wordOff;
    const u64* bitSize;
    DecTable* dec;
    u32* syms;                 // [capLeaves]
    u32* lut;                  // [T][1 << kLutBits]
    u32* blockOff;             // coding-block bit offsets, by table blockOff
    u32* blockSum;             // RLHuff: per zero-count block output lengths
    u64* rlTasks;              // RLHuff decode warp tasks (stream << 32 | first block); count at rlTasks[rlTaskCap]
    u32 rlTaskCap;
    char* zc;                  // decoded zero counts, by stream zcOff
    u64* planPart;             // sums of each chunk of the symbol plan (k_decSymPlan)
    u32* errors;
};

// Bounds-checked view of one bit stream's words.
struct WordSrc {
    const u32* w;
    u64 n;
    __device__ __forceinline__ u32 at(u64 i) const { return i < n ? w[i] : 0u; }
    __device__ __forceinline__ u32 bits(u64 bit, u32 count) const {
        if (count == 0) return 0;
        const u64 wi = bit >> 5;
        const u32 b = u32(bit & 31u);
        const u64 window = (u64(at(wi)) << 32) | at(wi + 1);
        return u32((window << b) >> (64 - count));
    }
};

__device__ __forceinline__ WordSrc srcOf(const DecParams& p, u32 stream) {
    const DecSource& s = p.sources[p.streams[stream].source];
    return WordSrc{s.words, s.wordCount};
}

__device__ __forceinline__ bool capacityFailed(const DecParams& p) {
    return (*reinterpret_cast<volatile const u32*>(p.errors) & DEV_ERR_TABLE_CAPACITY) != 0;
}

// Stream owning flattened block `b` of the RLHuff (or Huff) list.
__device__ __forceinline__ u32 streamOfBlock(const DecParams& p, const u32* list, u32 count, u32 b) {
    u32 lo = 0, hi = count;
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (p.streams[list[mid]].blockFirst <= b) lo = mid; else hi = mid;
    }
    return list[lo];
}

// ---------------------------------------------------------------------------
// Device walk (HuffmanTable.cu:117-151 header fields, Encode.cpp:473-646 /
// 792-917 stream layout, BitStream.h:290-308 alignment).
// ---------------------------------------------------------------------------
// A bit stream's reader: the walk is a chain of short reads, so the calling
// warp (every lane with the same values) reads through a window of 128 words
// in shared memory, loaded 16 bytes per lane wherever a read leaves it - one
// round trip per header for most tables, whose code lengths, symbols and code
// word count then come out of the window.  Word indices are 32-bit (a stream
// holds at most 2^31 symbols of 31 bits).  Three 256^3 streams (43 tables
// each): 37 us, against 56 with 64-bit positions and divisions by the coding
// block, and 81 for a thread per stream reading word by word.
constexpr u32 kWalkWindow = 128;

struct DevReader {
    const u32* aligned;   // the 16-byte aligned word at or below the stream's first
    u32 skew;             // words from it to the stream's first
    u32 end;              // one past the stream's last word, from `aligned`
    u64 size;             // readable bits
    u32* win;             // kWalkWindow words of shared memory
    u32 base;             // first word in it, from `aligned` (a multiple of 4)

    __device__ u32 word(u32 i) {
        const u32 a = i + skew;
        if (a >= end || a < skew) return 0u;
        if (a - base >= kWalkWindow) {   // also when the window lies behind (unsigned)
            base = a & ~3u;
            const u32 q = base + 4u * (threadIdx.x & 31u);   // this lane's four words, where they belong to the stream
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (q >= skew && q + 4 <= end) {
                v = *reinterpret_cast<const uint4*>(aligned + q);
            } else {
                if (q >= skew && q < end) v.x = aligned[q];
                if (q + 1 >= skew && q + 1 < end) v.y = aligned[q + 1];
                if (q + 2 >= skew && q + 2 < end) v.z = aligned[q + 2];
                if (q + 3 >= skew && q + 3 < end) v.w = aligned[q + 3];
            }
            __syncwarp();
            *reinterpret_cast<uint4*>(win + 4u * (threadIdx.x & 31u)) = v;
            __syncwarp();
        }
        return win[a - base];
    }
    // n <= 32 bits at bit `bit` after word w; false past the end
    __device__ bool bits(u32 w, u32 bit, u32 n, u32& v) {
        if (u64(w) * 32u + bit + n > size) return false;
        w += bit >> 5;
        bit &= 31u;
        const u32 hi = word(w), lo = bit + n > 32u ? word(w + 1) : 0u;
        v = __funnelshift_l(lo, hi, bit) >> (32u - n);
        return true;
    }
};

// Walks a table and its payload from bit `bit` of word w; w moves behind them.
__device__ bool walkTableDev(DevReader& r, u32& w, u32 bit, u32 count, u32 log2Max, u32 leavesMax, u32 cbLog,
                             DecTableDesc& d) {
    d.hdrBit = u64(w) * 32u + bit;
    if (!r.bits(w, bit, 5, d.nLen)) return false;
    bit += 5 + d.nLen * log2Max;
    if (!r.bits(w, bit, log2Max, d.nSym)) return false;
    bit += log2Max;
    const bool longSym = log2Max > 16;
    if (!r.bits(w, bit, longSym ? 5 : 4, d.symbolBits)) return false;
    bit += longSym ? 5 : 4;
    if (!longSym && d.symbolBits == 0 && d.nSym > 1) d.symbolBits = 16;   // HuffmanTable.cu:138-139
    if (d.nSym > leavesMax || d.nLen > 31) return false;
    const u64 symEnd = bit + u64(d.nSym) * d.symbolBits;
    w += u32((symEnd + 31) >> 5);
    if (!r.bits(w, 0, 32, d.cwBits)) return false;
    ++w;
    d.cwWord = w;
    w += (d.cwBits >> 5) + ((d.cwBits & 31u) ? 1u : 0u);
    d.offWord = w;
    w += (blocksOf(count, cbLog) + 1u) / 2u;
    d.count = count;
    return true;
}

// The walked fields of a table's descriptor (by one lane; blockOff and stream
// are the plan's).
__device__ __forceinline__ void storeWalked(DecTableDesc& to, const DecTableDesc& d) {
    to.hdrBit = d.hdrBit;
    to.cwWord = d.cwWord;
    to.offWord = d.offWord;
    to.cwBits = d.cwBits;
    to.count = d.count;
    to.symbolBits = d.symbolBits;
    to.nLen = d.nLen;
    to.nSym = d.nSym;
}

// A warp per source.
constexpr u32 kWalkWarps = 2;

__global__ void __launch_bounds__(kWalkWarps * 32) k_decWalk(DecParams p) {
    __shared__ __align__(16) u32 sWin[kWalkWarps][kWalkWindow];
    const u32 i = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    if (i >= p.nSrc) return;
    const bool first = (threadIdx.x & 31u) == 0;
    DecSource src = p.sources[i];
    if (p.wordOff) {
        const u64 bits = p.bitSize[i];
        src.words = p.wordsBase + p.wordOff[i];
        src.bitSize = bits;
        src.wordCount = ceilDiv(bits, 32);
    }
    const u64 wordBits = src.wordCount * 32ull;
    const u32 skew = u32(reinterpret_cast<uintptr_t>(src.words) & 15u) / 4u;
    DevReader r{src.words - skew, skew, u32(src.wordCount) + skew, src.bitSize < wordBits ? src.bitSize : wordBits,
                sWin[threadIdx.x >> 5], 0u - kWalkWindow};
    bool ok = src.wordCount < 0xFFFFFF00ull;
    u32 w = u32(src.startBit >> 5), bit = u32(src.startBit & 31u);
    u32 ns = 0, kinds = 0, firsts = 0;   // of this lane's stream of 32
    for (u32 k = 0; k < src.streamCount && ok; ++k) {
        if ((k & 31u) == 0) {
            const u32 q = k + (threadIdx.x & 31u);
            if (q < src.streamCount) {
                const DecStreamDesc& mine = p.streams[src.firstStream + q];
                ns = mine.n;
                kinds = mine.kind;
                firsts = mine.tableFirst;
            }
        }
        DecStreamDesc& sd = p.streams[src.firstStream + k];
        const u32 n = __shfl_sync(0xffffffffu, ns, int(k & 31u)), t0 = __shfl_sync(0xffffffffu, firsts, int(k & 31u));
        const u32 kind = __shfl_sync(0xffffffffu, kinds, int(k & 31u));
        DecTableDesc d0{}, d1{};
        if (kind == KIND_RLHUFF) {
            w += bit ? 1u : 0u;   // word aligned
            bit = 0;
            u32 m = 0;
            ok = r.bits(w, 0, 32, m) && m <= n;
            ++w;
            if (first) sd.m = ok ? m : 0u;
            ok = ok && walkTableDev(r, w, 0, m, p.log2Max, p.leavesMax, p.cbLog, d0) &&
                 walkTableDev(r, w, 0, m, p.log2Max, p.leavesMax, p.cbLog, d1);
            if (first) {
                storeWalked(p.tables[t0], d0);
                storeWalked(p.tables[t0 + 1], d1);
            }
        } else {
            ok = walkTableDev(r, w, bit, n, p.log2Max, p.leavesMax, p.cbLog, d0);
            bit = 0;
            if (first) {
                sd.m = n;
                storeWalked(p.tables[t0], d0);
            }
        }
    }
    if (!first) return;
    if (!ok) {
        atomicOr(p.errors, DEV_ERR_CORRUPT);
        // nothing of this source is decoded
        for (u32 k = 0; k < src.streamCount; ++k) {
            DecStreamDesc& sd = p.streams[src.firstStream + k];
            sd.m = 0;
            const u32 parts = sd.kind == KIND_RLHUFF ? 2u : 1u;
            for (u32 w = 0; w < parts; ++w) storeWalked(p.tables[sd.tableFirst + w], DecTableDesc{});
        }
    }
    src.endBit = min(u64(w) * 32u + bit, r.size);
    p.sources[i] = src;
}

// Symbol array offsets of the tables (prefix of nSym) and capacity check.
// CTA b takes the kPlanChunk tables of chunk b (four consecutive per thread):
// offsets within the chunk and the chunk's sum (planPart); with more than one
// chunk, k_decSymPlanCarry adds the chunks before each one.
__device__ __forceinline__ void symPlanChunk(const DecParams& p, u32 b, u32 chunks, u32* scratch) {
    constexpr u32 kPer = kPlanChunk / 1024;
    const u32 t0 = b * kPlanChunk + threadIdx.x * kPer;
    u32 v[kPer], sum = 0;
#pragma unroll
    for (u32 j = 0; j < kPer; ++j) {
        v[j] = t0 + j < p.T ? min(p.tables[t0 + j].nSym, p.leavesMax) : 0u;
        sum += v[j];
    }
    u32 tot;
    u32 at = blockExclusiveSum<1024>(sum, scratch, &tot);
#pragma unroll
    for (u32 j = 0; j < kPer; ++j) {
        if (t0 + j < p.T) p.tables[t0 + j].symOff = at;
        at += v[j];
    }
    if (threadIdx.x == 0) {
        if (chunks == 1) {
            if (tot > p.capLeaves) atomicOr(p.errors, DEV_ERR_TABLE_CAPACITY);
        } else {
            p.planPart[b] = tot;
        }
    }
}

__global__ void __launch_bounds__(1024) k_decSymPlan(DecParams p) {
    __shared__ u32 scratch[40];
    symPlanChunk(p, blockIdx.x, gridDim.x, scratch);
}

// Chunk b = blockIdx.x + 1 of a symbol plan of more than one chunk: the sum
// of chunks 0 .. b-1 added to its tables' offsets; the last chunk's CTA
// checks the capacity.
__global__ void __launch_bounds__(1024) k_decSymPlanCarry(DecParams p) {
    constexpr u32 kPer = kPlanChunk / 1024;
    __shared__ unsigned long long sC;
    const u32 b = blockIdx.x + 1;
    if (threadIdx.x < 32) {
        unsigned long long c = 0;
        for (u32 i = threadIdx.x; i < b; i += 32) c += p.planPart[i];
#pragma unroll
        for (u32 o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (threadIdx.x == 0) sC = c;
    }
    __syncthreads();
    const unsigned long long c = sC;
    const u32 t0 = b * kPlanChunk + threadIdx.x * kPer;
#pragma unroll
    for (u32 j = 0; j < kPer; ++j)
        if (t0 + j < p.T) p.tables[t0 + j].symOff += u32(c);
    if (b == gridDim.x && threadIdx.x == 0 && c + p.planPart[b] > p.capLeaves)
        atomicOr(p.errors, DEV_ERR_TABLE_CAPACITY);
}

// ---------------------------------------------------------------------------
// Table parse and decode structures (HuffmanTable.cu:117-151, :205-266).
// ---------------------------------------------------------------------------
// One CTA per table: 64 threads in calls of many tables (up to 32 tables per
// SM: the work per table is a short chain of dependent steps), 512 in calls of
// few, where the offsets of a long stream's blocks - 8 per thread and step -
// and the lookup table take the time (129 tables of 256^3 streams: 35 -> 18
// us): a table per SM, or as wideBlockScan has it.  120 tables of six blocks 7.7 us
// and 6.2 wide, 580 of them 7.9 and 11.9; 400 of 1024 blocks 8.4 and 8.3, of
// 2048 10.0 and 8.8.
constexpr u32 kDecThreads = 64, kDecThreadsWide = 512;

template <u32 kDecThreads>
__global__ void __launch_bounds__(kDecThreads) k_decTables(DecParams p) {
    __shared__ u32 cpl[32];
    __shared__ int sFirst[32], sMin[32], sMax[32];
    __shared__ u32 sLim[kLutBits + 1];
    __shared__ u32 sScan[40];
    __shared__ u32 sCarry, sFail, sUsable;   // sUsable: written once, before the barrier that publishes it
    const u32 t = blockIdx.x;
    if (threadIdx.x == 0) sFail = capacityFailed(p) ? 1u : 0u;
    __syncthreads();
    if (sFail) return;
    const DecTableDesc d = p.tables[t];
    const WordSrc ws = srcOf(p, d.stream);
    DecTable* D = p.dec + t;
    u32* syms = p.syms + d.symOff;
    u32* lut = p.lut + (u64(t) << kLutBits);
    const u64 cntBit = d.hdrBit + 5;
    if (threadIdx.x < 32) cpl[threadIdx.x] = threadIdx.x < d.nLen ? ws.bits(cntBit + u64(threadIdx.x) * p.log2Max, p.log2Max) : 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
        // canonical codes: codeword[i] = (codeword[i-1]+1) << (len_i - len_{i-1})
        u32 total = 0;
        bool ok = d.nLen <= 31 && d.nSym <= p.leavesMax;
        int code = 0, idx = 0;
        bool first = true;
        int prevLen = 0;
        for (u32 l = 1; l <= 31; ++l) {
            u32 c = cpl[l - 1];
            total += c;
            if (c) {
                if (first) { code = 0; first = false; }
                else code = (code + 1) << (int(l) - prevLen);
                sFirst[l - 1] = idx;
                sMin[l - 1] = code;
                code += int(c) - 1;
                sMax[l - 1] = code;
                idx += int(c);
                prevLen = int(l);
            } else {
                sFirst[l - 1] = sMin[l - 1] = sMax[l - 1] = -1;
            }
        }
        sFirst[31] = sMin[31] = sMax[31] = -1;
        // left-justified kLutBits-bit limits: a prefix e holds a code of
        // length l <= kLutBits iff sLim[l-1] <= e < sLim[l] (the canonical
        // codes of one length are consecutive, each length starting where
        // the previous one ends)
        sLim[0] = 0;
        for (u32 l = 1; l <= kLutBits; ++l)
            sLim[l] = sMax[l - 1] >= 0 ? u32(sMax[l - 1] + 1) << (kLutBits - l) : sLim[l - 1];
        if (d.nLen == 0) ok = ok && d.nSym <= 1;
        else ok = ok && total == d.nSym;
        if (!ok) atomicOr(p.errors, DEV_ERR_CORRUPT);
        sUsable = ok ? 1u : 0u;
        sCarry = 0;
    }
    __syncthreads();
    if (!sUsable) {
        if (threadIdx.x == 0) D->nSym = 0xFFFFFFFFu;   // marks the table unusable
        return;
    }
    const u64 symBit = cntBit + u64(d.nLen) * p.log2Max + p.log2Max + (p.log2Max > 16 ? 5u : 4u);
    for (u32 i = threadIdx.x; i < d.nSym; i += kDecThreads) {
        u32 v = ws.bits(symBit + u64(i) * d.symbolBits, d.symbolBits);
        syms[i] = p.symBytes == 2 ? (v & 0xFFFFu) : v;
    }
    // lookup table: first length l <= kLutBits whose prefix fits the canonical
    // range; the entry holds (l << 24) | the symbol's value for 16-bit
    // symbols, | its index otherwise
    const bool valueLut = p.symBytes == 2;
    if (valueLut) __syncthreads();   // syms[] of this table written above
    for (u32 e = threadIdx.x; e < (1u << kLutBits); e += kDecThreads) {
        u32 below = 0;   // lengths whose codes all lie below e
#pragma unroll
        for (u32 l = 1; l <= kLutBits; ++l) below += e >= sLim[l] ? 1u : 0u;
        const u32 l = below + 1;
        u32 entry = 0;
        if (l <= kLutBits) {
            const u32 idx = u32(sFirst[l - 1] + int(e >> (kLutBits - l)) - sMin[l - 1]);
            entry = (l << 24) | (valueLut ? syms[idx] : idx);
        }
        lut[e] = entry;
    }
    if (threadIdx.x < 32) {
        D->firstIndex[threadIdx.x] = sFirst[threadIdx.x];
        D->minCode[threadIdx.x] = sMin[threadIdx.x];
        D->maxCode[threadIdx.x] = sMax[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        D->nSym = d.nSym;
        const u32 v0 = d.nSym >= 1 ? ws.bits(symBit, d.symbolBits) : 0u;
        D->single = p.symBytes == 2 ? (v0 & 0xFFFFu) : v0;
    }
    // absolute block offsets: inclusive prefix of the u16 increments
    // (PackInc.cu:220-229), eight blocks (four words) per thread per step
    const u32 blocks = blocksOf(d.count, p.cbLog);
    u32* bo = p.blockOff + d.blockOff;
    __syncthreads();
    for (u32 base = 0; base < blocks; base += 8 * kDecThreads) {
        const u32 k0 = base + 8 * threadIdx.x;
        u32 inc[8], sum = 0;
#pragma unroll
        for (u32 j = 0; j < 4; ++j) {
            const u32 w = k0 + 2 * j < blocks ? ws.at(d.offWord + k0 / 2 + j) : 0u;
            inc[2 * j] = k0 + 2 * j < blocks ? (w & 0xFFFFu) : 0u;
            inc[2 * j + 1] = k0 + 2 * j + 1 < blocks ? (w >> 16) : 0u;
            sum += inc[2 * j] + inc[2 * j + 1];
        }
        u32 tot;
        const u32 ex = blockExclusiveSum<kDecThreads>(sum, sScan, &tot);
        u32 off = sCarry + ex;
#pragma unroll
        for (u32 j = 0; j < 8; ++j) {
            off += inc[j];
            if (k0 + j < blocks) {
                bo[k0 + j] = off;
                if (off > d.cwBits) atomicOr(p.errors, DEV_ERR_CORRUPT);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) sCarry += tot;
        __syncthreads();
    }
}

// One table's data for codes longer than the lookup table, in shared memory:
// last[l] = (maxCode[l] + 1 << (32 - l)) - 1, carried over lengths without
// codes, so a 32-bit window v holds a code longer than l iff v > last[l] (the
// canonical codes of one length are consecutive and each length starts where
// the shorter ones end, so last never decreases), for l from the shortest
// code's length on; off[l - 1]: first index - first code.
struct CanonSmem {
    u32 last[32];
    int off[32];
};
// The same for the lengths met in earnest, in registers: codes of more than
// kLutBits bits are `start` bits long or more; lengths kLutBits + 1 .. + 4 as
// in last[] (never exceeded below the shortest code, which start leaves out).
struct LongCodes {
    u32 start, l0, l1, l2, l3;
};

// Stages table t's long codes into cs (all 32 lanes of the calling warp; the
// caller synchronizes).
__device__ __forceinline__ LongCodes stageLongCodes(CanonSmem& cs, const DecParams& p, u32 t) {
    const u32 lane = threadIdx.x & 31u;
    const DecTable& D = p.dec[t];
    const int mc = D.maxCode[lane];
    cs.off[lane] = D.firstIndex[lane] - D.minCode[lane];
    // lane l holds length l + 1
    const u32 has = __ballot_sync(0xffffffffu, mc >= 0 && lane < 31u);
    const u32 upTo = has & (0xFFFFFFFFu >> (31u - lane));
    const u32 from = upTo ? 31u - u32(__clz(int(upTo))) : 0u;   // nearest length with codes
    u32 last = mc >= 0 && lane < 31u ? ((u32(mc) + 1u) << (31u - lane)) - 1u : 0xFFFFFFFFu;
    last = __shfl_sync(0xffffffffu, last, int(from));
    if (!upTo) last = 0xFFFFFFFFu;
    cs.last[lane] = last;
    LongCodes lc;
    const u32 shortest = has ? u32(__ffs(int(has))) : 32u;      // length of the shortest code
    lc.start = max(kLutBits + 1u, shortest);
    lc.l0 = __shfl_sync(0xffffffffu, last, int(kLutBits));
    lc.l1 = __shfl_sync(0xffffffffu, last, int(kLutBits + 1));
    lc.l2 = __shfl_sync(0xffffffffu, last, int(kLutBits + 2));
    lc.l3 = __shfl_sync(0xffffffffu, last, int(kLutBits + 3));
    return lc;
}
// Stages table t's lookup table, one of `threads` threads calling (the caller
// synchronizes).
__device__ __forceinline__ void stageLut(u32* lut, const DecParams& p, u32 t, u32 thread, u32 threads) {
    const uint4* g = reinterpret_cast<const uint4*>(p.lut + (u64(t) << kLutBits));
    for (u32 k = thread; k < (1u << kLutBits) / 4u; k += threads) reinterpret_cast<uint4*>(lut)[k] = g[k];
}

// Length and symbol index of a window holding a code longer than the lookup
// table; false past the longest.
__device__ __forceinline__ bool longCode(u32 v, const LongCodes& lc, const CanonSmem& cs, u32 nSym, u32& len,
                                         u32& idx) {
    len = lc.start + (v > lc.l0 ? 1u : 0u) + (v > lc.l1 ? 1u : 0u) + (v > lc.l2 ? 1u : 0u) + (v > lc.l3 ? 1u : 0u);
    if (len > kLutBits + 4u)
        while (len <= 31u && v > cs.last[len - 1]) ++len;
    if (len > 31u) return false;
    idx = (v >> (32u - len)) + u32(cs.off[len - 1]);
    return idx < nSym;
}

// The code words of a warp's coding blocks, which are consecutive: staged in
// shared memory by coalesced loads when they fit, else read where they are.  A
// lane that fetches its words from global memory as it goes waits for a cache
// miss, or for 31 other lanes' lines, about every other symbol.
struct StagedWords {   // s[n] = 0
    const u32* s;
    u32 n;
    __device__ __forceinline__ u32 at(u32 i) const { return s[min(i, n)]; }
};
struct SourceWords {
    WordSrc ws;
    u64 first;
    __device__ __forceinline__ u32 at(u32 i) const { return ws.at(first + i); }
};

// Copies words [first, first + n) of ws to stage (all lanes of the warp).
__device__ __forceinline__ void stageWords(u32* stage, const WordSrc& ws, u64 first, u32 n) {
    for (u32 base = 0; base < n; base += 256) {
        u32 v[8];
#pragma unroll
        for (u32 k = 0; k < 8; ++k) {
            const u32 i = base + 32 * k + (threadIdx.x & 31u);
            v[k] = i < n ? ws.at(first + i) : 0u;
        }
#pragma unroll
        for (u32 k = 0; k < 8; ++k) {
            const u32 i = base + 32 * k + (threadIdx.x & 31u);
            if (i < n) stage[i] = v[k];
        }
    }
    if ((threadIdx.x & 31u) == 0) stage[n] = 0;
}

// A lane's place in its words: two words in hand and the next on its way, so
// that a step waits for the lookup only.
struct BitReader {
    u32 w;          // index of the word after nx
    u32 bpos;       // bit position in hi
    u32 hi, lo, nx;
    template <class Words>
    __device__ __forceinline__ void start(const Words& ws, u32 bit) {
        w = bit >> 5;
        bpos = bit & 31u;
        hi = ws.at(w);
        lo = ws.at(w + 1);
        nx = ws.at(w + 2);
        w += 3;
    }
};

// One symbol from r: a lookup, or for a code longer than the lookup table its
// length from the limits.  A window that holds no code sets corrupt and moves
// on by a bit.  kValueLut: lookup entries hold symbol values (16-bit symbols),
// else symbol indices.
template <bool kValueLut, class Words>
__device__ __forceinline__ u32 decodeOne(const Words& ws, const u32* lut, const CanonSmem& cs, const LongCodes& lc,
                                         u32 nSym, const u32* syms, BitReader& r, bool& corrupt) {
    const u32 v = __funnelshift_l(r.lo, r.hi, r.bpos);
    const u32 e = lut[v >> (32 - kLutBits)];
    u32 len = e >> 24, val = e & 0xFFFFFFu;
    if (kValueLut) {
        if (!e) {
            u32 idx;
            if (longCode(v, lc, cs, nSym, len, idx)) val = syms[idx];
            else { corrupt = true; len = 1; }
        }
    } else {
        bool ok = val < nSym;
        if (!e) ok = longCode(v, lc, cs, nSym, len, val);
        if (ok) val = syms[val];
        else { corrupt = true; len = 1; }
    }
    r.bpos += len;
    const bool next = r.bpos >= 32u;
    r.hi = next ? r.lo : r.hi;
    r.lo = next ? r.nx : r.lo;
    if (next) r.nx = ws.at(r.w);
    r.w += next ? 1u : 0u;
    r.bpos &= 31u;
    return val;
}

// decodeHuff: one thread per coding block, a warp per 32 blocks of a stream
// (the plan numbers the streams' blocks from multiples of 32), its table and
// code words staged in shared memory (huffStageWords at most), its output too,
// and written coalesced.  The
// lane's serial chain per block bounds it: a lookup and a few selects per
// symbol, and for codes longer than the lookup table - half of a lowpass
// band's - the register limits, an offset and the symbol from L1.  24 warps of
// 256^3 lowpass streams: 79 us with words read from global memory, 47 with
// words staged, 39 with the limits in registers; six warps of 4675-symbol
// streams 93 -> 32, most of whose warps held blocks of two streams before.
CC_HD u32 huffStageWords(u32 cb) { return 12u * cb; }   // 12 bits per symbol
CC_HD u32 huffPitch(u32 cb, u32 symBytes) { return cb + (symBytes == 2 ? 2 : 1); }
template <class Sym>
CC_HD size_t huffSmem(u32 cb) {
    return 4 * size_t((1u << kLutBits) + huffStageWords(cb) + 4) + size_t(32) * huffPitch(cb, sizeof(Sym)) * sizeof(Sym);
}

template <class Sym>
__global__ void __launch_bounds__(32) k_decHuff(DecParams p) {
    extern __shared__ __align__(16) unsigned char stage[];
    __shared__ CanonSmem cs;
    if (__any_sync(0xffffffffu, capacityFailed(p))) return;
    const u32 lane = threadIdx.x;
    const u32 b0 = blockIdx.x * 32;
    const u32 s = streamOfBlock(p, p.hList, p.nH, b0);
    const DecStreamDesc sd = p.streams[s];
    const u32 bFirst = b0 - sd.blockFirst;
    const u32 blocks = blocksOf(sd.n, p.cbLog);
    if (bFirst >= blocks) return;
    const u32 nb = min(32u, blocks - bFirst);
    const u32 b = bFirst + lane;
    const u32 rowPitch = huffPitch(p.cb, sizeof(Sym));
    u32* lut = reinterpret_cast<u32*>(stage);
    u32* words = lut + (1u << kLutBits);
    Sym* rows = reinterpret_cast<Sym*>(words + huffStageWords(p.cb) + 4);
    Sym* out = reinterpret_cast<Sym*>(sd.out);
    bool corrupt = false;
    const bool mine = lane < nb;
    const u32 t = sd.tableFirst;
    const DecTableDesc td = p.tables[t];
    const u32* syms = p.syms + td.symOff;
    const u32 cnt = mine ? min(p.cb, sd.n - b * p.cb) : 0u;
    const u32 blockBit = mine ? p.blockOff[td.blockOff + b] : 0u;
    const WordSrc ws = srcOf(p, s);
    // the warp's words: from its first block's to the next warp's first, or the stream's end
    const u32 bit0 = __shfl_sync(0xffffffffu, blockBit, 0);
    const u32 bit1 = bFirst + 32 < blocks ? p.blockOff[td.blockOff + bFirst + 32] : td.cwBits;
    const u32 w0 = bit0 >> 5;
    const u32 nw = bit1 > bit0 ? (bit1 - 1) / 32 - w0 + 1 : 0u;
    const bool staged = nw <= huffStageWords(p.cb);   // warp-uniform
    const DecTable& D = p.dec[t];
    const u32 nSym = D.nSym;
    if (staged) stageWords(words, ws, td.cwWord + w0, nw);
    stageLut(lut, p, t, lane, 32);
    const LongCodes lc = stageLongCodes(cs, p, t);
    __syncwarp();
    if (mine) {
        Sym* row = rows + lane * rowPitch;
        if (nSym == 0xFFFFFFFFu) {
            corrupt = true;
        } else if (nSym <= 1) {
            const u32 single = D.single;
            for (u32 i = 0; i < cnt; ++i) row[i] = Sym(single);
        } else {
            BitReader rd;
            if (staged) {
                const StagedWords sw{words, nw};
                rd.start(sw, blockBit - 32u * w0);
                for (u32 i = 0; i < cnt; ++i)
                    row[i] = Sym(decodeOne<sizeof(Sym) == 2>(sw, lut, cs, lc, nSym, syms, rd, corrupt));
            } else {
                const SourceWords gw{ws, td.cwWord + w0};
                rd.start(gw, blockBit - 32u * w0);
                for (u32 i = 0; i < cnt; ++i)
                    row[i] = Sym(decodeOne<sizeof(Sym) == 2>(gw, lut, cs, lc, nSym, syms, rd, corrupt));
            }
        }
    }
    if (corrupt) atomicOr(p.errors, DEV_ERR_CORRUPT);
    __syncwarp();
    const u64 base = u64(bFirst) * p.cb;
    const u64 lim = u64(sd.n) - base;
    const u64 total = u64(nb) * p.cb < lim ? u64(nb) * p.cb : lim;
    for (u32 k = lane; k < u32(total); k += 32) out[base + k] = rows[(k >> p.cbLog) * rowPitch + (k & (p.cb - 1u))];
}

// Coding blocks of RLHuff stream s that a decode covers: its run-length
// symbol count in blocks, within the blocks planned for its length.
__device__ __forceinline__ u32 rlBlocksOf(const DecParams& p, const DecStreamDesc& sd) {
    return blocksOf(min(sd.m, sd.n), p.cbLog);
}

// Warp tasks of the run-length decode, once the headers are walked: every
// RLHuff stream's coding blocks in groups of 32, so that a warp's blocks
// belong to one stream and warps without blocks are not started.  CTA b
// takes the 1024 streams of chunk b; with more than one chunk,
// k_decRlTaskCounts first writes each chunk's task count (planPart) and CTA b
// starts its tasks after the counts of the chunks before it.
__device__ __forceinline__ u32 rlTaskWarps(const DecParams& p, u32 k, u32& s) {
    s = 0;
    if (k >= p.nRl) return 0;
    s = p.rlList[k];
    return (rlBlocksOf(p, p.streams[s]) + 31u) / 32u;
}

__global__ void __launch_bounds__(1024) k_decRlTaskCounts(DecParams p) {
    __shared__ u32 scratch[40];
    u32 s, tot;
    const u32 warps = rlTaskWarps(p, blockIdx.x * 1024 + threadIdx.x, s);
    blockExclusiveSum<1024>(warps, scratch, &tot);
    if (threadIdx.x == 0) p.planPart[blockIdx.x] = tot;
}

__device__ __forceinline__ void rlTasksChunk(const DecParams& p, u32 b, u32 chunks, u32* scratch) {
    __shared__ u32 sOff[1024], sStr[1024];   // the chunk's streams: first task, stream index
    __shared__ u32 sCarry;
    if (threadIdx.x < 32) {
        // tasks of the chunks before this one
        u32 c = 0;
        for (u32 i = threadIdx.x; i < b; i += 32) c += u32(p.planPart[i]);
        c = __reduce_add_sync(0xffffffffu, c);
        if (threadIdx.x == 0) sCarry = c;
    }
    const u32 base = b * 1024;
    u32 s, tot;
    const u32 warps = rlTaskWarps(p, base + threadIdx.x, s);
    const u32 ex = blockExclusiveSum<1024>(warps, scratch, &tot);   // synchronizes (sCarry visible)
    sOff[threadIdx.x] = ex;
    sStr[threadIdx.x] = s;
    __syncthreads();
    const u32 carry = sCarry;
    // the chunk's tasks over all threads: task i belongs to the last stream
    // whose first task is <= i (streams without tasks share their offset
    // with the next one, so that is never one of them)
    const int n = int(min(1024u, p.nRl - base));
    for (u32 i = threadIdx.x; i < tot; i += 1024) {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sOff[mid] <= i) lo = mid;
            else hi = mid - 1;
        }
        const u32 at = carry + i;
        if (at < p.rlTaskCap) p.rlTasks[at] = (u64(sStr[lo]) << 32) | (32u * (i - sOff[lo]));
    }
    if (b + 1 == chunks && threadIdx.x == 0)
        reinterpret_cast<u32*>(p.rlTasks + p.rlTaskCap)[0] = min(carry + tot, p.rlTaskCap);
}

__global__ void __launch_bounds__(1024) k_decRlTasks(DecParams p) {
    __shared__ u32 scratch[40];
    rlTasksChunk(p, blockIdx.x, gridDim.x, scratch);
}

// Both plans of a call of one chunk each: CTA 0 the symbols', CTA 1 the tasks.
__global__ void __launch_bounds__(1024) k_decPlans(DecParams p) {
    __shared__ u32 scratch[40];
    if (blockIdx.x == 0) symPlanChunk(p, 0, 1, scratch);
    else rlTasksChunk(p, 0, 1, scratch);
}

// The RLHuff streams' outputs, zeroed before the symbol pass writes the
// nonzero symbols (so callers need not zero them): CTA (k, c) zeroes chunk c
// of kZeroChunk symbols of RLHuff stream k, 16-byte stores.
constexpr u32 kZeroChunk = 16384;

template <class Sym>
__global__ void __launch_bounds__(256) k_decZero(DecParams p) {
    const DecStreamDesc& sd = p.streams[p.rlList[blockIdx.x]];
    const u64 lo = u64(blockIdx.y) * kZeroChunk;
    if (lo >= sd.n) return;
    const u64 hi = min(u64(sd.n), lo + kZeroChunk);
    Sym* o = reinterpret_cast<Sym*>(sd.out);
    constexpr u64 kPer = 16 / sizeof(Sym);
    const u64 mis = (reinterpret_cast<uintptr_t>(o + lo) & 15u) / sizeof(Sym);
    const u64 head = min(hi - lo, mis ? kPer - mis : 0);
    if (threadIdx.x < head) o[lo + threadIdx.x] = Sym(0);
    const u64 a = lo + head;
    const u64 nv = (hi - a) / kPer;
    uint4* v = reinterpret_cast<uint4*>(o + a);
    for (u64 k = threadIdx.x; k < nv; k += 256) v[k] = make_uint4(0u, 0u, 0u, 0u);
    for (u64 k = a + nv * kPer + threadIdx.x; k < hi; k += 256) o[k] = Sym(0);
}

// decodeRLHuff (RunLengthKernels.cui:56-66 for the scatter): one lane per
// coding block, 32 consecutive blocks of one stream per warp (k_decRlTasks),
// the warp's code words and long codes staged in its shared memory; the lookup
// table is the CTA's (kSharedLut: its first warp's, warps of another table
// read theirs from global memory - calls of long streams) or each warp's.
// Each lane decodes its block in rounds of kRlRound symbols into its row of
// the warp's shared rows, its bit reader staying in registers between rounds;
// after a round the warp moves the rows out block by block, lane k taking the
// block's element k of the round.  Zero counts (kSymbols false) are stored, 16
// bytes per lane, and their (zc + 1) summed per block.  Symbols are scattered
// to out[block start + sum of (zc + 1) before the element + zc]: the round's
// zero counts, fetched before its symbols are decoded, become positions in the
// round by the lane of the block, four per step beside its 31 neighbours.
// Rows are 36 elements: four 16-bit (8 bytes) per lane are free of conflicts.
// Bound: instruction issue and shared memory (two 256^3 volumes, 14 million
// entries: 36 warp instructions per 32 zero counts and 73 per 32 symbols, 56%
// and 46% of the issue slots), and the lane's chain per symbol (lookup, length,
// next word) where a call has few blocks.
// Three 256^3 streams (26 million entries): zero counts 61 -> 53, symbols 145
// -> 126 us against words read from global memory, a scan over the warp per
// block and round, and the limits searched in global memory; seven streams of
// 100003 symbols 33 -> 26 and 73 -> 38.
constexpr u32 kRlRound = 32;
constexpr u32 kRlWarps = 4;
constexpr u32 kRlPitch = 36;
constexpr u32 kRlSharedTasks = 8;   // mean warp tasks per stream from which a CTA shares one lookup table

CC_HD u32 rlStageWords(u32 cb) { return 6u * cb; }   // 6 bits per symbol
// Bytes of a warp's shared memory: long codes, rows, zero counts, words (and one behind them).
template <class Sym, bool kSymbols>
CC_HD size_t rlWarpSmem(u32 cb) {
    return sizeof(CanonSmem) + (kSymbols ? 2 : 1) * 32 * kRlPitch * sizeof(Sym) + 4 * size_t(rlStageWords(cb) + 4);
}
template <class Sym, bool kSymbols, bool kSharedLut>
CC_HD size_t rlSmem(u32 cb) {
    return kRlWarps * rlWarpSmem<Sym, kSymbols>(cb) + (kSharedLut ? 1 : kRlWarps) * (4u << kLutBits);
}

// Four consecutive elements of a row.
__device__ __forceinline__ void putFour(u16* row, u32 a, u32 b, u32 c, u32 d) {
    *reinterpret_cast<uint2*>(row) = make_uint2((a & 0xFFFFu) | (b << 16), (c & 0xFFFFu) | (d << 16));
}
__device__ __forceinline__ void putFour(u32* row, u32 a, u32 b, u32 c, u32 d) {
    *reinterpret_cast<uint4*>(row) = make_uint4(a, b, c, d);
}
__device__ __forceinline__ void getFour(const u16* row, u32 (&v)[4]) {
    const uint2 x = *reinterpret_cast<const uint2*>(row);
    v[0] = x.x & 0xFFFFu; v[1] = x.x >> 16; v[2] = x.y & 0xFFFFu; v[3] = x.y >> 16;
}
__device__ __forceinline__ void getFour(const u32* row, u32 (&v)[4]) {
    const uint4 x = *reinterpret_cast<const uint4*>(row);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
// 16 bytes of a row, 8-byte aligned.
__device__ __forceinline__ uint4 rowVec(const void* q) {
    const uint2* h = reinterpret_cast<const uint2*>(q);
    const uint2 a = h[0], b = h[1];
    return make_uint4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void rowVec(void* q, uint4 v) {
    uint2* h = reinterpret_cast<uint2*>(q);
    h[0] = make_uint2(v.x, v.y);
    h[1] = make_uint2(v.z, v.w);
}

template <class Sym, bool kSymbols, bool kSharedLut>
__global__ void __launch_bounds__(kRlWarps * 32) k_decRl(DecParams p) {
    constexpr u32 kVec = 16 / sizeof(Sym);        // elements of a 16-byte access
    constexpr u32 kParts = kRlRound / kVec;       // accesses per block and round
    constexpr u32 kWordsPer = 4 / sizeof(Sym);    // elements per 32-bit word
    constexpr bool kValueLut = sizeof(Sym) == 2;
    extern __shared__ __align__(16) unsigned char stage[];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 tasks = reinterpret_cast<const u32*>(p.rlTasks + p.rlTaskCap)[0];
    const u32 wt = blockIdx.x * kRlWarps + warp;
    if (blockIdx.x * kRlWarps >= tasks) return;   // CTA-uniform
    unsigned char* mem = stage + (kSharedLut ? 1 : kRlWarps) * (4u << kLutBits) + warp * rlWarpSmem<Sym, kSymbols>(p.cb);
    CanonSmem& cs = *reinterpret_cast<CanonSmem*>(mem);
    Sym* rows = reinterpret_cast<Sym*>(mem + sizeof(CanonSmem));
    Sym* zs = rows + 32 * kRlPitch;
    u32* words = reinterpret_cast<u32*>(rows + (kSymbols ? 2 : 1) * 32 * kRlPitch);
    u32* lutS = reinterpret_cast<u32*>(stage) + (kSharedLut ? 0u : warp << kLutBits);
    bool lutHere = true;   // warp-uniform: the warp's lookup table is in shared memory
    if (kSharedLut) {
        // the CTA's table: its first warp's
        const u32 t0 = p.streams[u32(p.rlTasks[blockIdx.x * kRlWarps] >> 32)].tableFirst + (kSymbols ? 0u : 1u);
        stageLut(lutS, p, t0, threadIdx.x, kRlWarps * 32);
        if (wt < tasks)
            lutHere = p.streams[u32(p.rlTasks[wt] >> 32)].tableFirst + (kSymbols ? 0u : 1u) == t0;
        __syncthreads();
    }
    if (wt >= tasks) return;   // no block-wide barriers below
    if (__any_sync(0xffffffffu, capacityFailed(p))) return;
    const u64 task = p.rlTasks[wt];
    const u32 s = u32(task >> 32), bFirst = u32(task);
    const DecStreamDesc sd = p.streams[s];
    const u32 t = sd.tableFirst + (kSymbols ? 0u : 1u);
    const u32 blocks = rlBlocksOf(p, sd);
    if (bFirst >= blocks) return;
    const u32 nMine = min(32u, blocks - bFirst);   // lanes 0 .. nMine-1 have a block
    const u32 b = bFirst + lane;
    const bool mine = lane < nMine;
    const DecTableDesc td = p.tables[t];
    const WordSrc ws = srcOf(p, s);
    const u32* symv = p.syms + td.symOff;
    const DecTable& D = p.dec[t];
    const u32 nSym = D.nSym;
    const bool single = nSym <= 1;
    const u32 singleVal = D.single;
    const bool bad = nSym == 0xFFFFFFFFu;   // warp-uniform: nothing is decoded
    bool corrupt = bad;
    const u32 cnt = mine ? min(p.cb, sd.m - b * p.cb) : 0u;
    const u32 blockBit = mine ? p.blockOff[td.blockOff + b] : 0u;
    // the warp's words: from its first block's to the next warp's first, or the stream's end
    const u32 bit0 = __shfl_sync(0xffffffffu, blockBit, 0);
    const u32 bit1 = bFirst + 32 < blocks ? p.blockOff[td.blockOff + bFirst + 32] : td.cwBits;
    const u32 w0 = bit0 >> 5;
    const u32 nw = bit1 > bit0 ? (bit1 - 1) / 32 - w0 + 1 : 0u;
    const bool staged = nw <= rlStageWords(p.cb);   // warp-uniform
    if (staged) stageWords(words, ws, td.cwWord + w0, nw);
    if (!kSharedLut) stageLut(lutS, p, t, lane, 32);
    const LongCodes lc = stageLongCodes(cs, p, t);
    __syncwarp();
    const StagedWords sw{words, nw};
    const SourceWords gw{ws, td.cwWord + w0};
    BitReader rd{0u, 0u, 0u, 0u, 0u};
    if (mine && !bad && !single) {
        if (staged) rd.start(sw, blockBit - 32u * w0);
        else rd.start(gw, blockBit - 32u * w0);
    }
    u32 sum = 0;   // zero counts: the block's sum of (zc + 1)
    // symbols: the block's next output position (its start from the zero-count scan)
    u32 pos = 0;
    if (kSymbols && mine) pos = p.blockSum[p.tables[t + 1].blockOff + b];
    Sym* row = rows + lane * kRlPitch;
    Sym* zcG = reinterpret_cast<Sym*>(p.zc) + sd.zcOff;
    Sym* out = reinterpret_cast<Sym*>(sd.out);
    const u32 cnt0 = __shfl_sync(0xffffffffu, cnt, 0);   // the first block is the longest
    for (u32 r0 = 0; r0 < cnt0; r0 += kRlRound) {
        const u32 n = cnt > r0 ? min(kRlRound, cnt - r0) : 0u;
        const bool full = __all_sync(0xffffffffu, n == kRlRound || !mine);
        // symbols: the round's zero counts of the warp's blocks, kVec elements
        // per lane and step, zero past the stream's m (a part lies whole in
        // them or is taken element by element)
        uint4 z[kSymbols ? kParts : 1];
        if (kSymbols) {
#pragma unroll
            for (u32 k = 0; k < kParts; ++k) {
                const u32 c = k * 32 + lane, j = c / kParts, e = (c % kParts) * kVec;
                const u32 at = (bFirst + j) * p.cb + r0 + e;
                z[k] = make_uint4(0u, 0u, 0u, 0u);
                if (at + kVec <= sd.m) {
                    z[k] = *reinterpret_cast<const uint4*>(zcG + at);
                } else if (at < sd.m) {
                    u32 v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (u32 q = 0; q < kVec; ++q)
                        if (at + q < sd.m) v[q / kWordsPer] |= u32(zcG[at + q]) << (16 * (q % kWordsPer));
                    z[k] = make_uint4(v[0], v[1], v[2], v[3]);
                }
            }
        }
        if (!bad) {
            if (full && staged && lutHere && !single) {
                if (mine) {
#pragma unroll 1
                    for (u32 i = 0; i < kRlRound; i += 4) {
                        u32 v[4];
#pragma unroll
                        for (u32 q = 0; q < 4; ++q)
                            v[q] = decodeOne<kValueLut>(sw, lutS, cs, lc, nSym, symv, rd, corrupt);
                        putFour(row + i, v[0], v[1], v[2], v[3]);
                        if (!kSymbols) sum += v[0] + v[1] + v[2] + v[3] + 4u;
                    }
                }
            } else {
                const u32* lut = lutHere ? lutS : p.lut + (u64(t) << kLutBits);
                for (u32 i = 0; i < n; ++i) {
                    const u32 v = single ? singleVal
                                : staged ? decodeOne<kValueLut>(sw, lut, cs, lc, nSym, symv, rd, corrupt)
                                         : decodeOne<kValueLut>(gw, lut, cs, lc, nSym, symv, rd, corrupt);
                    row[i] = Sym(v);
                    if (!kSymbols) sum += v + 1u;
                }
            }
        }
        if (!kSymbols) {
            __syncwarp();
#pragma unroll
            for (u32 k = 0; k < kParts; ++k) {
                const u32 c = k * 32 + lane, j = c / kParts, e = (c % kParts) * kVec;
                const u32 at = (bFirst + j) * p.cb + r0 + e;
                if (at + kVec <= sd.m) {
                    *reinterpret_cast<uint4*>(zcG + at) = rowVec(rows + j * kRlPitch + e);
                } else {
                    for (u32 q = 0; q < kVec && at + q < sd.m; ++q) zcG[at + q] = rows[j * kRlPitch + e + q];
                }
            }
        } else {
#pragma unroll
            for (u32 k = 0; k < kParts; ++k) {
                const u32 c = k * 32 + lane, j = c / kParts, e = (c % kParts) * kVec;
                rowVec(zs + j * kRlPitch + e, z[k]);
            }
            __syncwarp();
            // positions within the round, in place of the zero counts
            Sym* zrow = zs + lane * kRlPitch;
            u32 run = 0;
#pragma unroll
            for (u32 i = 0; i < kRlRound; i += 4) {
                u32 v[4];
                getFour(zrow + i, v);
                v[0] += run;
                v[1] += v[0] + 1u;
                v[2] += v[1] + 1u;
                v[3] += v[2] + 1u;
                run = v[3] + 1u;
                putFour(zrow + i, v[0], v[1], v[2], v[3]);
            }
            run -= kRlRound - n;   // counts past n are zero
            const bool fits = sizeof(Sym) == 4 || __all_sync(0xffffffffu, run <= 65536u);
            __syncwarp();
            if (fits) {
#pragma unroll 4
                for (u32 j = 0; j < nMine; ++j) {
                    const u32 c = full ? kRlRound : __shfl_sync(0xffffffffu, n, j);
                    const u32 start = __shfl_sync(0xffffffffu, pos, j);
                    if (lane < c) {
                        const u32 to = start + u32(zs[j * kRlPitch + lane]);
                        if (to < sd.n) out[to] = rows[j * kRlPitch + lane];
                        else corrupt = true;
                    }
                }
            } else {
                // zero counts past the format's 255, positions kept modulo
                // 2^16: the lane places its own, each count from the difference
                u32 at = pos - 1u, before = 0xFFFFu;
                for (u32 i = 0; i < n; ++i) {
                    const u32 now = u32(zrow[i]);
                    at += ((now - before - 1u) & 0xFFFFu) + 1u;
                    before = now;
                    if (at < sd.n) out[at] = row[i];
                    else corrupt = true;
                }
            }
            pos += run;
        }
        __syncwarp();
    }
    if (!kSymbols && mine) p.blockSum[td.blockOff + b] = sum;
    if (corrupt) atomicOr(p.errors, DEV_ERR_CORRUPT);
}

// Exclusive scan of the per-block output lengths: a warp per RLHuff stream.
__global__ void __launch_bounds__(256) k_decScan(DecParams p) {
    const u32 k = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (k >= p.nRl) return;
    const DecStreamDesc sd = p.streams[p.rlList[k]];
    const u32 blocks = blocksOf(sd.m, p.cbLog);
    u32* bs = p.blockSum + p.tables[sd.tableFirst + 1].blockOff;
    const u32 total = warpExclusiveScan8(bs, bs, blocks, 0u);
    // the last symbol's position must be < n: total length <= n
    if ((threadIdx.x & 31u) == 0 && total > sd.n) atomicOr(p.errors, DEV_ERR_CORRUPT);
}

// The same with a CTA per stream (wideBlockScan): a warp takes 38 us over the 16384
// blocks of a 256^3 volume's band, 512 threads 13.
__global__ void __launch_bounds__(512) k_decScanWide(DecParams p) {
    __shared__ u32 scratch[40];
    const DecStreamDesc sd = p.streams[p.rlList[blockIdx.x]];
    const u32 blocks = blocksOf(sd.m, p.cbLog);
    u32* bs = p.blockSum + p.tables[sd.tableFirst + 1].blockOff;
    const u32 total = blockExclusiveScan8<512>(bs, bs, blocks, scratch);
    if (threadIdx.x == 0 && total > sd.n) atomicOr(p.errors, DEV_ERR_CORRUPT);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct HostReader {
    const u32* w;
    u32 size;
    u64 pos;
    bool ok = true;
    u32 readBits(u32 n) {
        if (n == 0) return 0;
        if (pos + n > size) { ok = false; pos = size; return 0; }
        u32 v = 0;
        for (u32 k = 0; k < n;) {
            u32 bp = u32(pos & 31u);
            u32 cur = std::min(n - k, 32 - bp);
            u32 bits = (w[pos >> 5] >> (32 - bp - cur)) & (cur == 32 ? 0xffffffffu : ((1u << cur) - 1u));
            v = cur == 32 ? bits : ((v << cur) | bits);
            pos += cur;
            k += cur;
        }
        return v;
    }
    void align() {  // BitStream.h:290-308 (stops at the end)
        u64 a = ceilDiv(pos, 32) * 32;
        pos = std::min<u64>(a, size);
    }
    void skip(u64 n) { pos = std::min<u64>(pos + n, size); }
};

// Parses one table header (HuffmanTable.cu:117-151) into d (bit positions in
// the caller's stream) and returns false on a malformed header.
static bool walkTable(HostReader& r, u32 log2Max, u32 leavesMax, DecTableDesc& d) {
    d.hdrBit = r.pos;
    d.nLen = r.readBits(5);
    r.skip(u64(d.nLen) * log2Max);
    d.nSym = r.readBits(log2Max);
    const bool longSym = log2Max > 16;
    d.symbolBits = r.readBits(longSym ? 5 : 4);
    if (!longSym && d.symbolBits == 0 && d.nSym > 1) d.symbolBits = 16;   // HuffmanTable.cu:138-139
    r.skip(u64(d.nSym) * d.symbolBits);
    return r.ok && d.nSym <= leavesMax;
}

static bool walkPayload(HostReader& r, u32 count, u32 cb, DecTableDesc& d) {
    r.align();
    d.cwBits = r.readBits(32);
    d.cwWord = r.pos / 32;
    r.skip(ceilDiv(d.cwBits, 32) * 32);
    r.align();
    d.offWord = r.pos / 32;
    r.skip(ceilDiv(count, cb) * 16);
    r.align();
    d.count = count;
    return r.ok;
}

// Descriptor layout of one call in a host buffer and in device memory.
struct DecLayout {
    size_t offStreams = 0, offTables, offSources, offRl, offH, bytes;
    DecLayout(u32 S, u32 T, u32 B) {
        offTables = alignUp(sizeof(DecStreamDesc) * S, 64);
        offSources = alignUp(offTables + sizeof(DecTableDesc) * T, 64);
        offRl = alignUp(offSources + sizeof(DecSource) * B, 64);
        offH = alignUp(offRl + sizeof(u32) * S, 64);
        bytes = offH + sizeof(u32) * S;
    }
};

// Fills the stream/table skeleton (kinds, sizes, table and block offsets)
// and the RLHuff / Huff lists of a call.
static int planDecode(cc_instance* I, const u32* kinds, const u32* ns, void* const* outs, const u32* sourceOf, u32 S,
                      u32 B, char* slot, size_t slotBytes, DecPlan& dc) {
    dc = DecPlan{};
    u32 T = 0;
    for (u32 s = 0; s < S; ++s) T += kinds[s] == KIND_RLHUFF ? 2u : 1u;
    const DecLayout L(S, T, B);
    if (S > I->capStreams || T > I->capTables || L.bytes > slotBytes) {
        setError("decode: call exceeds the instance capacity (%u streams)", S);
        return CC_ERR_CAPACITY;
    }
    DecStreamDesc* sd = reinterpret_cast<DecStreamDesc*>(slot + L.offStreams);
    DecTableDesc* td = reinterpret_cast<DecTableDesc*>(slot + L.offTables);
    u32* rl = reinterpret_cast<u32*>(slot + L.offRl);
    u32* hl = reinterpret_cast<u32*>(slot + L.offH);
    u32 t = 0;
    u64 blocks = 0, zc = 0, rlBlocks = 0, hBlocks = 0;
    for (u32 s = 0; s < S; ++s) {
        const u32 nb = u32(ceilDiv(ns[s], I->codingBlockSize));
        DecStreamDesc d{};
        d.out = outs[s];
        d.n = ns[s];
        d.m = ns[s];
        dc.maxN = std::max<u32>(dc.maxN, ns[s]);
        d.kind = kinds[s];
        d.tableFirst = t;
        d.source = sourceOf[s];
        const u32 parts = d.kind == KIND_RLHUFF ? 2u : 1u;
        for (u32 w = 0; w < parts; ++w) {
            DecTableDesc tt{};
            tt.stream = s;
            tt.blockOff = u32(blocks);
            blocks += nb;
            td[t++] = tt;
        }
        if (d.kind == KIND_RLHUFF) {
            d.zcOff = zc;
            zc = alignUp(zc + ns[s], 8);   // 16-byte aligned zero counts of every stream
            d.blockFirst = u32(rlBlocks);
            rlBlocks += nb;
            rl[dc.nRl++] = s;
            dc.rlMaxN = std::max<u32>(dc.rlMaxN, ns[s]);
        } else {
            d.blockFirst = u32(hBlocks);
            hBlocks += huffBlocksPlanned(nb);
            hl[dc.nH++] = s;
        }
        sd[s] = d;
    }
    if (blocks > I->capBlocks || zc > I->capCompact + 8ull * I->capStreams) {
        setError("decode: call exceeds the instance capacity (%llu coding blocks, %llu run-length symbols)",
                 (unsigned long long)blocks, (unsigned long long)zc);
        return CC_ERR_CAPACITY;
    }
    dc.S = S;
    dc.T = T;
    dc.B = B;
    dc.rlBlocks = u32(rlBlocks);
    dc.hBlocks = u32(hBlocks);
    dc.bytes = L.bytes;
    dc.offStreams = L.offStreams;
    dc.offTables = L.offTables;
    dc.offSources = L.offSources;
    dc.offRl = L.offRl;
    dc.offH = L.offH;
    return CC_OK;
}

// The run-length decode kernels by symbol and lookup table place, with their
// dynamic shared memory.
template <class Sym, bool kSymbols, bool kSharedLut>
static cudaError_t rlSmemAttribute(cc_instance* I) {
    const int which = kAttrDecRl + (sizeof(Sym) == 4 ? 4 : 0) + (kSymbols ? 2 : 0) + (kSharedLut ? 1 : 0);
    return ensureSmemAttribute(reinterpret_cast<const void*>(k_decRl<Sym, kSymbols, kSharedLut>), which, I->device,
                               rlSmem<Sym, kSymbols, kSharedLut>(I->codingBlockSize));
}

template <class Sym>
static cudaError_t decodeSmemAttributes(cc_instance* I) {
    cudaError_t e = ensureSmemAttribute(reinterpret_cast<const void*>(k_decHuff<Sym>),
                                        sizeof(Sym) == 4 ? kAttrDecHuff32 : kAttrDecHuff16, I->device,
                                        huffSmem<Sym>(I->codingBlockSize));
    if (e == cudaSuccess) e = rlSmemAttribute<Sym, false, false>(I);
    if (e == cudaSuccess) e = rlSmemAttribute<Sym, false, true>(I);
    if (e == cudaSuccess) e = rlSmemAttribute<Sym, true, false>(I);
    if (e == cudaSuccess) e = rlSmemAttribute<Sym, true, true>(I);
    return e;
}

template <class Sym, bool kSymbols>
static void launchRl(const DecParams& p, u32 ctas, cudaStream_t st) {
    if (p.rlBlocks / 32 >= u64(kRlSharedTasks) * p.nRl)
        k_decRl<Sym, kSymbols, true><<<ctas, kRlWarps * 32, rlSmem<Sym, kSymbols, true>(p.cb), st>>>(p);
    else
        k_decRl<Sym, kSymbols, false><<<ctas, kRlWarps * 32, rlSmem<Sym, kSymbols, false>(p.cb), st>>>(p);
    countLaunch();
}

template <class Sym>
static int launchDecodeBackEnd(cc_instance* I, const DecParams& p) {
    cudaStream_t st = I->stream;
    CC_TRY_CUDA(decodeSmemAttributes<Sym>(I), "decode smem");
    // a side stream beside the RLHuff chain: the zero fill of its outputs,
    // which it needs before the symbols, and the Huff streams' decode (the two
    // share only the read-only tables and the error flags), joined at the end
    const bool fork = p.hBlocks && p.rlBlocks;
    cudaStream_t hs = fork ? I->buildSide2 : st;
    auto zeroFill = [&](cudaStream_t q) {
        SectionTimer t(I, "dec.zero_fill", q);
        k_decZero<Sym><<<dim3(p.nRl, u32(ceilDiv(p.rlMaxN, kZeroChunk))), 256, 0, q>>>(p);
        countLaunch();
    };
    if (fork) {
        CC_TRY_CUDA(cudaEventRecord(I->decFork, st), "decode fork");
        CC_TRY_CUDA(cudaStreamWaitEvent(hs, I->decFork, 0), "decode fork");
        zeroFill(hs);
        CC_TRY_CUDA(cudaEventRecord(I->decZeroed, hs), "decode zero fill");
    }
    const u32 symChunks = std::max<u32>(1, u32(ceilDiv(p.T, kPlanChunk)));
    const u32 rlChunks = std::max<u32>(1, u32(ceilDiv(p.nRl, 1024)));
    const bool onePlan = symChunks == 1 && rlChunks == 1 && p.rlBlocks;
    {
        SectionTimer t(I, "dec.sym_plan", st);
        if (onePlan) k_decPlans<<<2, 1024, 0, st>>>(p);
        else k_decSymPlan<<<symChunks, 1024, 0, st>>>(p);
        countLaunch();
        if (symChunks > 1) { k_decSymPlanCarry<<<symChunks - 1, 1024, 0, st>>>(p); countLaunch(); }
    }
    {
        SectionTimer t(I, "dec.tables", st);
        if (p.T <= I->smCount || wideBlockScan(p.T, u32(ceilDiv(p.maxN, p.cb)), I->smCount))
            k_decTables<kDecThreadsWide><<<p.T, kDecThreadsWide, 0, st>>>(p);
        else k_decTables<kDecThreads><<<p.T, kDecThreads, 0, st>>>(p);
        countLaunch();
    }
    if (fork) {
        CC_TRY_CUDA(cudaEventRecord(I->decTablesReady, st), "decode tables");
        CC_TRY_CUDA(cudaStreamWaitEvent(hs, I->decTablesReady, 0), "decode tables");
    }
    if (p.hBlocks) {
        SectionTimer t(I, "dec.huffman", hs);
        k_decHuff<Sym><<<u32(ceilDiv(p.hBlocks, 32)), 32, huffSmem<Sym>(p.cb), hs>>>(p);
        countLaunch();
    }
    if (fork) CC_TRY_CUDA(cudaEventRecord(I->decJoin, hs), "decode join");
    if (p.rlBlocks) {
        const u32 g = u32(ceilDiv(u64(p.rlBlocks) / 32 + p.nRl, kRlWarps));   // warp tasks <= rlBlocks / 32 + nRl
        if (!onePlan) {
            SectionTimer t(I, "dec.rl_tasks", st);
            if (rlChunks > 1) { k_decRlTaskCounts<<<rlChunks, 1024, 0, st>>>(p); countLaunch(); }
            k_decRlTasks<<<rlChunks, 1024, 0, st>>>(p);
            countLaunch();
        }
        if (!fork) zeroFill(st);
        {
            SectionTimer t(I, "dec.zero_counts", st);
            launchRl<Sym, false>(p, g, st);
        }
        {
            SectionTimer t(I, "dec.run_scan", st);
            if (wideBlockScan(p.nRl, u32(ceilDiv(p.rlMaxN, p.cb)), I->smCount)) k_decScanWide<<<p.nRl, 512, 0, st>>>(p);
            else k_decScan<<<u32(ceilDiv(p.nRl, 8)), 256, 0, st>>>(p);
            countLaunch();
        }
        if (fork) CC_TRY_CUDA(cudaStreamWaitEvent(st, I->decZeroed, 0), "decode zero fill");
        {
            SectionTimer t(I, "dec.symbols_scatter", st);
            launchRl<Sym, true>(p, g, st);
        }
    }
    if (fork) CC_TRY_CUDA(cudaStreamWaitEvent(st, I->decJoin, 0), "decode join");
    CC_TRY_CUDA(cudaGetLastError(), "decode launch");
    return CC_OK;
}

int prepareDecodeAttributes(cc_instance* I) {
    CC_TRY_CUDA(I->symBytes == 2 ? decodeSmemAttributes<u16>(I) : decodeSmemAttributes<u32>(I), "decode smem");
    return CC_OK;
}

static DecParams makeDecParams(cc_instance* I, const DecPlan& dc) {
    char* d = static_cast<char*>(dc.dev);
    DecParams p{};
    p.S = dc.S;
    p.T = dc.T;
    p.nSrc = dc.B;
    p.nRl = dc.nRl;
    p.nH = dc.nH;
    p.rlBlocks = dc.rlBlocks;
    p.rlMaxN = dc.rlMaxN;
    p.maxN = dc.maxN;
    p.hBlocks = dc.hBlocks;
    p.cb = I->codingBlockSize;
    p.cbLog = 31u - u32(__builtin_clz(p.cb));
    p.log2Max = I->log2Max;
    p.symBytes = I->symBytes;
    p.leavesMax = I->leavesMax;
    p.capLeaves = I->capLeaves;
    p.streams = reinterpret_cast<DecStreamDesc*>(d + dc.offStreams);
    p.tables = reinterpret_cast<DecTableDesc*>(d + dc.offTables);
    p.sources = reinterpret_cast<DecSource*>(d + dc.offSources);
    p.rlList = reinterpret_cast<const u32*>(d + dc.offRl);
    p.hList = reinterpret_cast<const u32*>(d + dc.offH);
    p.wordsBase = dc.wordsBase;
    p.wordOff = dc.wordOff;
    p.bitSize = dc.bitSize;
    p.dec = I->decTables;
    p.syms = I->decSyms;
    p.lut = I->decLut;
    p.blockOff = I->blockOff;
    p.blockSum = I->blockSum;
    p.rlTasks = I->decRlTasks;
    p.rlTaskCap = u32(u64(I->capBlocks) / 32 + I->capStreams);
    p.zc = static_cast<char*>(I->zc);
    p.planPart = I->planPart + planPartWords(I->capTables);
    p.errors = I->errors + 4;
    return p;
}

// Host-walk front end (cc_decode): the reference's decode entry points.
int decodeDevice(cc_instance* I, int kind, const u32* const* words, const u32* bitSizes, u32* bitPos, u32 bsCount,
                 const u32* bsIndex, void* const* outs, u32 S, u32 n) {
    if (S == 0) return CC_OK;
    if (S > I->streamCountMax) { setError("stream count %u exceeds instance limit %u", S, I->streamCountMax); return CC_ERR_CAPACITY; }
    if (n > I->elemCountPerStreamMax) { setError("symbol count %u exceeds instance limit %u", n, I->elemCountPerStreamMax); return CC_ERR_CAPACITY; }
    std::vector<u32> kinds(S, u32(kind)), ns(S, n), srcOf(S);
    for (u32 s = 0; s < S; ++s) {
        srcOf[s] = bsIndex ? bsIndex[s] : 0u;
        if (srcOf[s] >= bsCount) { setError("decode: bit stream index out of range"); return CC_ERR_INVALID_ARGUMENT; }
    }
    char* slot = I->takeRingSlot();
    DecPlan dc;
    int rc = planDecode(I, kinds.data(), ns.data(), outs, srcOf.data(), S, bsCount, slot, I->hostRingBytes, dc);
    if (rc) return rc;
    const DecLayout L(dc.S, dc.T, dc.B);
    DecStreamDesc* sd = reinterpret_cast<DecStreamDesc*>(slot + L.offStreams);
    DecTableDesc* td = reinterpret_cast<DecTableDesc*>(slot + L.offTables);
    DecSource* src = reinterpret_cast<DecSource*>(slot + L.offSources);
    // walk the headers
    std::vector<u64> lo(bsCount, ~0ull), hi(bsCount, 0);
    std::vector<HostReader> rd(bsCount);
    for (u32 k = 0; k < bsCount; ++k) rd[k] = HostReader{words[k], bitSizes[k], bitPos[k]};
    for (u32 s = 0; s < S; ++s) {
        const u32 k = srcOf[s];
        HostReader& r = rd[k];
        u64 start = r.pos;
        bool ok = true;
        u32 m = n;
        DecTableDesc& t0 = td[sd[s].tableFirst];
        if (kind == KIND_RLHUFF) {
            r.align();
            start = r.pos;
            m = r.readBits(32);
            ok = r.ok && m <= n;
            DecTableDesc& t1 = td[sd[s].tableFirst + 1];
            ok = ok && walkTable(r, I->log2Max, I->leavesMax, t0) && walkPayload(r, m, I->codingBlockSize, t0);
            ok = ok && walkTable(r, I->log2Max, I->leavesMax, t1) && walkPayload(r, m, I->codingBlockSize, t1);
        } else {
            ok = walkTable(r, I->log2Max, I->leavesMax, t0) && walkPayload(r, n, I->codingBlockSize, t0);
        }
        if (!ok) { setError("decode: corrupt or truncated bit stream (stream %u)", s); return CC_ERR_CORRUPT_STREAM; }
        lo[k] = std::min<u64>(lo[k], start / 32);
        hi[k] = std::max<u64>(hi[k], ceilDiv(r.pos, 32));
        sd[s].m = m;
    }
    // stage the touched words of every bit stream and rebase the positions
    std::vector<u64> base(bsCount, 0);
    u64 total = 0;
    for (u32 k = 0; k < bsCount; ++k) {
        if (hi[k] <= lo[k]) continue;
        base[k] = total;
        total += hi[k] - lo[k] + 2;
    }
    if (total > I->stagedWordsMax) { setError("decode: bit stream larger than the instance staging (%llu words)", (unsigned long long)total); return CC_ERR_CAPACITY; }
    cudaStream_t st = I->stream;
    for (u32 k = 0; k < bsCount; ++k) {
        const u64 span = hi[k] > lo[k] ? hi[k] - lo[k] + 2 : 0;
        src[k] = DecSource{I->stagedWords + base[k], span, span * 32, 0, 0, 0, 0};
        if (hi[k] <= lo[k]) continue;
        const u64 nw = std::min<u64>(hi[k], ceilDiv(bitSizes[k], 32)) - lo[k];
        CC_TRY_CUDA(cudaMemcpyAsync(I->stagedWords + base[k], words[k] + lo[k], nw * 4, cudaMemcpyHostToDevice, st), "stage bit stream");
        CC_TRY_CUDA(cudaMemsetAsync(I->stagedWords + base[k] + nw, 0, (span - nw) * 4, st), "pad staging");
    }
    for (u32 t = 0; t < dc.T; ++t) {
        const u32 k = srcOf[td[t].stream];
        td[t].hdrBit -= lo[k] * 32;
        td[t].cwWord -= lo[k];
        td[t].offWord -= lo[k];
    }
    dc.dev = I->dPlan;
    CC_TRY_CUDA(cudaMemcpyAsync(I->dPlan, slot, L.bytes, cudaMemcpyHostToDevice, st), "upload decode plan");
    cudaEventRecord(I->ringEvent[(I->ringNext + cc_instance::kRing - 1) % cc_instance::kRing], st);
    CC_TRY_CUDA(cudaMemsetAsync(I->errors + 4, 0, sizeof(u32), st), "memset errors");
    const DecParams p = makeDecParams(I, dc);
    rc = I->symBytes == 2 ? launchDecodeBackEnd<u16>(I, p) : launchDecodeBackEnd<u32>(I, p);
    if (rc) return rc;
    for (u32 k = 0; k < bsCount; ++k) bitPos[k] = u32(rd[k].pos);
    return CC_OK;
}

// Device-walk front end, step 1: descriptors into `slot`.
int decodePrepare(cc_instance* I, const DecStreamSpec* streams, u32 S, const DecSourceSpec* sources, u32 B,
                  char* slot, size_t slotBytes, DecPlan& dc) {
    std::vector<u32> kinds(S), ns(S), srcOf(S);
    std::vector<void*> outs(S);
    for (u32 s = 0; s < S; ++s) {
        kinds[s] = streams[s].kind;
        ns[s] = streams[s].n;
        outs[s] = streams[s].out;
        srcOf[s] = streams[s].source;
        if (srcOf[s] >= B) { setError("decode: source index out of range"); return CC_ERR_INVALID_ARGUMENT; }
        if (s > 0 && srcOf[s] < srcOf[s - 1]) { setError("decode: streams must be grouped by source"); return CC_ERR_INVALID_ARGUMENT; }
    }
    int rc = planDecode(I, kinds.data(), ns.data(), outs.data(), srcOf.data(), S, B, slot, slotBytes, dc);
    if (rc) return rc;
    const DecLayout L(dc.S, dc.T, dc.B);
    DecSource* src = reinterpret_cast<DecSource*>(slot + L.offSources);
    for (u32 k = 0; k < B; ++k)
        src[k] = DecSource{sources[k].words, ceilDiv(sources[k].bitSize, 32), sources[k].bitSize, sources[k].startBit, 0, 0, 0};
    for (u32 s = 0; s < S; ++s) {
        DecSource& d = src[srcOf[s]];
        if (d.streamCount == 0) d.firstStream = s;
        ++d.streamCount;
    }
    return CC_OK;
}

// Device-walk front end, step 2: the launches (descriptors at dc.dev).
int decodeLaunch(cc_instance* I, const DecPlan& dc) {
    if (dc.S == 0) return CC_OK;
    cudaStream_t st = I->stream;
    CC_TRY_CUDA(cudaMemsetAsync(I->errors + 4, 0, sizeof(u32), st), "memset errors");
    const DecParams p = makeDecParams(I, dc);
    { SectionTimer t(I, "dec.walk", st); k_decWalk<<<u32(ceilDiv(dc.B, kWalkWarps)), kWalkWarps * 32, 0, st>>>(p); countLaunch(); }
    return I->symBytes == 2 ? launchDecodeBackEnd<u16>(I, p) : launchDecodeBackEnd<u32>(I, p);
}

}  // namespace ccb

using namespace ccb;

extern "C" {

int cc_decode(cc_instance* I, int kind, int symbolBytes, const uint32_t* const* words, const uint32_t* bitSizes,
              uint32_t* bitPositions, uint32_t bsCount, const uint32_t* bsIndex, void* const* dOut, uint32_t S,
              uint32_t n) {
    if (!I || (S && (!words || !bitSizes || !bitPositions || !dOut || bsCount == 0))) {
        setError("cc_decode: null argument");
        return CC_ERR_INVALID_ARGUMENT;
    }
    if (kind != KIND_RLHUFF && kind != KIND_HUFF) { setError("cc_decode: bad kind %d", kind); return CC_ERR_INVALID_ARGUMENT; }
    if (u32(symbolBytes) != I->symBytes) {
        setError("cc_decode: %d-byte symbols need an instance with log2HuffmanDistinctSymbolCountMax %s 16",
                 symbolBytes, symbolBytes == 2 ? "<=" : ">");
        return CC_ERR_INVALID_ARGUMENT;
    }
    DeviceGuard deviceGuard(I->device);
    return decodeDevice(I, kind, words, bitSizes, bitPositions, bsCount, bsIndex, dOut, S, n);
}

// Reads the device error flags of the last decode (synchronizes the stream).
int cc_decode_status(cc_instance* I) {
    if (!I) return CC_ERR_INVALID_ARGUMENT;
    u32 flags = 0;
    CC_TRY_CUDA(cudaMemcpyAsync(&flags, I->errors + 4, sizeof(u32), cudaMemcpyDeviceToHost, I->stream), "decode status");
    CC_TRY_CUDA(cudaStreamSynchronize(I->stream), "decode status");
    return deviceErrorStatus(flags, "decode");
}

}  // extern "C"
