// encode.cu - device entropy encoder: zero-run RLE, histograms, Huffman table
// construction, codeword packing and bit-stream assembly, all on the GPU.
// Replaces encodeRLHuff / encodeHuff (Encode.cpp:207-471, :648-790) and the
// Tier-0 pieces they call (RunLength.cu:82-188, Histogram.cu:109-289,
// HuffmanTable.cu:385-596, Huffman.cu:73-187, PackInc.cu:210-219).
//
// One call codes a batch of streams of any sizes and of both kinds (a whole
// volume: the lowpass band with encodeHuff and every level's bands with
// encodeRLHuff, or many bricks).  Work is flattened: run-length tiles and
// coding blocks are numbered across all streams and found back by binary
// search over the per-stream / per-table offsets, so one launch of each
// kernel covers the batch and all Huffman tables are built concurrently.
// Launch sequence (no host round trip until the result is read):
//   summary -> scan -> histPlan -> zeroHist -> write(+histograms)
//   -> tableBuild -> blockBits -> blockScan -> layout -> pack (with the headers)
#include <cstring>

#include "capi_internal.cuh"
#include "table_build.cuh"

namespace ccb {

struct EncParams {
    u32 S, T;
    u32 totalTiles, totalBlocks;
    u32 maxCount;     // symbols of the longest stream
    u32 cb, cbLog, log2Max, bins, symBytes;   // cb = 2^cbLog
    const EncStreamDev* streams;
    const EncTableDev* tables;
    char* compact;
    char* zc;
    RunSum* tiles;
    TileStart* tileStart;
    u32* streamMax;
    u32* counts;
    u32* hist;
    uint2* enc;
    TableMeta* meta;
    u32* headers;
    u32* blockBits;
    u32* blockOff;
    u32* runTable;    // [runs] table of each run of coding blocks (k_planFill)
    u32* tileStream;  // [totalTiles] stream of each run-length tile (k_encBegin)
    SegmentLayout* layout;
    u32* out;
    u64 outWordsMax;
    u64 capHist, capLeaves, capHdr;
    u32* errors;
    u64* totals;
    u64* leafWork;
    u32* parentWork;
    u32* orderWork;
    u32* leafSymWork;
    u32* tierTables;  // [4][T]: the tables of each leaf-count tier (k_leafTiers); counts in totals[4..7]
    u64* planPart;    // [8 per chunk]: sums of each plan chunk (k_histPlan)
    u32 heapCap;      // bound of the call's leaf counts (at most kBuildSmemLeaves)
    u32 buildLo, buildHi;   // k_tableBuild builds the tables with buildLo <= leaves <= buildHi
    u32 buildTier;    // k_tableBuild: kBuildEach (table blockIdx.x) or the tier whose list its CTAs walk
};


// Error flag of the call, read once per block and shared so that every
// thread of the block takes the same branch.
__device__ __forceinline__ bool blockFailed(const EncParams& p) {
    __shared__ u32 sFailed;
    if (threadIdx.x == 0) sFailed = *reinterpret_cast<volatile const u32*>(p.errors);
    __syncthreads();
    return sFailed != 0;
}
__device__ __forceinline__ bool warpFailed(const EncParams& p) {
    return __any_sync(0xffffffffu, *reinterpret_cast<volatile const u32*>(p.errors) != 0);
}

// Stream owning run-length tile `tile`: one load from the map k_encBegin
// writes at the start of a call.
__device__ __forceinline__ u32 streamOfTile(const EncParams& p, u32 tile) { return p.tileStream[tile]; }

// Input symbols of table t and their count.
template <class Sym>
__device__ __forceinline__ const Sym* tableInput(const EncParams& p, const EncTableDev& td, u32& count) {
    const EncStreamDev& sd = p.streams[td.stream];
    if (sd.kind == KIND_RLHUFF) {
        count = p.counts[td.stream];
        return reinterpret_cast<const Sym*>(td.which ? p.zc : p.compact) + sd.compactOff;
    }
    count = sd.n;
    return reinterpret_cast<const Sym*>(sd.in);
}

// Run-length tiles: kRleWarps warps x 32 groups x 32 symbols.  Warp w
// covers symbols [w * 1024, (w + 1) * 1024) of the tile; group k of it is 32
// consecutive symbols, lane k's.  They pass through shared memory, a padded
// row per group, so that global memory is read 16 bytes per lane and a lane
// has its own symbols at hand: a nonzero mask per lane describes the warp's
// 1024 symbols, and the run-length bookkeeping is warp scans over the groups.
// Positions are kept +1 so that 0 means "no nonzero".
constexpr u32 kRleWarps = kRleThreads / 32;
constexpr u32 kRlePitch = 36;   // elements per row: a lane's 8 (16-bit: 16 bytes of 4) are free of conflicts
static_assert(kRleTile == kRleWarps * 1024, "a tile is 32 groups of 32 symbols per warp");

// Group data of lane k of the calling warp (its group k).
struct GroupRuns {
    u32 mask, cnt, firstP1, lastP1;
};

__device__ __forceinline__ void putRow(u16* row, uint4 v) {   // 8-byte aligned
    reinterpret_cast<uint2*>(row)[0] = make_uint2(v.x, v.y);
    reinterpret_cast<uint2*>(row)[1] = make_uint2(v.z, v.w);
}
__device__ __forceinline__ void putRow(u32* row, uint4 v) { *reinterpret_cast<uint4*>(row) = v; }

// Loads the warp's 1024 symbols from stream position wbase (zero beyond n)
// into its rows and returns lane k's group k mask data; maxSym receives the
// warp's largest symbol.
template <class Sym>
__device__ __forceinline__ GroupRuns loadGroups(const Sym* in, u32 wbase, u32 n, Sym* rows, u32& maxSym) {
    constexpr u32 kVec = 16 / sizeof(Sym), kParts = 32 / kVec;   // elements per access, accesses per group
    const u32 lane = threadIdx.x & 31u;
    maxSym = 0;
    if (wbase >= n) return GroupRuns{0u, 0u, 0u, 0u};   // warp-uniform
    if ((reinterpret_cast<uintptr_t>(in + wbase) & 15u) == 0) {
        uint4 v[kParts];
#pragma unroll
        for (u32 k = 0; k < kParts; ++k) {
            const u32 at = wbase + (k * 32u + lane) * kVec;
            v[k] = make_uint4(0u, 0u, 0u, 0u);
            if (at + kVec <= n) {
                v[k] = *reinterpret_cast<const uint4*>(in + at);
            } else if (at < n) {
                u32 x[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (u32 q = 0; q < kVec; ++q)
                    if (at + q < n) x[q * sizeof(Sym) / 4] |= u32(in[at + q]) << (sizeof(Sym) == 2 ? 16 * (q & 1) : 0);
                v[k] = make_uint4(x[0], x[1], x[2], x[3]);
            }
        }
#pragma unroll
        for (u32 k = 0; k < kParts; ++k) {
            const u32 c = k * 32u + lane;
            putRow(rows + (c / kParts) * kRlePitch + (c % kParts) * kVec, v[k]);
        }
    } else {
#pragma unroll 8
        for (u32 k = 0; k < 32; ++k) {
            const u32 pos = wbase + 32u * k + lane;
            rows[k * kRlePitch + lane] = pos < n ? in[pos] : Sym(0);
        }
    }
    __syncwarp();
    GroupRuns g{0u, 0u, 0u, 0u};
    const Sym* row = rows + lane * kRlePitch;
    u32 m = 0;
    if (sizeof(Sym) == 2) {
#pragma unroll
        for (u32 k = 0; k < 8; ++k) {
            const uint2 x = *reinterpret_cast<const uint2*>(row + 4 * k);
            m = __vmaxu2(m, __vmaxu2(x.x, x.y));
            // bit 15 / 31 of each: that half is not zero
            const u32 a = (((x.x & 0x7FFF7FFFu) + 0x7FFF7FFFu) | x.x) & 0x80008000u;
            const u32 b = (((x.y & 0x7FFF7FFFu) + 0x7FFF7FFFu) | x.y) & 0x80008000u;
            const u32 ab = (a >> 15) | (b >> 13);   // bits 0, 16 and 2, 18
            g.mask |= ((ab | (ab >> 15)) & 15u) << (4 * k);
        }
        m = max(m & 0xFFFFu, m >> 16);
    } else {
#pragma unroll
        for (u32 k = 0; k < 8; ++k) {
            const uint4 x = *reinterpret_cast<const uint4*>(row + 4 * k);
            m = max(max(m, max(x.x, x.y)), max(x.z, x.w));
            g.mask |= ((x.x ? 1u : 0u) | (x.y ? 2u : 0u) | (x.z ? 4u : 0u) | (x.w ? 8u : 0u)) << (4 * k);
        }
    }
    maxSym = __reduce_max_sync(0xffffffffu, m);
    const u32 gb = wbase + 32u * lane;
    g.cnt = __popc(g.mask);
    g.firstP1 = g.mask ? gb + u32(__ffs(g.mask)) : 0u;
    g.lastP1 = g.mask ? gb + 32u - u32(__clz(g.mask)) : 0u;
    return g;
}

// Exclusive max-scan of lastP1 over the warp's lanes (0 for lane 0).
__device__ __forceinline__ u32 warpExclusiveMax(u32 v) {
    const u32 lane = threadIdx.x & 31u;
#pragma unroll
    for (u32 d = 1; d < 32; d <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v = max(v, t);
    }
    const u32 e = __shfl_up_sync(0xffffffffu, v, 1);
    return lane ? e : 0u;
}

__device__ __forceinline__ RunSum shflUpRun(RunSum r, int delta) {
    RunSum t;
    t.cnt = __shfl_up_sync(0xffffffffu, r.cnt, delta);
    t.ext = __shfl_up_sync(0xffffffffu, r.ext, delta);
    t.firstP1 = __shfl_up_sync(0xffffffffu, r.firstP1, delta);
    t.lastP1 = __shfl_up_sync(0xffffffffu, r.lastP1, delta);
    return t;
}

__device__ __forceinline__ RunSum warpInclusiveRun(RunSum r) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        RunSum t = shflUpRun(r, o);
        if (lane >= o) r = runCombine(t, r);
    }
    return r;
}

// The start of a call: CTA s writes the stream index over its tiles (the
// prefix layout of the call's descriptors) and clears the stream's largest
// symbol; the first also the error flags.
__global__ void __launch_bounds__(256) k_encBegin(EncParams p) {
    const u32 i = blockIdx.x;
    if (i == 0 && threadIdx.x < 4) p.errors[threadIdx.x] = 0;
    if (threadIdx.x == 0) p.streamMax[i] = 0;
    const EncStreamDev& sd = p.streams[i];
    const u32 tiles = u32(ceilDiv(sd.n, kRleTile));
    for (u32 k = threadIdx.x; k < tiles; k += 256) p.tileStream[sd.tileOff + k] = i;
}

// ---------------------------------------------------------------------------
// Run-length encode (RunLength.cu:82-188 semantics: each nonzero symbol with
// the count of zeros before it; runs of 256+ zeros emit (0, 255) entries;
// trailing zeros dropped).
// Pass 1: per tile, the run summary (RLHuff) and the largest symbol, from
// the warps' group masks.
// ---------------------------------------------------------------------------
template <class Sym>
__global__ void __launch_bounds__(kRleThreads) k_summary(EncParams p) {
    __shared__ RunSum sRun[kRleWarps];
    __shared__ u32 sStream, sMaxSym;
    __shared__ __align__(16) Sym sRows[kRleWarps][32 * kRlePitch];
    const u32 tile = blockIdx.x;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) { sStream = streamOfTile(p, tile); sMaxSym = 0; }
    __syncthreads();
    const u32 s = sStream;
    const EncStreamDev sd = p.streams[s];
    const u32 n = sd.n;
    const Sym* in = reinterpret_cast<const Sym*>(sd.in);
    const u32 wbase = (tile - sd.tileOff) * kRleTile + warp * 1024u;
    u32 m;
    const GroupRuns g = loadGroups(in, wbase, n, sRows[warp], m);
    if (lane == 0 && m) atomicMax(&sMaxSym, m);
    if (sd.kind == KIND_RLHUFF) {
        // the warp's summary: (0, 255) entries of the gaps whose previous
        // nonzero lies in the warp
        const u32 prevW = warpExclusiveMax(g.lastP1);
        const u32 e = (g.mask && prevW) ? (g.firstP1 - prevW - 1u) / 256u : 0u;
        RunSum w;
        w.cnt = __reduce_add_sync(0xffffffffu, g.cnt);
        w.ext = __reduce_add_sync(0xffffffffu, e);
        w.firstP1 = __reduce_min_sync(0xffffffffu, g.mask ? g.firstP1 : 0xFFFFFFFFu);
        w.lastP1 = __reduce_max_sync(0xffffffffu, g.lastP1);
        if (!w.cnt) w.firstP1 = 0;
        if (lane == 0) sRun[warp] = w;
        __syncthreads();
        if (threadIdx.x == 0) {
            RunSum acc{0, 0, 0, 0};
#pragma unroll
            for (u32 k = 0; k < kRleWarps; ++k) acc = runCombine(acc, sRun[k]);
            p.tiles[tile] = acc;
        }
    } else {
        __syncthreads();
    }
    if (threadIdx.x == 0 && sMaxSym) atomicMax(p.streamMax + s, sMaxSym);
}

constexpr u32 kScanWarps = 8;   // warps (streams or tables) per CTA of the per-unit scans

// Pass 2: the scan of each stream's tile summaries, a warp per stream.
__device__ __forceinline__ void scanStream(const EncParams& p, u32 s) {
    const u32 lane = threadIdx.x & 31u;
    const EncStreamDev sd = p.streams[s];
    if (sd.kind != KIND_RLHUFF) {
        if (lane == 0) p.counts[s] = sd.n;
        return;
    }
    const u32 tiles = u32(ceilDiv(sd.n, kRleTile));
    const RunSum* T = p.tiles + sd.tileOff;
    TileStart* TS = p.tileStart + sd.tileOff;
    RunSum carry{0, 0, 0, 0};
    for (u32 base = 0; base < tiles; base += 32) {
        const u32 i = base + lane;
        const RunSum inc = warpInclusiveRun(i < tiles ? T[i] : RunSum{0, 0, 0, 0});
        RunSum ex = shflUpRun(inc, 1);
        if (lane == 0) ex = RunSum{0, 0, 0, 0};
        const RunSum E = runCombine(carry, ex);
        if (i < tiles) {
            TileStart ts;
            ts.prevP1 = E.cnt ? E.lastP1 : 0u;
            ts.out = E.cnt ? E.cnt + E.ext + (E.firstP1 - 1u) / 256u : 0u;
            TS[i] = ts;
        }
        RunSum last;
        last.cnt = __shfl_sync(0xffffffffu, inc.cnt, 31);
        last.ext = __shfl_sync(0xffffffffu, inc.ext, 31);
        last.firstP1 = __shfl_sync(0xffffffffu, inc.firstP1, 31);
        last.lastP1 = __shfl_sync(0xffffffffu, inc.lastP1, 31);
        carry = runCombine(carry, last);
    }
    if (lane == 0) p.counts[s] = carry.cnt ? carry.cnt + carry.ext + (carry.firstP1 - 1u) / 256u : 0u;
}

__global__ void __launch_bounds__(kScanWarps * 32) k_scan(EncParams p) {
    const u32 s = blockIdx.x * kScanWarps + (threadIdx.x >> 5);
    if (s < p.S) scanStream(p, s);
}

// The same with a CTA per stream, for long ones: a warp takes 0.7 us for 32
// tiles, one step after the other.  63 streams of up to 1024 tiles (three 256^3
// volumes): 5 us, and 6 for the plan, where two streams per warp of one CTA
// took 38 with the plan; a 512^3 volume's encode 1729 -> 1531 us, one stream of
// 64 million symbols 1608 -> 934.
constexpr u32 kScanThreads = 512;

__global__ void __launch_bounds__(kScanThreads) k_scanWide(EncParams p) {
    constexpr u32 kWarps = kScanThreads / 32;
    __shared__ RunSum sWarp[kWarps];
    const u32 s = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const EncStreamDev sd = p.streams[s];
    if (sd.kind != KIND_RLHUFF) {   // block-uniform
        if (threadIdx.x == 0) p.counts[s] = sd.n;
        return;
    }
    const u32 tiles = u32(ceilDiv(sd.n, kRleTile));
    const RunSum* T = p.tiles + sd.tileOff;
    TileStart* TS = p.tileStart + sd.tileOff;
    const RunSum none{0, 0, 0, 0};
    RunSum carry = none;
    RunSum next = threadIdx.x < tiles ? T[threadIdx.x] : none;
    for (u32 base = 0; base < tiles; base += kScanThreads) {
        const u32 i = base + threadIdx.x;
        const RunSum inc = warpInclusiveRun(next);
        next = i + kScanThreads < tiles ? T[i + kScanThreads] : none;   // in flight over this step
        RunSum ex = shflUpRun(inc, 1);
        if (lane == 0) ex = none;
        if (lane == 31) sWarp[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const RunSum w = warpInclusiveRun(lane < kWarps ? sWarp[lane] : none);
            if (lane < kWarps) sWarp[lane] = w;
        }
        __syncthreads();
        const RunSum E = runCombine(carry, warp ? runCombine(sWarp[warp - 1], ex) : ex);
        carry = runCombine(carry, sWarp[kWarps - 1]);
        if (i < tiles) {
            TileStart ts;
            ts.prevP1 = E.cnt ? E.lastP1 : 0u;
            ts.out = E.cnt ? E.cnt + E.ext + (E.firstP1 - 1u) / 256u : 0u;
            TS[i] = ts;
        }
        __syncthreads();   // sWarp is read
    }
    if (threadIdx.x == 0) p.counts[s] = carry.cnt ? carry.cnt + carry.ext + (carry.firstP1 - 1u) / 256u : 0u;
}

// Which of them.  Up to 64 streams: one CTA scans them, a warp for one or two
// streams, and makes the plan in the same launch, as long as its warps take at
// most four steps (0.7 us each); a scan of its own costs a launch, 2.5 us (an
// image's nine streams of 96 tiles: 476 us there and back with it, 469
// without).  More streams: where the longest has more than 64 tiles, unless
// that many CTAs would take longer than its warp (2 us per 1184).
constexpr u32 kScanPlanStreams = 64;
static bool wideTileScan(u32 streams, u32 tiles) {
    if (streams <= kScanPlanStreams) return ceilDiv(streams, 32) * ceilDiv(tiles, 32) > 4;
    return tiles > 64 && streams / 16 <= tiles;
}

// Table builders by leaf count (k_leafTiers sorts the tables, k_tableBuild
// builds them): the heap merge is a latency-bound chain on one warp, so a
// smaller table gets a smaller CTA and heap and more of them share an SM.
//   tier 0: up to 256 leaves, a warp, 5 KB of heap (21 per SM, by registers;
//           the grid has 32, those past the first 21 start as others end)
//   tier 1: up to 1024 leaves, 64 threads, 20 KB (10 per SM)
//   tier 2: up to 2048 leaves, 128 threads, 41 KB (5 per SM)
//   tier 3: more, 512 threads, the full heap (one per SM)
constexpr u32 kTinyLeaves = 256;
constexpr u32 kSmallLeaves = 1024;
constexpr u32 kBuildSplitLeaves = 2048;
constexpr u32 kBuildEach = 0xFFFFFFFFu;                  // buildTier: one table per CTA
constexpr u32 kTierMinTables = 64;                       // calls of more tables use the tiers

// Pass 3: histogram / builder / header offsets of every table, sized from
// the largest symbol of its stream.  A symbol outside the instance's
// 2^log2Max range fails the call (HuffmanTable.cu:411-419).  CTA b plans the
// kPlanChunk tables of chunk b, four consecutive per thread with their loads
// in flight together: their offsets within the chunk, and the chunk's sums
// (planPart); with more than one chunk, k_histPlanCarry adds the sums of the
// chunks before each one - every CTA's work independent, so a call of 10^5
// tables takes two short launches instead of a loop on one SM.
constexpr u32 kPlanPer = 4;
static_assert(kPlanChunk == 1024 * kPlanPer, "a plan chunk is one 1024-thread CTA's tables");

constexpr u32 kPlanSums = 5;   // bins, leaves, header words, coding blocks, runs

// The call's totals from the offsets' grand sums c[0..4] (bins, leaves,
// header words, coding blocks, runs), and the capacity check.
__device__ __forceinline__ void planTotals(const EncParams& p, const unsigned long long (&c)[kPlanSums]) {
    p.totals[2] = c[3];
    p.totals[3] = c[4];
    for (u32 k = 4; k < 8; ++k) p.totals[k] = 0;   // the tier lists' counts (k_leafTiers)
    p.totals[1] = c[0];
    if (c[0] > p.capHist || c[1] > p.capLeaves || c[2] > p.capHdr) atomicOr(p.errors, DEV_ERR_TABLE_CAPACITY);
}

__device__ __forceinline__ void histPlanChunk(const EncParams& p, u32* scratch) {
    const u32 t0 = blockIdx.x * kPlanChunk + threadIdx.x * kPlanPer;
    // per table: bins, leaves, header words, blocks, runs
    u32 v[kPlanPer][kPlanSums];
    TableMeta m[kPlanPer];
#pragma unroll
    for (u32 j = 0; j < kPlanPer; ++j) {
        const u32 t = t0 + j;
        m[j] = TableMeta{};
        u32 hs = 0, ls = 0, ws = 0;
        if (t < p.T) {
            const EncTableDev td = p.tables[t];
            const u32 smax = p.streamMax[td.stream];
            const u32 count = p.counts[td.stream];
            if (td.which == 0 && smax >= p.bins) atomicOr(p.errors, DEV_ERR_SYMBOL_RANGE);
            hs = td.which ? min(256u, p.bins) : min(smax, p.bins - 1u) + 1u;
            ls = min(hs, count + 1u);
            ws = headerWordsFor(ls, p.log2Max);
            m[j].count = count;
            m[j].histSize = hs;
            m[j].blocks = blocksOf(count, p.cbLog);
        }
        v[j][0] = hs;
        v[j][1] = ls;
        v[j][2] = ws;
        v[j][3] = m[j].blocks;
        v[j][4] = blocksOf(m[j].blocks, kRunLog - p.cbLog);
    }
    u32 sum[kPlanSums], ex[kPlanSums], tot[kPlanSums];
#pragma unroll
    for (u32 k = 0; k < kPlanSums; ++k) {
        sum[k] = 0;
#pragma unroll
        for (u32 j = 0; j < kPlanPer; ++j) sum[k] += v[j][k];
    }
    blockExclusiveSumN<1024, kPlanSums>(sum, ex, tot, scratch);
    unsigned long long at[kPlanSums];
#pragma unroll
    for (u32 k = 0; k < kPlanSums; ++k) at[k] = ex[k];
#pragma unroll
    for (u32 j = 0; j < kPlanPer; ++j) {
        const u32 t = t0 + j;
        if (t < p.T) {
            m[j].histOff = at[0];
            m[j].leafOff = at[1];
            m[j].hdrOff = at[2];
            m[j].runOff = u32(at[4]);
            p.meta[t] = m[j];
        }
#pragma unroll
        for (u32 k = 0; k < kPlanSums; ++k) at[k] += v[j][k];
    }
    if (threadIdx.x == 0) {
        if (gridDim.x == 1) {
            unsigned long long c[kPlanSums];
#pragma unroll
            for (u32 k = 0; k < kPlanSums; ++k) c[k] = tot[k];
            planTotals(p, c);
        } else {
#pragma unroll
            for (u32 k = 0; k < kPlanSums; ++k) p.planPart[u64(blockIdx.x) * 8 + k] = tot[k];
        }
    }
}

__global__ void __launch_bounds__(1024) k_histPlan(EncParams p) {
    __shared__ u32 scratch[33 * kPlanSums];
    histPlanChunk(p, scratch);
}

// Passes 2 and 3 of a call of few and short streams in one CTA (wideTileScan).

__global__ void __launch_bounds__(1024) k_scanPlan(EncParams p) {
    __shared__ u32 scratch[33 * kPlanSums];
    for (u32 s = threadIdx.x >> 5; s < p.S; s += 32) scanStream(p, s);
    __syncthreads();   // the CTA's counts
    histPlanChunk(p, scratch);
}

// Chunk b = blockIdx.x + 1 of a plan of more than one chunk: the sums of
// chunks 0 .. b-1 (a warp over planPart) added to its tables' offsets; the
// last chunk's CTA forms the call's totals.
__global__ void __launch_bounds__(1024) k_histPlanCarry(EncParams p) {
    __shared__ unsigned long long sC[kPlanSums];
    const u32 b = blockIdx.x + 1;
    if (threadIdx.x < 32) {
        unsigned long long c[kPlanSums] = {0, 0, 0, 0, 0};
        for (u32 i = threadIdx.x; i < b; i += 32)
#pragma unroll
            for (u32 k = 0; k < kPlanSums; ++k) c[k] += p.planPart[u64(i) * 8 + k];
#pragma unroll
        for (u32 k = 0; k < kPlanSums; ++k)
#pragma unroll
            for (u32 o = 16; o > 0; o >>= 1) c[k] += __shfl_xor_sync(0xffffffffu, c[k], o);
        if (threadIdx.x == 0)
#pragma unroll
            for (u32 k = 0; k < kPlanSums; ++k) sC[k] = c[k];
    }
    __syncthreads();
    const u32 t0 = b * kPlanChunk + threadIdx.x * kPlanPer;
#pragma unroll
    for (u32 j = 0; j < kPlanPer; ++j) {
        const u32 t = t0 + j;
        if (t < p.T) {
            TableMeta& m = p.meta[t];
            m.histOff += sC[0];
            m.leafOff += sC[1];
            m.hdrOff += sC[2];
            m.runOff += u32(sC[4]);
        }
    }
    if (b == gridDim.x && threadIdx.x == 0) {
        unsigned long long c[kPlanSums];
#pragma unroll
        for (u32 k = 0; k < kPlanSums; ++k) c[k] = sC[k] + p.planPart[u64(b) * 8 + k];
        planTotals(p, c);
    }
}

// After the plan: the call's histograms zeroed, and the runs of coding blocks
// in use (those holding symbols after the run-length step) listed table by
// table - warp t writes t over its runs from meta.runOff.  The block-level
// kernels walk this list instead of every block a table could have.
__global__ void __launch_bounds__(256) k_planFill(EncParams p) {
    if (warpFailed(p)) return;
    const u32 thread = blockIdx.x * 256u + threadIdx.x, threads = gridDim.x * 256u, lane = threadIdx.x & 31u;
    const u64 total = p.totals[1];
    for (u64 i = thread; i < total; i += threads) p.hist[i] = 0;
    for (u32 t = thread >> 5; t < p.T; t += threads >> 5) {
        const u32 runs = blocksOf(p.meta[t].blocks, kRunLog - p.cbLog), off = p.meta[t].runOff;
        for (u32 k = lane; k < runs; k += 32) p.runTable[off + k] = t;
    }
}

// The leaf count of every table (the nonzero bins of its histogram; a warp
// per table) and the tier list it goes on (tierTables, counts totals[4..7]).
// A table whose histogram is empty (its stream has no symbols) goes on tier
// 0, the only builder that may then give it a leaf.
__global__ void __launch_bounds__(256) k_leafTiers(EncParams p) {
    if (warpFailed(p)) return;
    const u32 t = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (t >= p.T) return;
    const TableMeta m = p.meta[t];
    const u32* h = p.hist + m.histOff;
    u32 c = 0;
    for (u32 b = lane; b < m.histSize; b += 32) c += h[b] ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) {
        const u32 tier = c <= kTinyLeaves ? 0u : c <= kSmallLeaves ? 1u : c <= kBuildSplitLeaves ? 2u : 3u;
        const u32 pos = u32(atomicAdd(reinterpret_cast<unsigned long long*>(p.totals + 4 + tier), 1ull));
        p.tierTables[u64(tier) * p.T + pos] = t;
    }
}

// Pass 4: compact symbols + zero counts (RLHuff) and both histograms, or the
// plain histogram of a Huff stream.  Symbol bins below kWriteSymBins are
// counted in shared memory.
//
// RLHuff: a tile's run-length entries form one contiguous range of the
// stream's compact arrays.  Group k of a warp starts its entries after the
// entries of the tile's groups before it (a warp scan of the groups' counts
// plus their (0, 255) entries, and a block combine over the warps); its lane
// then walks its nonzeros, the distance to the one before being the zero
// count.  Entries are staged in shared memory at their positions within the
// tile, shifted so that 16-byte chunks there are 16-byte chunks of the compact
// arrays, and copied out by them.  The eight most frequent keys of each
// histogram (zero counts 0..7, symbols 1..8) are counted in the lane's
// registers on the way, the others with shared-memory atomics.  The stage
// (dynamic shared memory) holds an entry per symbol and eight more for 16-bit
// symbols, half as many for 32-bit ones.  A tile of more - all nonzero after a
// run of 2304 zeros, one nonzero after 526336, 32-bit symbols mostly nonzero -
// writes its entries directly.  Bound: instruction issue; walking a group's
// nonzeros on its lane instead of a group's lanes together took three 256^3 streams'
// highpass bands (50 million symbols, 26 million entries) from 191 to 123 us.
constexpr u32 kWriteSymBins = 768;   // symbol bins counted in shared memory by k_write

// Counts of the symbols above them.  Where these repeat - two of the first
// symbols of a warp's 32 groups are like others - atomics on global memory
// would queue at a few words: 8 million symbols of value 2000 took 5670 us.  A
// word of shared memory then holds a count (a tile has at most kRleTile) and
// the upper bits of the symbol that took the slot of its low byte first; others
// of that byte go to global memory (215 us; 400 with 4096 bins in shared
// memory).  Where they do not, every one goes there directly: a slot's look and
// claim hold up a warp for some 150 cycles, and the write of the lowpass
// streams of three 256^3 volumes, on the batch's longest chain, took 12.4 us
// instead of 7.5.  Bins and slots are 4 KB together, twelve tiles per SM; with
// 5 KB, eleven, their highpass streams took 125 us instead of 121.
constexpr u32 kHotSlots = 256;
static_assert(kRleTile < 65536u && kWriteSymBins >= kHotSlots, "16-bit counts; a symbol's upper bits are not 0");

__device__ __forceinline__ void countLarge(u32* hot, u32* global, u32 sym) {
    u32* slot = hot + (sym & (kHotSlots - 1u));
    const u32 tag = sym / kHotSlots << 16;   // symbols have at most 24 bits
    u32 v = *reinterpret_cast<volatile const u32*>(slot);
    if (v == 0 && (v = atomicCAS(slot, 0u, tag | 1u)) == 0) return;
    if ((v & 0xFFFF0000u) == tag) atomicAdd(slot, 1u);
    else atomicAdd(global + sym, 1u);
}

template <class Sym>
constexpr u32 writeStage() { return sizeof(Sym) == 2 ? kRleTile + kRleTile / 256u : kRleTile / 2u; }
template <class Sym>
constexpr u32 writeVec() { return 16 / sizeof(Sym); }   // elements of a 16-byte chunk
// Staged symbols and zero counts (with room for the shift), and the warps' rows.
template <class Sym>
constexpr size_t writeSmem() {
    return sizeof(Sym) * (2 * (size_t(writeStage<Sym>()) + writeVec<Sym>()) + size_t(kRleWarps) * 32 * kRlePitch);
}

template <class Sym>
__global__ void __launch_bounds__(kRleThreads) k_write(EncParams p) {
    constexpr u32 kStage = writeStage<Sym>(), kVec = writeVec<Sym>();
    extern __shared__ __align__(16) unsigned char dynWrite[];
    __shared__ u32 sLast[kRleWarps], sEnt[kRleWarps];
    __shared__ u32 hSym[kWriteSymBins];
    __shared__ u32 hZc[256];
    __shared__ u32 hHot[kHotSlots];
    Sym* const sComp = reinterpret_cast<Sym*>(dynWrite);
    Sym* const sZcs = sComp + kStage + kVec;
    __shared__ u32 sStream;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    Sym* const rows = sZcs + kStage + kVec + warp * (32 * kRlePitch);
    if (threadIdx.x == 0) sStream = streamOfTile(p, blockIdx.x);
    if (blockFailed(p)) return;   // synchronizes (sStream visible)
    const u32 tile = blockIdx.x;
    const u32 s = sStream;
    const EncStreamDev sd = p.streams[s];
    const u32 n = sd.n;
    const TableMeta mS = p.meta[sd.tableFirst];
    const u32 smemBins = min(mS.histSize, kWriteSymBins);
    for (u32 i = threadIdx.x; i < smemBins; i += kRleThreads) hSym[i] = 0;
    for (u32 i = threadIdx.x; i < 256u; i += kRleThreads) hZc[i] = 0;
    const bool large = mS.histSize > kWriteSymBins;   // block-uniform
    if (large)
        for (u32 i = threadIdx.x; i < kHotSlots; i += kRleThreads) hHot[i] = 0;
    const Sym* in = reinterpret_cast<const Sym*>(sd.in);
    const u32 wbase = (tile - sd.tileOff) * kRleTile + warp * 1024u;
    u32 mUnused;
    const GroupRuns g = loadGroups(in, wbase, n, rows, mUnused);
    u32* gSym = p.hist + mS.histOff;
    bool slots = false;   // warp-uniform
    if (large) {
        const u32 x = g.mask ? u32(rows[lane * kRlePitch + u32(__ffs(int(g.mask))) - 1u]) : 0u;
        const bool is = x >= kWriteSymBins;
        const u32 peers = __match_any_sync(0xffffffffu, x);
        const u32 of = __popc(__ballot_sync(0xffffffffu, is));
        const u32 distinct = __popc(__ballot_sync(0xffffffffu, is && lane == u32(__ffs(int(peers))) - 1u));
        slots = of >= distinct + 2u;
    }
    auto addLarge = [&](u32 sym) {
        if (slots) countLarge(hHot, gSym, sym);
        else atomicAdd(gSym + sym, 1u);
    };
    auto flush = [&] {
        for (u32 i = threadIdx.x; i < smemBins; i += kRleThreads)
            if (hSym[i]) atomicAdd(gSym + i, hSym[i]);
        if (large)
            for (u32 i = threadIdx.x; i < kHotSlots; i += kRleThreads)
                if (const u32 v = hHot[i]) atomicAdd(gSym + (v >> 16) * kHotSlots + i, v & 0xFFFFu);
    };
    if (sd.kind != KIND_RLHUFF) {
        __syncthreads();
        for (u32 k = 0; k < 32; ++k) {
            if (wbase + 32u * k + lane >= n) break;
            const u32 x = rows[k * kRlePitch + lane];
            if (x < smemBins) atomicAdd(hSym + x, 1u);
            else if (x < mS.histSize) addLarge(x);
        }
        __syncthreads();
        flush();
        return;
    }
    const TableMeta mZ = p.meta[sd.tableFirst + 1];
    u32* gZc = p.hist + mZ.histOff;
    // the nonzero before each group: in the warp, in the warps before, or
    // before the tile
    const u32 lastW = __reduce_max_sync(0xffffffffu, g.lastP1);
    if (lane == 0) sLast[warp] = lastW;
    __syncthreads();   // also orders the histogram zeroing
    u32 lastBefore = 0;
#pragma unroll
    for (u32 w = 0; w < kRleWarps; ++w)
        if (w < warp) lastBefore = max(lastBefore, sLast[w]);
    const TileStart ts = p.tileStart[tile];
    u32 prev = max(warpExclusiveMax(g.lastP1), lastBefore);
    if (!prev) prev = ts.prevP1;
    const u32 e = g.mask ? (g.firstP1 - prev - 1u) / 256u : 0u;   // (0, 255) entries before the group
    const u32 ent = g.cnt + e;
    const u32 entIncl = warpInclusiveSum(ent);
    if (lane == 31) sEnt[warp] = entIncl;
    __syncthreads();
    u32 warpOut = 0, entries = 0;
#pragma unroll
    for (u32 w = 0; w < kRleWarps; ++w) {
        const u32 x = sEnt[w];
        if (w < warp) warpOut += x;
        entries += x;
    }
    const u64 first = sd.compactOff + ts.out;          // the tile's first entry in the compact arrays
    Sym* comp = reinterpret_cast<Sym*>(p.compact) + first;
    Sym* zcs = reinterpret_cast<Sym*>(p.zc) + first;
    const u32 shift = u32(first) & (kVec - 1u);        // both arrays are 16-byte aligned
    const bool staged = entries <= kStage;             // block-uniform
    const bool fast = mZ.histSize == 256u && smemBins > 8u;
    // the eight most frequent keys of each histogram in per-lane 8-bit
    // counters, four keys per register (at most 32 entries per lane)
    u32 z03 = 0, z47 = 0, s03 = 0, s47 = 0;
    bool rangeErr = false;
    auto walk = [&](Sym* oc, Sym* oz) {
        const u32 at = warpOut + entIncl - ent;        // the group's first entry in the tile
        // (0, 255) entries, by the whole warp
        for (u32 lanes = __ballot_sync(0xffffffffu, e != 0u); lanes; lanes &= lanes - 1u) {
            const int j = __ffs(int(lanes)) - 1;
            const u32 ej = __shfl_sync(0xffffffffu, e, j), aj = __shfl_sync(0xffffffffu, at, j);
            for (u32 t = lane; t < ej; t += 32) {
                oc[aj + t] = Sym(0);
                oz[aj + t] = Sym(255);
            }
        }
        if (e) {
            atomicAdd(hSym, e);                        // smemBins >= 1
            if (255u < mZ.histSize) atomicAdd(hZc + 255, e);
            else rangeErr = true;
        }
        const Sym* row = rows + lane * kRlePitch;
        const u32 gb1 = wbase + 32u * lane + 1u;
        u32 o = at + e, before = prev;
        for (u32 mask = g.mask; mask; mask &= mask - 1u) {
            const u32 b = u32(__ffs(int(mask))) - 1u;
            const u32 sym = row[b], q = gb1 + b;
            const u32 zc = (q - before - 1u) & 255u;
            before = q;
            oc[o] = Sym(sym);
            oz[o] = Sym(zc);
            ++o;
            if (fast) {
                const u32 zi = 1u << ((zc & 3u) << 3);
                if (zc < 4u) z03 += zi;
                else if (zc < 8u) z47 += zi;
                else atomicAdd(hZc + zc, 1u);
                const u32 k = sym - 1u;                // keys 1..8 -> 0..7
                const u32 si = 1u << ((k & 3u) << 3);
                if (k < 4u) s03 += si;
                else if (k < 8u) s47 += si;
                else if (sym < smemBins) atomicAdd(hSym + sym, 1u);
                else if (sym < mS.histSize) addLarge(sym);
            } else {
                if (sym < smemBins) atomicAdd(hSym + sym, 1u);
                else if (sym < mS.histSize) addLarge(sym);
                if (zc < mZ.histSize) atomicAdd(hZc + zc, 1u);
                else rangeErr = true;
            }
        }
    };
    if (staged) {
        walk(sComp + shift, sZcs + shift);
        __syncthreads();
        // chunk c of the stage: elements [c kVec, (c + 1) kVec) from `first - shift`
        const u32 end = shift + entries, chunks = (end + kVec - 1u) / kVec;
        Sym* const compA = comp - shift;
        Sym* const zcsA = zcs - shift;
        for (u32 c = threadIdx.x; c < chunks; c += kRleThreads) {
            const u32 lo = c * kVec;
            if (lo >= shift && lo + kVec <= end) {
                *reinterpret_cast<uint4*>(compA + lo) = *reinterpret_cast<const uint4*>(sComp + lo);
                *reinterpret_cast<uint4*>(zcsA + lo) = *reinterpret_cast<const uint4*>(sZcs + lo);
            } else {
                for (u32 i = max(lo, shift); i < min(lo + kVec, end); ++i) {
                    compA[i] = sComp[i];
                    zcsA[i] = sZcs[i];
                }
            }
        }
    } else {
        walk(comp, zcs);
    }
    if (fast) {
        // widen to 16-bit fields (keys k, k + 2 per register) and sum over the warp
        u32 a[8] = {z03 & 0x00FF00FFu, (z03 >> 8) & 0x00FF00FFu, z47 & 0x00FF00FFu, (z47 >> 8) & 0x00FF00FFu,
                    s03 & 0x00FF00FFu, (s03 >> 8) & 0x00FF00FFu, s47 & 0x00FF00FFu, (s47 >> 8) & 0x00FF00FFu};
#pragma unroll
        for (u32 o = 16; o > 0; o >>= 1)
#pragma unroll
            for (u32 i = 0; i < 8; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
        if (lane == 0) {
            // a[0]: keys 0, 2; a[1]: 1, 3; a[2]: 4, 6; a[3]: 5, 7 (zero counts); a[4..7] the same for symbols - 1
            const u32 key[4] = {0u, 1u, 4u, 5u};
#pragma unroll
            for (u32 i = 0; i < 4; ++i) {
                const u32 zl = a[i] & 0xFFFFu, zh = a[i] >> 16, sl = a[4 + i] & 0xFFFFu, sh = a[4 + i] >> 16;
                if (zl) atomicAdd(hZc + key[i], zl);
                if (zh) atomicAdd(hZc + key[i] + 2u, zh);
                if (sl) atomicAdd(hSym + key[i] + 1u, sl);
                if (sh) atomicAdd(hSym + key[i] + 3u, sh);
            }
        }
    }
    if (rangeErr) atomicOr(p.errors, DEV_ERR_SYMBOL_RANGE);
    __syncthreads();
    flush();
    for (u32 i = threadIdx.x; i < min(mZ.histSize, 256u); i += kRleThreads)
        if (hZc[i]) atomicAdd(gZc + i, hZc[i]);
}

// ---------------------------------------------------------------------------
// Table construction: one block per table, all tables of the call at once.
// Leaf gathering, depths, the sort (an exact warp-parallel replay of
// std::sort), canonical codes and serialization are block parallel; the heap
// merge runs on one warp in shared memory (table_build.cuh).  Tables with
// more leaves than the shared-memory builder holds run sequentially on
// global memory (huffman_build.cuh).
// ---------------------------------------------------------------------------
constexpr u32 kBuildThreads = 256, kMidThreads = 128;
// the full builder, a CTA of its own on an SM: the merge is one warp's, the
// sort's deep rounds and the walks over leaves take all
constexpr u32 kBigThreads = 512;

__device__ __forceinline__ void putBits(u32* words, u32 pos, u32 value, u32 count) {
    // MSB-first, count <= 32, words pre-zeroed; atomics because neighbouring
    // fields written by other threads share words.
    if (count == 0) return;
    value &= count == 32 ? 0xffffffffu : ((1u << count) - 1u);
    const u32 w = pos >> 5, b = pos & 31u;
    const int shift = int(32 - b) - int(count);
    if (shift >= 0) {
        atomicOr(words + w, value << shift);
    } else {
        atomicOr(words + w, value >> (-shift));
        atomicOr(words + w + 1, value << (32 + shift));
    }
}

// Builds table t (all kThreads threads of the block; returns uniformly).
// Tables of up to kCap leaves are built in shared memory.  kWide (alphabets of
// more than kWideBins): the leaves are gathered a range of bins per warp.  A
// range per thread, which small alphabets keep, reads a cache line per lane,
// and the full builder's heap leaves 28 KB of L1: seven streams over 300000
// bins 690 us, 201 so; over 60000 bins 284 and 139; a hundred of them, by one
// warp with a load in flight, 622 and 446.  The merge loop's time changes by 1
// to 5% with the code around it, which is why the two are compiled apart.
constexpr u32 kWideBins = 1u << 14;

template <u32 kThreads, u32 kCap, bool kWide>
__device__ __forceinline__ void buildTable(const EncParams& p, u32 t) {
    constexpr int kSegs = int(kCap / 17u) + 1;   // the sort's queue: segments longer than 16 keys
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ u32 sScan[40];
    __shared__ u32 sMax, sMaxLen, sAllEmpty;
    __shared__ u32 lenCount[32], firstIndex[33], firstCode[33];
    __shared__ tb::Seg sSegA[kSegs], sSegB[kSegs];
    __shared__ int sSegCount[4];
    if (threadIdx.x == 0) { sMax = 0; sAllEmpty = 1; }
    if (blockFailed(p)) return;
    const EncTableDev td = p.tables[t];
    const EncStreamDev es = p.streams[td.stream];
    TableMeta meta = p.meta[t];
    const u32 count = meta.count;
    const u32* hist = p.hist + meta.histOff;
    const bool isZc = es.kind == KIND_RLHUFF && td.which == 1;

    // 1. largest present symbol
    if (es.kind == KIND_RLHUFF)
        for (u32 s = es.groupFirst + threadIdx.x; s < es.groupFirst + es.groupSize; s += kThreads)
            if (p.counts[s]) atomicAnd(&sAllEmpty, 0u);
    if (kThreads > 32 && !kWide) {
        u32 localMax = 0;
        bool any = false;
        for (u32 b = threadIdx.x; b < meta.histSize; b += kThreads)
            if (hist[b]) { localMax = b; any = true; }
        if (any) atomicMax(&sMax, localMax);
    }
    __syncthreads();
    u32 symbolMax = count ? sMax : 0u;   // kThreads == 32, kWide: with the leaves, below
    // Histogram.cu:117-121: with every stream of the reference call empty the
    // reference builds its tables from stale arena words; for zero-count table
    // i that word is the low half of a device pointer when 2+2i < S (nonzero),
    // else the all-zero run-length scan output.
    const bool quirkLeaf = isZc && sAllEmpty && (2u + 2u * (td.stream - es.groupFirst) < es.groupSize);
    // 2. leaves in symbol order: straight into the shared-memory heap
    //    (1-based, see heap_merge.cuh) when the table fits
    u32* leafSym = p.leafSymWork + meta.leafOff;
    u64* heapG = p.leafWork + meta.leafOff;
    using At = hm::Layout<kCap>;
    u32* heapP = reinterpret_cast<u32*>(dyn);
    u32* heapI = reinterpret_cast<u32*>(dyn + At::kIds);
    const u16* parentS = reinterpret_cast<const u16*>(dyn + At::kParents);
    u32* orderS = heapP;   // takes the probabilities' place after the merge, sorted the ids'
    const u32 smemLeaves = count < hm::kInf - 1u ? kCap : 0u;
    u32 L;
    if (quirkLeaf) {
        L = 1;
        if (L < p.buildLo || L > p.buildHi) return;   // uniform: the other build launch has it
        if (threadIdx.x == 0) {
            leafSym[0] = 0;
            if (L > smemLeaves) heapG[0] = u64(1) << 32;
        }
    } else if (count == 0) {
        L = 0;
        if (L < p.buildLo || L > p.buildHi) return;
    } else if constexpr (kWide) {
        // large alphabets: a range of bins per warp, 32 bins at a time and
        // kFlight of them in flight, counted, then written behind the warps
        // before
        constexpr u32 kWarps = kThreads / 32, kFlight = 8;
        const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
        const u32 per = (meta.histSize + 32u * kWarps - 1u) / (32u * kWarps) * 32u;
        const u32 b0 = min(meta.histSize, warp * per), b1 = min(meta.histSize, b0 + per);
        u32 c = 0, top = 0;
        for (u32 b = b0; b < b1; b += 32u * kFlight) {
            u32 h[kFlight];
#pragma unroll
            for (u32 q = 0; q < kFlight; ++q) h[q] = b + 32u * q + lane < b1 ? hist[b + 32u * q + lane] : 0u;
#pragma unroll
            for (u32 q = 0; q < kFlight; ++q) {
                const u32 m = __ballot_sync(0xffffffffu, h[q] != 0);
                c += __popc(m);
                if (m) top = b + 32u * q + 31u - u32(__clz(int(m)));
            }
        }
        if (lane == 0) {
            sScan[warp] = c;
            if (c) atomicMax(&sMax, top);
        }
        __syncthreads();
        u32 off = 0;
        L = 0;
#pragma unroll
        for (u32 w = 0; w < kWarps; ++w) {
            if (w < warp) off += sScan[w];
            L += sScan[w];
        }
        symbolMax = sMax;
        if (L < p.buildLo || L > p.buildHi) return;
        const bool toSmem = L <= smemLeaves;
        const bool quirk65535 = p.symBytes == 2 && p.bins == 65536u && symbolMax == 65535u;
        for (u32 b = b0; b < b1; b += 32u * kFlight) {
            u32 hs[kFlight];
#pragma unroll
            for (u32 q = 0; q < kFlight; ++q) hs[q] = b + 32u * q + lane < b1 ? hist[b + 32u * q + lane] : 0u;
#pragma unroll
            for (u32 q = 0; q < kFlight; ++q) {
                const u32 sym = b + 32u * q + lane, m = __ballot_sync(0xffffffffu, hs[q] != 0);
                if (hs[q]) {
                    u32 h = hs[q];
                    if (quirk65535 && sym == 65535u) h += count & 1u;   // HistogramKernels.cui:165,200 padding word
                    const u32 to = off + __popc(m & below);
                    leafSym[to] = sym;
                    if (toSmem) {
                        heapP[to + 1] = h;
                        heapI[to + 1] = 2u * to;
                    } else {
                        heapG[to] = (u64(h) << 32) | to;
                    }
                }
                off += __popc(m);
            }
        }
    } else if (kThreads == 32) {
        // one warp: largest symbol and leaves in one pass, 32 bins at a time
        const u32 below = (1u << threadIdx.x) - 1u;
        L = 0;
        u32 next = threadIdx.x < meta.histSize ? hist[threadIdx.x] : 0u;
        for (u32 base = 0; base < meta.histSize; base += 32) {
            const u32 b = base + threadIdx.x;
            u32 h = next;
            next = b + 32u < meta.histSize ? hist[b + 32u] : 0u;   // in flight over this step's stores
            const u32 m = __ballot_sync(0xffffffffu, h != 0);
            if (h) {
                const u32 off = L + __popc(m & below);
                if (p.symBytes == 2 && p.bins == 65536u && b == 65535u) h += count & 1u;   // as below
                leafSym[off] = b;
                if (!smemLeaves) {
                    heapG[off] = (u64(h) << 32) | off;
                } else if (off < kCap) {
                    heapP[off + 1] = h;
                    heapI[off + 1] = 2u * off;
                }
            }
            if (m) symbolMax = base + 31u - u32(__clz(int(m)));
            L += __popc(m);
        }
        if (L < p.buildLo || L > p.buildHi) return;   // at most kCap leaves (k_leafTiers)
    } else {
        const u32 nb = symbolMax + 1;
        const u32 per = (nb + kThreads - 1) / kThreads;
        const u32 b0 = threadIdx.x * per, b1 = min(nb, b0 + per);
        u32 c = 0;
        for (u32 b = b0; b < b1; ++b) c += hist[b] ? 1u : 0u;
        u32 tot;
        u32 off = blockExclusiveSum<kThreads>(c, sScan, &tot);
        L = tot;
        if (L < p.buildLo || L > p.buildHi) return;
        const bool toSmem = L <= smemLeaves;
        const bool quirk65535 = p.symBytes == 2 && p.bins == 65536u && symbolMax == 65535u;
        for (u32 b = b0; b < b1; ++b) {
            u32 h = hist[b];
            if (h) {
                if (quirk65535 && b == 65535u) h += count & 1u;   // HistogramKernels.cui:165,200 padding word
                leafSym[off] = b;
                if (toSmem) {
                    heapP[off + 1] = h;
                    heapI[off + 1] = 2u * off;
                } else {
                    heapG[off] = (u64(h) << 32) | off;
                }
                ++off;
            }
        }
    }
    const bool inSmem = L <= smemLeaves;
    u32* order = inSmem ? orderS : p.orderWork + meta.leafOff;
    if (threadIdx.x == 0) sMaxLen = 0;
    __syncthreads();
    // 3. tree, depths and sort
    if (inSmem) {
        if (L >= 2) tb::blockBuildTree<kCap>(dyn, L);
        const u32 root = L >= 2 ? 2 * L - 2 : 0;
        u32 localMax = 0;
        for (u32 i = threadIdx.x; i < L; i += kThreads) {
            u32 d = 0, node = i;
            while (node != root && d < 32) { node = parentS[node]; ++d; }
            order[i] = (min(d, 31u) << 27) | i;
            localMax = max(localMax, d);
        }
        if (localMax) atomicMax(&sMaxLen, localMax);
        __syncthreads();
        if (sMaxLen <= 31) {
            // the ids' and the tails' places
            u16* lList = reinterpret_cast<u16*>(heapI);
            u16* rList = lList + kCap;
            u32* seg = reinterpret_cast<u32*>(dyn + At::kTails);
            tb::blockIntrosort<kThreads>(orderS, int(L), lList, rList, seg, sSegA, sSegB, sSegCount, heapI);
            order = heapI;
        }
    } else {
        // tables larger than the shared-memory builder: the merges and the sort
        // run sequentially, on the same area where it holds the heap (8 bytes
        // per leaf) and then the sort's keys, else on global memory.  The area
        // leaves 28 KB of L1, so that 16000 leaves took 47.5 ms on global
        // memory (44.7 when a smaller builder left more); 34.0 so.
        u32* parent = p.parentWork + 2 * meta.leafOff;
        u64* heap = heapG;
        if (sizeof(u64) * L <= At::kBytes) {
            heap = reinterpret_cast<u64*>(dyn);
            for (u32 i = threadIdx.x; i < L; i += kThreads) heap[i] = heapG[i];
            __syncthreads();
        }
        if (threadIdx.x == 0) hb::buildTree(heap, parent, int(L));
        __syncthreads();
        if (sizeof(u32) * L <= At::kBytes) order = reinterpret_cast<u32*>(dyn);
        const u32 root = 2 * L - 2;
        u32 localMax = 0;
        for (u32 i = threadIdx.x; i < L; i += kThreads) {
            u32 d = 0, node = i;
            while (node != root && d < 32) { node = parent[node]; ++d; }
            order[i] = (min(d, 31u) << 27) | i;
            localMax = max(localMax, d);
        }
        if (localMax) atomicMax(&sMaxLen, localMax);
        __syncthreads();
        if (threadIdx.x == 0 && sMaxLen <= 31) hb::introsort(order, int(L), hb::LenLess());
    }
    if (threadIdx.x < 32) lenCount[threadIdx.x] = 0;
    __syncthreads();
    const u32 maxLen = sMaxLen;
    if (maxLen > 31) {
        if (threadIdx.x == 0) atomicOr(p.errors, DEV_ERR_CODEWORD_TOO_LONG);
        return;
    }
    // 4. canonical codes (HuffmanTable.cu:551-593)
    for (u32 k = threadIdx.x; k < L; k += kThreads) {
        u32 len = order[k] >> 27;
        if (len) atomicAdd(&lenCount[len - 1], 1u);
    }
    __syncthreads();
    // first index and code of every length l: index[l + 1] = index[l] + c[l],
    // code[l + 1] = 2 (code[l] + c[l]), scanned over the lanes (lane l - 1)
    if (threadIdx.x < 32) {
        const u32 c = lenCount[threadIdx.x];   // none of length 32
        u32 idx = c, code = c;
#pragma unroll
        for (u32 d = 1; d < 32; d <<= 1) {
            const u32 i = __shfl_up_sync(0xffffffffu, idx, d), k = __shfl_up_sync(0xffffffffu, code, d);
            if (threadIdx.x >= d) {
                idx += i;
                code += k << d;
            }
        }
        code = __shfl_up_sync(0xffffffffu, code, 1) << 1;
        firstIndex[threadIdx.x + 1] = idx - c;
        firstCode[threadIdx.x + 1] = threadIdx.x ? code : 0u;
    }
    __syncthreads();
    uint2* enc = p.enc + meta.histOff;
    for (u32 k = threadIdx.x; k < L; k += kThreads) {
        u32 len = order[k] >> 27;
        u32 sym = leafSym[order[k] & hb::kLeafMask];
        u32 code = len ? firstCode[len] + (k - firstIndex[len]) : 0u;
        enc[sym] = make_uint2(code, len);
    }
    // 5. serialized table (HuffmanTable.cu:470-485)
    const bool longSym = p.log2Max > 16;
    const u32 symbolBits = requiredBits(symbolMax);
    const u32 fixedBits = 5 + maxLen * p.log2Max + p.log2Max + (longSym ? 5u : 4u);
    const u32 headerBits = fixedBits + L * symbolBits;
    u32* hdr = p.headers + meta.hdrOff;
    const u32 hdrWords = u32(ceilDiv(headerBits, 32));
    for (u32 w = threadIdx.x; w < hdrWords; w += kThreads) hdr[w] = 0;
    __syncthreads();
    if (threadIdx.x < maxLen) putBits(hdr, 5 + threadIdx.x * p.log2Max, lenCount[threadIdx.x], p.log2Max);
    if (threadIdx.x == 0) {
        putBits(hdr, 0, maxLen, 5);
        putBits(hdr, 5 + maxLen * p.log2Max, L, p.log2Max);
        putBits(hdr, 5 + (maxLen + 1) * p.log2Max, symbolBits, longSym ? 5 : 4);
    }
    for (u32 k = threadIdx.x; k < L; k += kThreads)
        putBits(hdr, fixedBits + k * symbolBits, leafSym[order[k] & hb::kLeafMask], symbolBits);
    if (threadIdx.x == 0) {
        meta.symbolMax = symbolMax;
        meta.leaves = L;
        meta.maxLen = maxLen;
        meta.headerBits = headerBits;
        meta.codeBits = 0;
        p.meta[t] = meta;
    }
}

// One table per CTA (kBuildEach), or the CTAs walk the list of one tier.
// Bounding the one-warp tier to 72 registers (28 CTAs per SM instead of 21)
// left 4096 bricks at the same time.
template <u32 kThreads, u32 kCap, bool kWide>
__global__ void __launch_bounds__(kThreads, 1) k_tableBuild(EncParams p) {
    if (p.buildTier == kBuildEach) {
        buildTable<kThreads, kCap, kWide>(p, blockIdx.x);
        return;
    }
    const u32 n = u32(p.totals[4 + p.buildTier]);
    const u32* list = p.tierTables + u64(p.buildTier) * p.T;
    for (u32 i = blockIdx.x; i < n; i += gridDim.x) {
        buildTable<kThreads, kCap, kWide>(p, list[i]);
        __syncthreads();   // the next table reuses the shared memory
    }
}

// Dynamic shared memory that leaves no room on an SM for another table-build
// CTA or most other kernels' CTAs: the device's per-block opt-in limit minus
// the kernel's static shared memory.
template <bool kWide>
static size_t tableBuildSoloSmem(int device) {
    static size_t cached[64] = {};
    if (device < 0 || device >= 64) return 0;
    if (!cached[device]) {
        int optin = 0;
        cudaFuncAttributes fa{};
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
        cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(k_tableBuild<kBigThreads, kBuildSmemLeaves, kWide>));
        cached[device] = optin > int(fa.sharedSizeBytes) ? size_t(optin) - fa.sharedSizeBytes : 0;
    }
    return cached[device];
}

// ---------------------------------------------------------------------------
// Huffman encode (Huffman.cu:73-187): per coding block bit totals, per table
// scan to block offsets, then packing.  One warp per coding block.
// ---------------------------------------------------------------------------
constexpr u32 kPackWarps = 8;

// A lane's 32 symbols of a run, packed as they lie in memory (two 16-bit
// symbols or one 32-bit symbol per word): one 16-byte vector per 8 or 4
// symbols when the run lies inside the stream and is aligned, else element
// loads.  Positions at or past count read 0.
template <class Sym>
struct LaneRun {
    static constexpr u32 kWords = 32 * sizeof(Sym) / 4;
    u32 w[kWords];
    __device__ __forceinline__ u32 at(u32 k) const {   // k a compile-time constant after unrolling
        return sizeof(Sym) == 2 ? (w[k >> 1] >> (16 * (k & 1))) & 0xFFFFu : w[k];
    }
    __device__ __forceinline__ void load(const Sym* in, u32 j0, u32 count) {
        const Sym* q = in + j0;
        if (j0 + 32u <= count && (reinterpret_cast<uintptr_t>(q) & 15u) == 0) {
#pragma unroll
            for (u32 c = 0; c < kWords / 4; ++c) {
                const uint4 v = reinterpret_cast<const uint4*>(q)[c];
                w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
            }
            return;
        }
#pragma unroll
        for (u32 c = 0; c < kWords; ++c) {
            if (sizeof(Sym) == 2) {
                const u32 lo = j0 + 2 * c < count ? u32(q[2 * c]) : 0u;
                const u32 hi = j0 + 2 * c + 1 < count ? u32(q[2 * c + 1]) : 0u;
                w[c] = lo | (hi << 16);
            } else {
                w[c] = j0 + c < count ? u32(q[c]) : 0u;
            }
        }
    }
};

// Bits of every coding block in use.  Warps walk the call's run list
// (k_planFill): a run is kRunSymbols consecutive symbols of one table, 32
// per lane, so cb / 32 lanes share a coding block; each lane sums the code
// lengths of its symbols and the block's lanes add theirs.
template <class Sym>
__global__ void __launch_bounds__(kPackWarps * 32) k_blockBits(EncParams p) {
    const u32 lane = threadIdx.x & 31;
    if (warpFailed(p)) return;
    const u32 runs = u32(p.totals[3]);
    const u32 lpb = p.cb >> 5, bpr = kRunSymbols >> p.cbLog;
    const u32 stride = gridDim.x * kPackWarps;
    for (u32 r = blockIdx.x * kPackWarps + (threadIdx.x >> 5); r < runs; r += stride) {
        const u32 t = p.runTable[r];
        const TableMeta& m = p.meta[t];
        const EncTableDev td = p.tables[t];
        const u32 rb = r - m.runOff;
        u32 count;
        const Sym* in = tableInput<Sym>(p, td, count);
        const uint2* enc = p.enc + m.histOff;
        const u32 hs = m.histSize;
        const u32 j0 = rb * kRunSymbols + lane * 32u;
        LaneRun<Sym> sv;
        sv.load(in, j0, count);
        u32 bits = 0;
#pragma unroll
        for (u32 k = 0; k < 32; ++k)
            if (j0 + k < count) bits += enc[min(sv.at(k), hs - 1u)].y;
        for (u32 o = 1; o < lpb; o <<= 1) bits += __shfl_xor_sync(0xffffffffu, bits, o);
        const u32 b = rb * bpr + (lane >> (p.cbLog - 5u));
        if ((lane & (lpb - 1u)) == 0 && b < m.blocks) p.blockBits[td.blockOff + b] = bits;
    }
}

// Exclusive scan of each table's block bits: a warp per table, each lane
// summing eight consecutive blocks per step (256 blocks per step).
__global__ void __launch_bounds__(kScanWarps * 32) k_blockScan(EncParams p) {
    if (warpFailed(p)) return;
    const u32 t = blockIdx.x * kScanWarps + (threadIdx.x >> 5);
    if (t >= p.T) return;
    const u32 blocks = p.meta[t].blocks;
    const u32 off = p.tables[t].blockOff;
    const u32 total = warpExclusiveScan8(p.blockBits + off, p.blockOff + off, blocks, 0u);
    if ((threadIdx.x & 31u) == 0) p.meta[t].codeBits = total;
}

// The same with a CTA per table (wideBlockScan): 512 threads over the 16384 blocks of
// a 256^3 volume's band take 6 us, a warp 25.

__global__ void __launch_bounds__(512) k_blockScanWide(EncParams p) {
    __shared__ u32 scratch[40];
    if (blockFailed(p)) return;
    const u32 t = blockIdx.x;
    const u32 off = p.tables[t].blockOff;
    const u32 total = blockExclusiveScan8<512>(p.blockBits + off, p.blockOff + off, p.meta[t].blocks, scratch);
    if (threadIdx.x == 0) p.meta[t].codeBits = total;
}

// Segment layout per stream (a thread per stream), then the exclusive scan
// of the segments' words over the streams (k_layout, k_layoutCarry).
__device__ __forceinline__ SegmentLayout segmentOf(const EncParams& p, u32 s) {
    SegmentLayout L{};
    const EncStreamDev sd = p.streams[s];
    const u32 offW = (blocksOf(p.counts[s], p.cbLog) + 1u) / 2u;
    const TableMeta ms = p.meta[sd.tableFirst];
    u32 words;
    if (sd.kind == KIND_RLHUFF) {
        const TableMeta mz = p.meta[sd.tableFirst + 1];
        L.countWord = 0;
        L.hdrWord[0] = 1;
        L.cwWord[0] = L.hdrWord[0] + u32(ceilDiv(ms.headerBits, 32)) + 1;
        L.offWord[0] = L.cwWord[0] + u32(ceilDiv(ms.codeBits, 32));
        L.hdrWord[1] = L.offWord[0] + offW;
        L.cwWord[1] = L.hdrWord[1] + u32(ceilDiv(mz.headerBits, 32)) + 1;
        L.offWord[1] = L.cwWord[1] + u32(ceilDiv(mz.codeBits, 32));
        words = L.offWord[1] + offW;
        L.startBit = 0;
    } else {
        const u32 r = sd.startBit;
        L.hdrWord[0] = 0;
        L.cwWord[0] = u32(ceilDiv(r + ms.headerBits, 32)) + 1;
        L.offWord[0] = L.cwWord[0] + u32(ceilDiv(ms.codeBits, 32));
        words = L.offWord[0] + offW;
        L.startBit = r;
    }
    L.words = words;
    L.bitLength = words * 32u;
    return L;
}

__global__ void __launch_bounds__(256) k_layoutSegments(EncParams p) {
    if (*reinterpret_cast<volatile const u32*>(p.errors)) return;   // no barriers in this kernel
    const u32 s = blockIdx.x * 256u + threadIdx.x;
    if (s < p.S) p.layout[s] = segmentOf(p, s);
}

// Both steps of a call of at most 1024 streams.
__global__ void __launch_bounds__(1024) k_layoutOne(EncParams p) {
    __shared__ u32 scratch[40];
    if (blockFailed(p)) return;
    const u32 s = threadIdx.x;
    SegmentLayout L{};
    if (s < p.S) L = segmentOf(p, s);
    u32 tot;
    L.startWord = blockExclusiveSum<1024>(L.words, scratch, &tot);
    if (s < p.S) p.layout[s] = L;
    if (threadIdx.x == 0) {
        p.totals[0] = tot;
        if (tot > p.outWordsMax) atomicOr(p.errors, DEV_ERR_OUTPUT_CAPACITY);
    }
}

// CTA b scans the segment words of streams 1024 b .. 1024 b + 1023; with more
// than one chunk its sum goes to planPart and k_layoutCarry adds the chunks
// before each one (the histogram plan's sums are consumed by then).
__global__ void __launch_bounds__(1024) k_layout(EncParams p) {
    __shared__ u32 scratch[40];
    if (blockFailed(p)) return;
    const u32 s = blockIdx.x * 1024u + threadIdx.x;
    const u32 words = s < p.S ? p.layout[s].words : 0u;
    u32 tot;   // a chunk's words fit 32 bits; the offsets over chunks are 64-bit
    const u32 ex = blockExclusiveSum<1024>(words, scratch, &tot);
    if (s < p.S) p.layout[s].startWord = ex;
    if (threadIdx.x == 0) {
        if (gridDim.x == 1) {
            p.totals[0] = tot;
            if (tot > p.outWordsMax) atomicOr(p.errors, DEV_ERR_OUTPUT_CAPACITY);
        } else {
            p.planPart[blockIdx.x] = tot;
        }
    }
}

// Chunk b = blockIdx.x + 1 of a layout of more than one chunk: the words of
// chunks 0 .. b-1 added to its streams' start words; the last chunk's CTA
// forms the call's total and checks the output capacity.
__global__ void __launch_bounds__(1024) k_layoutCarry(EncParams p) {
    __shared__ unsigned long long sC;
    if (blockFailed(p)) return;
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
    const u32 s = b * 1024u + threadIdx.x;
    if (s < p.S) p.layout[s].startWord += c;
    if (b == gridDim.x && threadIdx.x == 0) {
        const unsigned long long total = c + p.planPart[b];
        p.totals[0] = total;
        if (total > p.outWordsMax) atomicOr(p.errors, DEV_ERR_OUTPUT_CAPACITY);
    }
}

// a << n for n in 0 .. 32 and up (0 from 32 on).
__device__ __forceinline__ u32 shl32(u32 a, u32 n) { return __funnelshift_lc(0u, a, n); }

// Or the part of codeword `code` (len bits at absolute bit `pos`) that falls
// in words [wLo, wHi) into win[] (win[0] = word wLo).
__device__ __forceinline__ void orCodeword(u32* win, u32 wLo, u32 wHi, u32 pos, u32 code, u32 len) {
    if (len == 0) return;
    const u32 w0 = pos >> 5;
    const int shift = int(32 - (pos & 31u)) - int(len);
    if (shift >= 0) {
        if (w0 >= wLo && w0 < wHi) atomicOr(win + (w0 - wLo), code << shift);
    } else {
        if (w0 >= wLo && w0 < wHi) atomicOr(win + (w0 - wLo), code >> (-shift));
        if (w0 + 1 >= wLo && w0 + 1 < wHi) atomicOr(win + (w0 + 1 - wLo), code << (32 + shift));
    }
}

// Packing, by runs of coding blocks (as k_blockBits): the run's codewords
// are contiguous in the table's bit stream from its first block's offset, so
// a lane's start bit is that offset plus the code lengths of the lanes
// before it.  Each warp writes the output words whose first bit lies in its
// run (gather ownership: no atomics on global memory, no pre-zeroing),
// assembling them in a shared-memory window; the bits of the last owned word
// that belong to the next run are recomputed from that run's first symbols.
// A lane looks each code up once, keeps pairs of codes until its bit offset is
// known, and puts four codes at a time.  Bound: instruction issue; putting one
// code at a time took the same streams' 52 million codes 106 us, this 80.
constexpr u32 kPackWindowWords = kRunSymbols * 31u / 32u + 2u;

__device__ void writeHeaders(const EncParams& p, u32 s, u32 gt, u32 g);

// The first headCtas CTAs write the streams' headers beside the packing, g
// threads per stream.
template <class Sym>
__global__ void __launch_bounds__(kPackWarps * 32, 3) k_pack(EncParams p, u32 headCtas, u32 g) {
    __shared__ u32 winAll[kPackWarps * kPackWindowWords];
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warpFailed(p)) return;
    if (blockIdx.x < headCtas) {
        const u32 s = (blockIdx.x * (kPackWarps * 32u) + threadIdx.x) / g;
        if (s < p.S) writeHeaders(p, s, threadIdx.x & (g - 1u), g);
        return;
    }
    u32* win = winAll + warp * kPackWindowWords;
    const u32 runs = u32(p.totals[3]);
    const u32 bpr = kRunSymbols >> p.cbLog;
    const u32 stride = (gridDim.x - headCtas) * kPackWarps;
    for (u32 r = (blockIdx.x - headCtas) * kPackWarps + warp; r < runs; r += stride) {
        const u32 t = p.runTable[r];
        const TableMeta m = p.meta[t];
        const EncTableDev td = p.tables[t];
        const u32 rb = r - m.runOff;
        const u32 bFirst = rb * bpr, bEnd = min(bFirst + bpr, m.blocks);
        u32 count;
        const Sym* in = tableInput<Sym>(p, td, count);
        const u32* bo = p.blockOff + td.blockOff;
        const u32 off0 = bo[bFirst];
        const u32 off1 = bEnd < m.blocks ? bo[bEnd] : m.codeBits;
        const u32 wLo = (off0 + 31) >> 5, wHi = (off1 + 31) >> 5;
        if (wLo >= wHi) continue;
        for (u32 w = lane; w < wHi - wLo; w += 32) win[w] = 0;
        const uint2* enc = p.enc + m.histOff;
        const u32 hs = m.histSize;
        const u32 j0 = rb * kRunSymbols + lane * 32u;
        // one lookup per symbol; two codes at a time joined in a word (first
        // code upper), four pairs' lengths in a register, while the lane's bit
        // offset is scanned.  A warp meeting a pair of more than 32 bits looks
        // its codes up again one by one instead.
        u32 pair[16], plen[4] = {0u, 0u, 0u, 0u};
        u32 lsum = 0;
        bool longPair = false;
        {
            LaneRun<Sym> sv;
            sv.load(in, j0, count);
#pragma unroll
            for (u32 k = 0; k < 16; ++k) {
                const uint2 a = j0 + 2 * k < count ? enc[min(sv.at(2 * k), hs - 1u)] : make_uint2(0u, 0u);
                const uint2 b = j0 + 2 * k + 1 < count ? enc[min(sv.at(2 * k + 1), hs - 1u)] : make_uint2(0u, 0u);
                const u32 l = a.y + b.y;
                longPair |= l > 32u;
                pair[k] = (a.x << (b.y & 31u)) | b.x;   // b.y = 32 cannot be: codes are at most 31 bits
                plen[k >> 2] |= l << (8 * (k & 3));
                lsum += l;
            }
        }
        const bool reload = __any_sync(0xffffffffu, longPair);
        __syncwarp();
        // the lane's codewords are consecutive: concatenate them in a word
        // (bits left-aligned from the lane's start bit in its first word) and
        // OR whole words into the window - one shared atomic per word touched
        const u32 pos = off0 + warpInclusiveSum(lsum) - lsum;
        {
            u32 w = pos >> 5;
            u32 n = pos & 31u;   // bits of cur in use
            u32 cur = 0;
            auto put = [&](u32 code, u32 len) {   // len <= 32; shifts by 32 give 0
                const u32 left = shl32(code, 32u - len);
                cur |= left >> n;
                const u32 total = n + len;
                if (total >= 32u) {
                    if (w >= wLo && w < wHi) atomicOr(win + (w - wLo), cur);
                    ++w;
                    cur = shl32(left, 32u - n);
                }
                n = total & 31u;
            };
            if (!reload) {
#pragma unroll
                for (u32 k = 0; k < 16; k += 2) {
                    const u32 la = (plen[k >> 2] >> (8 * (k & 3))) & 255u, lb = (plen[k >> 2] >> (8 * (k & 3) + 8)) & 255u;
                    if (la + lb <= 32u) {
                        put(shl32(pair[k], lb) | pair[k + 1], la + lb);
                    } else {
                        put(pair[k], la);
                        put(pair[k + 1], lb);
                    }
                }
            } else {
                LaneRun<Sym> sv;
                sv.load(in, j0, count);
#pragma unroll
                for (u32 k = 0; k < 32; ++k) {
                    const uint2 c = j0 + k < count ? enc[min(sv.at(k), hs - 1u)] : make_uint2(0u, 0u);
                    put(c.x, c.y);
                }
            }
            if (n && w >= wLo && w < wHi) atomicOr(win + (w - wLo), cur);
        }
        // bits of the next run inside the last owned word
        if (bEnd < m.blocks && (wHi << 5) > off1) {
            const u32 j = bEnd * p.cb + lane;
            const uint2 c = j < count ? enc[min(u32(in[j]), hs - 1u)] : make_uint2(0, 0);
            const u32 q = off1 + warpInclusiveSum(c.y) - c.y;
            if (q < (wHi << 5)) orCodeword(win, wLo, wHi, q, c.x, c.y);
        }
        __syncwarp();
        const u32 which = (p.streams[td.stream].kind == KIND_RLHUFF && td.which) ? 1u : 0u;
        const SegmentLayout& L = p.layout[td.stream];
        u32* dst = p.out + L.startWord + L.cwWord[which];
        for (u32 w = lane; w < wHi - wLo; w += 32) dst[wLo + w] = win[w];
        __syncwarp();   // the window is cleared for the next run only after these reads
    }
}

// Count words, table headers, codeword bit counts and offset increments of
// stream s, by g threads (a power of two, 32 .. 256; this one gt): a call of
// many streams packs several into a CTA (as many as still leave four CTAs per
// SM).
__device__ void writeHeaders(const EncParams& p, u32 s, u32 gt, u32 g) {
    const EncStreamDev sd = p.streams[s];
    const SegmentLayout L = p.layout[s];
    u32* seg = p.out + L.startWord;
    const bool rl = sd.kind == KIND_RLHUFF;
    const u32 parts = rl ? 2u : 1u;
    if (rl && gt == 0) seg[L.countWord] = p.counts[s];
    for (u32 part = 0; part < parts; ++part) {
        const u32 t = sd.tableFirst + part;
        const TableMeta m = p.meta[t];
        const u32* hdr = p.headers + m.hdrOff;
        const u32 r = part == 0 ? L.startBit : 0u;
        const u32 hw = u32(ceilDiv(r + m.headerBits, 32));
        u32* dst = seg + L.hdrWord[part];
        const u32 srcWords = u32(ceilDiv(m.headerBits, 32));
        for (u32 w = gt; w < hw; w += g) {
            u32 v;
            if (r == 0) {
                v = hdr[w];
            } else {
                const u32 hi = (w >= 1 && w - 1 < srcWords) ? hdr[w - 1] : 0u;
                const u32 lo = w < srcWords ? hdr[w] : 0u;
                v = (hi << (32 - r)) | (lo >> r);
            }
            dst[w] = v;
        }
        if (gt == 0) seg[L.cwWord[part] - 1] = m.codeBits;
        // offsets: u16 increments, two per word, first in the low half (LE memcpy)
        const u32 nOff = m.blocks;
        const u32* bo = p.blockOff + p.tables[t].blockOff;
        u32* od = seg + L.offWord[part];
        for (u32 w = gt; w < (nOff + 1) / 2; w += g) {
            const u32 k0 = 2 * w, k1 = 2 * w + 1;
            const u32 a = k0 == 0 ? bo[0] : bo[k0] - bo[k0 - 1];
            const u32 b = k1 < nOff ? bo[k1] - bo[k1 - 1] : 0u;
            od[w] = (a & 0xFFFFu) | ((b & 0xFFFFu) << 16);
        }
    }
}

// Word offset and bit size of each volume's stream in a batched encode's
// output: volume v owns streams first[v] .. first[v+1]-1, written back to back.
__global__ void k_volumeExtents(const SegmentLayout* layout, const u32* first, u32 count, u64* wordOff,
                                u64* bitSize, const u32* errors) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= count) return;
    if (*errors) { wordOff[v] = 0; bitSize[v] = 0; return; }
    const u32 a = first[v], b = first[v + 1];
    const u64 off = layout[a].startWord;
    const u64 end = layout[b - 1].startWord + layout[b - 1].words;
    wordOff[v] = off;
    bitSize[v] = (end - off) * 32ull;
}

// ---------------------------------------------------------------------------
// Host orchestration.
// ---------------------------------------------------------------------------
// Writes the stream and table descriptors of a call into `slot` (host) and
// returns its summary; slotBytes bounds the descriptors.
int encodePrepare(cc_instance* I, const EncStream* streams, u32 S, char* slot, size_t slotBytes, EncPlan& hp) {
    hp = EncPlan{};
    hp.S = S;
    for (u32 s = 0; s < S; ++s) {
        const EncStream& e = streams[s];
        const u64 nb = ceilDiv(e.n, I->codingBlockSize);
        hp.T += e.kind == KIND_RLHUFF ? 2u : 1u;
        hp.tiles += u32(ceilDiv(e.n, kRleTile));
        hp.blocks += u32(e.kind == KIND_RLHUFF ? 2 * nb : nb);
        hp.maxCount = std::max(hp.maxCount, e.n);
        if (e.kind == KIND_RLHUFF) hp.compact += e.n;
    }
    if (S > I->capStreams || hp.T > I->capTables || hp.tiles > I->capTiles || hp.blocks > I->capBlocks ||
        hp.compact > I->capCompact) {
        setError("encode: call exceeds the instance capacity (%u streams, %llu run-length symbols)", S,
                 (unsigned long long)hp.compact);
        return CC_ERR_CAPACITY;
    }
    hp.offTables = alignUp(sizeof(EncStreamDev) * S, 64);
    hp.bytes = hp.offTables + sizeof(EncTableDev) * hp.T;
    if (hp.bytes > slotBytes) { setError("encode: descriptors exceed the staging slot"); return CC_ERR_CAPACITY; }
    EncStreamDev* sd = reinterpret_cast<EncStreamDev*>(slot);
    EncTableDev* td = reinterpret_cast<EncTableDev*>(slot + hp.offTables);
    u32 tile = 0, table = 0, block = 0;
    u64 compact = 0;
    for (u32 s = 0; s < S; ++s) {
        const EncStream& e = streams[s];
        EncStreamDev d{};
        d.in = e.in;
        d.n = e.n;
        d.kind = e.kind;
        d.startBit = e.kind == KIND_HUFF ? (e.startBit & 31u) : 0u;
        d.groupFirst = e.groupFirst;
        d.groupSize = e.groupSize;
        d.tileOff = tile;
        d.tableFirst = table;
        d.compactOff = compact;
        sd[s] = d;
        tile += u32(ceilDiv(e.n, kRleTile));
        if (e.kind == KIND_RLHUFF) compact += e.n;
        const u32 parts = e.kind == KIND_RLHUFF ? 2u : 1u;
        const u32 nb = u32(ceilDiv(e.n, I->codingBlockSize));
        for (u32 w = 0; w < parts; ++w) {
            td[table++] = EncTableDev{s, w, block, nb};
            block += nb;
        }
    }
    return CC_OK;
}

// The full builder's dynamic shared memory, allowed for its launch.
template <bool kWide>
static cudaError_t tableBuildSmem(const cc_instance* I, bool solo, size_t& bytes) {
    bytes = hm::Layout<kBuildSmemLeaves>::kBytes;
    if (solo) bytes = std::max(bytes, tableBuildSoloSmem<kWide>(I->device));
    return ensureSmemAttribute(reinterpret_cast<const void*>(k_tableBuild<kBigThreads, kBuildSmemLeaves, kWide>),
                               kWide ? kAttrTableBuildWide : kAttrTableBuild, I->device, bytes);
}

template <bool kWide>
static int launchTableBuild(cc_instance* I, const EncParams& p) {
    cudaStream_t st = I->stream;
    const u32 sms = I->smCount;
    // an instance whose tables run beside other kernels (the batched codec's
    // lowpass encode) may ask for an SM of its own per table: the sequential
    // heap merge is latency-bound and loses issue slots to co-resident CTAs
    const bool solo = I->tableBuildSoloSM && p.T <= sms;
    size_t buildSmem;
    CC_TRY_CUDA(tableBuildSmem<kWide>(I, solo, buildSmem), "tableBuild smem");
    {
        SectionTimer t(I, "enc.table_build", st);
        EncParams q = p;
        q.buildLo = 0;
        q.buildHi = ~0u;
        q.buildTier = kBuildEach;
        // a call of few tables builds them in one launch, a CTA each (the
        // tiers' pre-pass, launches and stream forks would cost it more than
        // they save)
        if (!solo && p.T > kTierMinTables) {
            // tables sorted by leaf count, each tier's list walked by its own
            // builder, at the same time: tier 0 on the instance stream, tier 1
            // on the second side stream, tiers 3 and 2 on the first
            k_leafTiers<<<u32(ceilDiv(p.T, 8)), 256, 0, st>>>(q);
            countLaunch();
            const bool side = p.heapCap > kSmallLeaves, side2 = p.heapCap > kTinyLeaves;
            if (side2) {
                CC_TRY_CUDA(cudaEventRecord(I->buildFork, st), "table build fork");
                CC_TRY_CUDA(cudaStreamWaitEvent(I->buildSide2, I->buildFork, 0), "table build fork");
                EncParams small = q;
                small.buildTier = 1;
                small.buildLo = kTinyLeaves + 1;
                small.buildHi = kSmallLeaves;
                k_tableBuild<64u, kSmallLeaves, kWide>
                    <<<std::min(p.T, 10u * sms), 64, hm::Layout<kSmallLeaves>::kBytes, I->buildSide2>>>(small);
                countLaunch();
                CC_TRY_CUDA(cudaEventRecord(I->buildJoin2, I->buildSide2), "table build join");
            }
            if (side) {
                CC_TRY_CUDA(cudaStreamWaitEvent(I->buildSide, I->buildFork, 0), "table build fork");
                if (p.heapCap > kBuildSplitLeaves) {
                    EncParams big = q;
                    big.buildTier = 3;
                    big.buildLo = kBuildSplitLeaves + 1;
                    k_tableBuild<kBigThreads, kBuildSmemLeaves, kWide>
                        <<<std::min(p.T, sms), kBigThreads, buildSmem, I->buildSide>>>(big);
                    countLaunch();
                }
                EncParams mid = q;
                mid.buildTier = 2;
                mid.buildLo = kSmallLeaves + 1;
                mid.buildHi = kBuildSplitLeaves;
                k_tableBuild<kMidThreads, kBuildSplitLeaves, kWide>
                    <<<std::min(p.T, 5u * sms), kMidThreads, hm::Layout<kBuildSplitLeaves>::kBytes, I->buildSide>>>(mid);
                countLaunch();
                CC_TRY_CUDA(cudaEventRecord(I->buildJoin, I->buildSide), "table build join");
            }
            EncParams tiny = q;
            tiny.buildTier = 0;
            tiny.buildHi = kTinyLeaves;
            k_tableBuild<32u, kTinyLeaves, kWide>
                <<<std::min(p.T, 32u * sms), 32, hm::Layout<kTinyLeaves>::kBytes, st>>>(tiny);
            countLaunch();
            if (side2) CC_TRY_CUDA(cudaStreamWaitEvent(st, I->buildJoin2, 0), "table build join");
            if (side) CC_TRY_CUDA(cudaStreamWaitEvent(st, I->buildJoin, 0), "table build join");
        } else {
            if (!solo && p.heapCap <= kSmallLeaves)
                k_tableBuild<kBuildThreads, kSmallLeaves, kWide>
                    <<<p.T, kBuildThreads, hm::Layout<kSmallLeaves>::kBytes, st>>>(q);
            else if (!solo && p.heapCap <= kBuildSplitLeaves)
                k_tableBuild<kBuildThreads, kBuildSplitLeaves, kWide>
                    <<<p.T, kBuildThreads, hm::Layout<kBuildSplitLeaves>::kBytes, st>>>(q);
            else
                k_tableBuild<kBigThreads, kBuildSmemLeaves, kWide><<<p.T, kBigThreads, buildSmem, st>>>(q);
            countLaunch();
        }
    }
    return CC_OK;
}

template <class Sym>
static int launchEncode(cc_instance* I, const EncParams& p) {
    cudaStream_t st = I->stream;
    k_encBegin<<<p.S, 256, 0, st>>>(p);   // S > 0: encodeDevice returns early, a batch has volumes
    countLaunch();
    if (p.totalTiles) { SectionTimer t(I, "enc.summary", st); k_summary<Sym><<<p.totalTiles, kRleThreads, 0, st>>>(p); countLaunch(); }
    const u32 chunks = std::max<u32>(1, u32(ceilDiv(p.T, kPlanChunk)));
    const bool wide = wideTileScan(p.S, u32(ceilDiv(p.maxCount, kRleTile)));
    if (p.S <= kScanPlanStreams && !wide) {   // then one chunk
        SectionTimer t(I, "enc.hist_plan", st);
        k_scanPlan<<<1, 1024, 0, st>>>(p);
        countLaunch();
    } else {
        {
            SectionTimer t(I, "enc.rle_scan", st);
            if (wide) k_scanWide<<<p.S, kScanThreads, 0, st>>>(p);
            else k_scan<<<u32(ceilDiv(p.S, kScanWarps)), kScanWarps * 32, 0, st>>>(p);
            countLaunch();
        }
        SectionTimer t(I, "enc.hist_plan", st);
        k_histPlan<<<chunks, 1024, 0, st>>>(p);
        countLaunch();
        if (chunks > 1) { k_histPlanCarry<<<chunks - 1, 1024, 0, st>>>(p); countLaunch(); }
    }
    if (I->encFillAfter) CC_TRY_CUDA(cudaStreamWaitEvent(st, I->encFillAfter, 0), "encode order");
    { SectionTimer t(I, "enc.hist_zero", st); k_planFill<<<2 * I->smCount, 256, 0, st>>>(p); countLaunch(); }
    if (p.totalTiles) {
        CC_TRY_CUDA(ensureSmemAttribute(reinterpret_cast<const void*>(k_write<Sym>),
                                        sizeof(Sym) == 2 ? kAttrWrite16 : kAttrWrite32, I->device, writeSmem<Sym>()),
                    "write smem");
        SectionTimer t(I, "enc.rle_write_hist", st);
        k_write<Sym><<<p.totalTiles, kRleThreads, writeSmem<Sym>(), st>>>(p);
        countLaunch();
    }
    if (I->encBuildNext) CC_TRY_CUDA(cudaEventRecord(I->encBuildNext, st), "encode order");
    int rc = p.bins > kWideBins ? launchTableBuild<true>(I, p) : launchTableBuild<false>(I, p);
    if (rc) return rc;
    const u32 sms = I->smCount;
    // the block kernels walk the run list (k_planFill) with a few CTAs per SM
    const u32 blockGrid = sms * 8u;
    // runs of the call: at most the used blocks / blocks per run, plus one per table
    const u32 runBound = u32(ceilDiv(p.totalBlocks, kRunSymbols / p.cb)) + p.T;
    if (p.totalBlocks) {
        const u32 g = std::min<u32>(blockGrid, u32(ceilDiv(runBound, kPackWarps)));
        { SectionTimer t(I, "enc.block_bits", st); k_blockBits<Sym><<<g, kPackWarps * 32, 0, st>>>(p); countLaunch(); }
        {
            SectionTimer t(I, "enc.block_scan", st);
            if (wideBlockScan(p.T, u32(ceilDiv(p.maxCount, p.cb)), sms)) k_blockScanWide<<<p.T, 512, 0, st>>>(p);
            else k_blockScan<<<u32(ceilDiv(p.T, kScanWarps)), kScanWarps * 32, 0, st>>>(p);
            countLaunch();
        }
    }
    {
        SectionTimer t(I, "enc.layout", st);
        if (p.S <= 1024) {
            k_layoutOne<<<1, 1024, 0, st>>>(p);
            countLaunch();
        } else {
            k_layoutSegments<<<u32(ceilDiv(p.S, 256)), 256, 0, st>>>(p);
            const u32 chunks = u32(ceilDiv(p.S, 1024));
            k_layout<<<chunks, 1024, 0, st>>>(p);
            k_layoutCarry<<<chunks - 1, 1024, 0, st>>>(p);
            countLaunch(3);
        }
    }
    {
        SectionTimer t(I, "enc.pack", st);
        const u32 packCtas = p.totalBlocks ? std::min<u32>(blockGrid, u32(ceilDiv(runBound, kPackWarps))) : 0u;
        // streams per CTA: as few as keep four CTAs per SM busy
        u32 per = 1;
        while (per < 8 && u64(2 * per) * 4 * sms <= p.S) per <<= 1;
        const u32 headCtas = u32(ceilDiv(p.S, per));
        k_pack<Sym><<<headCtas + packCtas, kPackWarps * 32, 0, st>>>(p, headCtas, kPackWarps * 32 / per);
        countLaunch();
    }
    CC_TRY_CUDA(cudaGetLastError(), "encode launch");
    return CC_OK;
}

int prepareDecodeAttributes(cc_instance* I);

int prepareKernelAttributes(cc_instance* I) {
    size_t bytes;
    CC_TRY_CUDA(I->bins > kWideBins ? tableBuildSmem<true>(I, I->tableBuildSoloSM, bytes)
                                    : tableBuildSmem<false>(I, I->tableBuildSoloSM, bytes),
                "tableBuild smem");
    if (I->symBytes == 2)
        CC_TRY_CUDA(ensureSmemAttribute(reinterpret_cast<const void*>(k_write<u16>), kAttrWrite16, I->device,
                                        writeSmem<u16>()), "write smem");
    else
        CC_TRY_CUDA(ensureSmemAttribute(reinterpret_cast<const void*>(k_write<u32>), kAttrWrite32, I->device,
                                        writeSmem<u32>()), "write smem");
    return prepareDecodeAttributes(I);
}

void volumeExtents(cc_instance* I, const u32* first, u32 count, u64* wordOff, u64* bitSize, cudaStream_t st) {
    k_volumeExtents<<<u32(ceilDiv(count, 256)), 256, 0, st>>>(I->layout, first, count, wordOff, bitSize, I->errors);
    countLaunch();
}

// Launches the encode of a prepared call whose descriptors are at
// plan.dev (device); writes the segments to out (at most outCap words).
// Only kernel launches and device-side memsets.
int encodeLaunch(cc_instance* I, const EncPlan& hp, u32* out, u64 outCap) {
    const char* dPlan = static_cast<const char*>(hp.dev);
    EncParams p{};
    p.S = hp.S;
    p.T = hp.T;
    p.totalTiles = hp.tiles;
    p.maxCount = hp.maxCount;
    p.totalBlocks = hp.blocks;
    p.cb = I->codingBlockSize;
    p.cbLog = 31u - u32(__builtin_clz(p.cb));
    p.log2Max = I->log2Max;
    p.bins = I->bins;
    p.symBytes = I->symBytes;
    p.streams = reinterpret_cast<const EncStreamDev*>(dPlan);
    p.tables = reinterpret_cast<const EncTableDev*>(dPlan + hp.offTables);
    p.compact = static_cast<char*>(I->compact);
    p.zc = static_cast<char*>(I->zc);
    p.tiles = I->tiles;
    p.tileStart = I->tileStart;
    p.streamMax = I->streamMax;
    p.counts = I->counts;
    p.hist = I->hist;
    p.enc = I->enc;
    p.meta = I->meta;
    p.headers = I->headers;
    p.blockBits = I->blockBits;
    p.blockOff = I->blockOff;
    p.runTable = I->runTable;
    p.tileStream = I->tileStream;
    p.layout = I->layout;
    p.out = out;
    p.outWordsMax = outCap;
    p.capHist = I->capHist;
    p.capLeaves = I->capLeaves;
    p.capHdr = I->capHdr;
    p.errors = I->errors;
    p.totals = I->totals;
    p.leafWork = I->leafWork;
    p.parentWork = I->parentWork;
    p.orderWork = I->orderWork;
    p.leafSymWork = I->leafSymWork;
    p.tierTables = I->tierTables;
    p.planPart = I->planPart;
    p.heapCap = std::min<u32>(std::min<u32>(I->leavesMax, kBuildSmemLeaves), hp.maxCount + 1u);
    return I->symBytes == 2 ? launchEncode<u16>(I, p) : launchEncode<u32>(I, p);
}

int encodeDevice(cc_instance* I, const EncStream* streams, u32 S, const EncOutput& outSpec, bool download,
                 u64* totalWords) {
    if (totalWords) *totalWords = 0;
    if (S == 0) { I->lastLayout.clear(); return CC_OK; }
    cudaStream_t st = I->stream;
    char* slot = I->takeRingSlot();
    EncPlan hp;
    int rc = encodePrepare(I, streams, S, slot, I->hostRingBytes, hp);
    if (rc) return rc;
    hp.dev = I->dPlan;
    CC_TRY_CUDA(cudaMemcpyAsync(I->dPlan, slot, hp.bytes, cudaMemcpyHostToDevice, st), "upload plan");
    cudaEventRecord(I->ringEvent[(I->ringNext + cc_instance::kRing - 1) % cc_instance::kRing], st);
    u32* out = outSpec.words ? outSpec.words : I->out;
    rc = encodeLaunch(I, hp, out, outSpec.words ? outSpec.capacity : I->outWordsMax);
    if (rc) return rc;
    // results: layout, total words, error flags
    char* down = I->hostDown;
    CC_TRY_CUDA(cudaMemcpyAsync(down, I->layout, sizeof(SegmentLayout) * S, cudaMemcpyDeviceToHost, st), "download layout");
    char* tail = down + alignUp(sizeof(SegmentLayout) * S, 64);
    CC_TRY_CUDA(cudaMemcpyAsync(tail, I->totals, sizeof(u64), cudaMemcpyDeviceToHost, st), "download totals");
    CC_TRY_CUDA(cudaMemcpyAsync(tail + 64, I->errors, sizeof(u32), cudaMemcpyDeviceToHost, st), "download errors");
    CC_TRY_CUDA(cudaStreamSynchronize(st), "encode");
    const u32 flags = *reinterpret_cast<u32*>(tail + 64);
    if (flags) return deviceErrorStatus(flags, "encode");
    const u64 total = *reinterpret_cast<u64*>(tail);
    I->lastLayout.assign(reinterpret_cast<SegmentLayout*>(down), reinterpret_cast<SegmentLayout*>(down) + S);
    if (totalWords) *totalWords = total;
    if (download && total) {
        if (total > I->hostWordsMax) { setError("encode: result larger than the host staging"); return CC_ERR_CAPACITY; }
        CC_TRY_CUDA(cudaMemcpyAsync(I->hostWords, out, total * 4, cudaMemcpyDeviceToHost, st), "download words");
        CC_TRY_CUDA(cudaStreamSynchronize(st), "download words");
    }
    return CC_OK;
}

}  // namespace ccb

using namespace ccb;

extern "C" {

int cc_encode(cc_instance* I, int kind, int symbolBytes, const void* const* dStreams, uint32_t S, uint32_t n,
              const uint32_t* startBits) {
    if (!I || (S && !dStreams)) { setError("cc_encode: null argument"); return CC_ERR_INVALID_ARGUMENT; }
    if (kind != KIND_RLHUFF && kind != KIND_HUFF) { setError("cc_encode: bad kind %d", kind); return CC_ERR_INVALID_ARGUMENT; }
    if (u32(symbolBytes) != I->symBytes) {
        setError("cc_encode: %d-byte symbols need an instance with log2HuffmanDistinctSymbolCountMax %s 16",
                 symbolBytes, symbolBytes == 2 ? "<=" : ">");
        return CC_ERR_INVALID_ARGUMENT;
    }
    if (S > I->streamCountMax) { setError("stream count %u exceeds instance limit %u", S, I->streamCountMax); return CC_ERR_CAPACITY; }
    if (n > I->elemCountPerStreamMax) { setError("symbol count %u exceeds instance limit %u", n, I->elemCountPerStreamMax); return CC_ERR_CAPACITY; }
    DeviceGuard deviceGuard(I->device);
    std::vector<EncStream> st(S);
    for (u32 i = 0; i < S; ++i) {
        st[i].in = dStreams[i];
        st[i].n = n;
        st[i].startBit = (kind == KIND_HUFF && startBits) ? (startBits[i] & 31u) : 0u;
        st[i].groupFirst = 0;
        st[i].groupSize = S;
        st[i].kind = u32(kind);
    }
    return encodeDevice(I, st.data(), S, EncOutput{}, true);
}

int cc_encoded_segment(const cc_instance* I, uint32_t i, const uint32_t** words, uint32_t* wordCount,
                       uint32_t* startBit, uint32_t* bitLength) {
    if (!I || i >= I->lastLayout.size()) { setError("cc_encoded_segment: index out of range"); return CC_ERR_INVALID_ARGUMENT; }
    const SegmentLayout& L = I->lastLayout[i];
    if (words) *words = I->hostWords + L.startWord;
    if (wordCount) *wordCount = L.words;
    if (startBit) *startBit = L.startBit;
    if (bitLength) *bitLength = L.bitLength;
    return CC_OK;
}

// Appends the segments to a word buffer with BitStream::write* semantics
// (BitStream.h:377-480): RLHuff segments start at the next word boundary,
// Huff segments at the current bit; bits before the position are kept.
int cc_encode_to_buffer(cc_instance* I, int kind, int symbolBytes, const void* const* dStreams, uint32_t S,
                        uint32_t n, uint32_t* words, uint32_t capacity, uint32_t* bitSize, uint32_t* bitPos) {
    if (!bitSize || !bitPos) { setError("cc_encode_to_buffer: null size/position"); return CC_ERR_INVALID_ARGUMENT; }
    u32 pos = *bitPos;
    std::vector<u32> sb(S, 0);
    if (S) sb[0] = pos & 31u;
    int rc = cc_encode(I, kind, symbolBytes, dStreams, S, n, sb.data());
    if (rc) return rc;
    u64 end = pos;
    for (u32 i = 0; i < S; ++i) {
        const SegmentLayout& L = I->lastLayout[i];
        u64 w0 = kind == KIND_RLHUFF ? ceilDiv(end, 32) : end / 32;
        end = w0 * 32 + L.bitLength;
    }
    u64 needWords = ceilDiv(std::max<u64>(end, *bitSize), 32);
    if (needWords > capacity) {
        *bitSize = u32(std::max<u64>(end, *bitSize));
        setError("cc_encode_to_buffer: need %llu words, capacity %u", (unsigned long long)needWords, capacity);
        return CC_ERR_CAPACITY;
    }
    u32 oldWords = u32(ceilDiv(*bitSize, 32));
    for (u64 w = oldWords; w < needWords; ++w) words[w] = 0;
    u64 cur = pos;
    for (u32 i = 0; i < S; ++i) {
        const SegmentLayout& L = I->lastLayout[i];
        const u32* src = I->hostWords + L.startWord;
        u64 w0 = kind == KIND_RLHUFF ? ceilDiv(cur, 32) : cur / 32;
        u32 r = kind == KIND_RLHUFF ? 0u : u32(cur & 31u);
        u32 keep = r ? (0xffffffffu << (32 - r)) : 0u;
        words[w0] = (words[w0] & keep) | (src[0] & ~keep);
        std::memcpy(words + w0 + 1, src + 1, size_t(L.words - 1) * 4);
        cur = w0 * 32 + L.bitLength;
    }
    *bitPos = u32(cur);
    *bitSize = u32(std::max<u64>(cur, *bitSize));
    return CC_OK;
}

}  // extern "C"
