// table_build.cuh - the device side of the Huffman table construction: the
// same observable result as the reference's host builder (HuffmanTable.cu:
// 487-596, libstdc++ priority_queue + std::sort) with the work a block can
// share done by the block.
//
//  * tree: make_heap runs level by level over the block; the merge loop, a
//    chain of pops and pushes, runs on one warp with a lane per heap level
//    (heap_merge.cuh);
//  * depths: one thread per leaf walks to the root;
//  * sort: std::sort's introsort is replayed exactly, but every partition
//    step runs on a warp: the left scan stops at the k-th element not less
//    than the pivot and the right scan at the k-th element not greater than
//    it, so the swap pairs, their count and the cut follow from two ordered
//    lists made with ballots; disjoint segments are partitioned by different
//    warps at the same time; segments left at <= 16 elements get the final
//    insertion sort independently (no element crosses a partition cut,
//    because every element left of a cut is not greater than any right of
//    it and the insertion only moves past strictly greater elements), as a
//    stable rank within the segment, a thread per element.
#pragma once

#include "heap_merge.cuh"
#include "huffman_build.cuh"

namespace ccb {
namespace tb {

// ---------------------------------------------------------------------------
// Tree (HuffmanTable.cu:507-529): probabilities P and ids I of heap_merge.cuh's
// layout, 1-based (node k holds heap element k - 1).  "less(a, b)" is b.prob <
// a.prob (the top is the smallest probability; ties are not broken by id, so
// the result depends on the exact libstdc++ heap moves, which are replayed).
// ---------------------------------------------------------------------------

// make_heap (libstdc++ __make_heap): __adjust_heap of every parent from
// len / 2 down to 1.  Parents at one depth have disjoint subtrees and all
// deeper parents come first in that order, so the parents of one depth are
// adjusted in parallel, deepest depth first, with the same result.  The hole
// of an adjustment sinks along the smaller children and the value rises again
// from the leaf; that path ascends, so stopping at the first child above the
// value places it the same.  All threads of the block.
__device__ void blockMakeHeap(u32* P, u32* I, u32 len) {
    for (int d = 31 - __clz(len / 2); d >= 0; --d) {
        const u32 first = 1u << d, last = min(2u * first - 1u, len / 2u);
        for (u32 node = first + threadIdx.x; node <= last; node += blockDim.x) {
            const u32 v = P[node];
            const u32 id = I[node];
            u32 hole = node;
            while (2u * hole <= len) {
                u32 c = 2u * hole;
                if (c < len && !(P[c] < P[c + 1])) ++c;   // the right child unless the left is strictly smaller
                const u32 cp = P[c];
                if (v < cp) break;
                P[hole] = cp;
                I[hole] = I[c];
                hole = c;
            }
            P[hole] = v;
            I[hole] = id;
        }
        __syncthreads();
    }
}

// The tails (x 4) of a heap: the bottom end of every node's path of smaller
// children.
__device__ void blockTails(const u32* P, u32* T, u32 len) {
    const u32 D = hm::log2Floor(len);
    for (int d = int(D); d >= 0; --d) {
        const u32 first = 1u << d, last = min(2u * first - 1u, len);
        for (u32 node = first + threadIdx.x; node <= last; node += blockDim.x) {
            const u32 c = 2u * node;
            T[node] = c > len ? 4u * (node << (D - d)) : (c == len || P[c] < P[c + 1]) ? T[c] : T[c + 1];
        }
        __syncthreads();
    }
}

// The tree of 2 <= L <= kCap leaves (P and I of nodes 1 .. L in symbol order,
// in the block's dynamic shared memory): parent links in the layout's parents.
// All threads of the block.
template <u32 kCap>
__device__ void blockBuildTree(unsigned char* dyn, u32 L) {
    using At = hm::Layout<kCap>;
    u32* P = reinterpret_cast<u32*>(dyn);
    for (u32 i = L + 1 + threadIdx.x; i < (2u << hm::log2Floor(L)); i += blockDim.x) P[i] = hm::kInf;
    if (threadIdx.x < 2) P[At::kNodes + threadIdx.x] = hm::kInf;
    if (threadIdx.x == 0) P[0] = hm::kInf;
    blockMakeHeap(P, reinterpret_cast<u32*>(dyn + At::kIds), L);
    blockTails(P, reinterpret_cast<u32*>(dyn + At::kTails), L);
    if (threadIdx.x < 32) {
        hm::Merge<hm::DeviceWarp, kCap> m(hm::DeviceWarp(), L);
        m.run(L);
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Sort (HuffmanTable.cu:538, libstdc++ std::sort) of keys (len << 27 | leaf).
// ---------------------------------------------------------------------------
struct Seg {
    u16 f, l;
    int d;
};
constexpr int kSortThreshold = 16;

__device__ __forceinline__ u32 keyOf(u32 v) { return v >> 27; }

// Exact replay of __unguarded_partition(a + f + 1, a + l, a + f) by one warp.
// lList / rList: scratch positions for [f, l) (entries f .. l-1 are used).
__device__ int warpPartition(u32* a, int f, int l, u16* lList, u16* rList) {
    const u32 lane = threadIdx.x & 31u;
    const u32 ltMask = (1u << lane) - 1u;
    const u32 p = keyOf(a[f]);
    int nL = 0, nR = 0;
    // four groups of 32 per step, their loads in flight together
    for (int base = f + 1; base < l; base += 128) {
        bool pred[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int j = base + 32 * q + int(lane);
            pred[q] = j < l && !(keyOf(a[min(j, l - 1)]) < p);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const u32 m = __ballot_sync(0xffffffffu, pred[q]);
            if (pred[q]) lList[f + nL + __popc(m & ltMask)] = u16(base + 32 * q + int(lane));
            nL += __popc(m);
        }
    }
    for (int top = l - 1; top > f; top -= 128) {
        bool pred[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int j = top - 32 * q - int(lane);
            pred[q] = j > f && !(p < keyOf(a[max(j, f)]));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const u32 m = __ballot_sync(0xffffffffu, pred[q]);
            if (pred[q]) rList[f + nR + __popc(m & ltMask)] = u16(top - 32 * q - int(lane));
            nR += __popc(m);
        }
    }
    __syncwarp();
    // K = number of leading k with lList[k] < rList[k] (monotone in k)
    const int kMax = min(nL, nR);
    int K = 0;
    for (int base = 0; base < kMax; base += 32) {
        const int k = base + int(lane);
        const bool ok = k < kMax && lList[f + k] < rList[f + k];
        const u32 m = __ballot_sync(0xffffffffu, ok);
        const int run = (m == 0xffffffffu) ? 32 : __ffs(~m) - 1;
        K += run;
        if (run < 32) break;
    }
    // swaps (disjoint positions)
    for (int k = int(lane); k < K; k += 32) {
        const int x = lList[f + k], y = rList[f + k];
        const u32 t = a[x];
        a[x] = a[y];
        a[y] = t;
    }
    int cut;
    if (K == 0) cut = lList[f];
    else cut = min(K < nL ? int(lList[f + K]) : 0x7fffffff, int(rList[f + K - 1]));
    __syncwarp();
    return cut;
}

// Block-cooperative introsort of a[0, n) (n <= 16384) into out[0, n).
// Scratch: lList, rList (n u16 each; out may take their place), seg (n words),
// two segment queues.  All threads call it.
template <int kThreads>
__device__ void blockIntrosort(u32* a, int n, u16* lList, u16* rList, u32* seg, Seg* qA, Seg* qB, int* counters,
                               u32* out) {
    constexpr int kWarps = kThreads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // seg: first element | length << 16 of each element's final segment
    if (n <= kSortThreshold)
        for (int i = threadIdx.x; i < n; i += kThreads) seg[i] = u32(n) << 16;
    if (threadIdx.x == 0) {
        counters[0] = 0;
        if (n > kSortThreshold) {
            qA[0] = Seg{0, u16(n), 2 * hb::floorLog2(n)};
            counters[0] = 1;
        }
    }
    __syncthreads();
    Seg* cur = qA;
    Seg* nxt = qB;
    int nCur = counters[0];
    while (nCur > 0) {
        // counters[1] counts the next round's segments.  Its reset comes
        // after the barrier that ends the previous round's reads of it (the
        // third barrier below), and the barrier after the reset orders it
        // before this round's additions.
        if (threadIdx.x == 0) counters[1] = 0;
        __syncthreads();
        for (int s = warp; s < nCur; s += kWarps) {
            const Seg g = cur[s];
            if (g.d == 0) {
                if (lane == 0) {
                    hb::makeHeap(a + g.f, g.l - g.f, hb::LenLess());
                    hb::sortHeap(a + g.f, g.l - g.f, hb::LenLess());
                }
                // sorted: segments of one element
                for (int i = g.f + lane; i < g.l; i += 32) seg[i] = u32(i) | (1u << 16);
                __syncwarp();
                continue;
            }
            if (lane == 0) hb::moveMedianToFirst(a, g.f, g.f + 1, g.f + (g.l - g.f) / 2, g.l - 1, hb::LenLess());
            __syncwarp();
            const int cut = warpPartition(a, g.f, g.l, lList, rList);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int f = k ? cut : g.f, l = k ? int(g.l) : cut;
                if (l - f > kSortThreshold) {
                    if (lane == 0) nxt[atomicAdd(&counters[1], 1)] = Seg{u16(f), u16(l), g.d - 1};
                } else if (lane < l - f) {
                    seg[f + lane] = u32(f) | (u32(l - f) << 16);
                }
            }
            __syncwarp();
        }
        __syncthreads();
        nCur = counters[1];
        __syncthreads();   // every thread has read the count before thread 0 resets it
        Seg* t = cur;
        cur = nxt;
        nxt = t;
    }
    // The final insertion sort is stable (an element moves past strictly
    // greater ones only) and stays within its segment of at most 16 elements:
    // an element's place is the number of smaller ones, and of equal ones
    // before it.  A thread per element: 16 independent loads, where one thread
    // per segment moves up to 120 elements one after the other.  With the code
    // lengths' scan and the header's lengths on a warp's lanes, the tables of
    // a 2048^2 heightfield and back (up to 8000 leaves): 1.82 -> 1.58 ms the
    // case; of a 128^3 volume 428 -> 406 us.
    for (int i = threadIdx.x; i < n; i += kThreads) {
        const u32 v = a[i], g = seg[i], key = keyOf(v);
        const int f = int(g & 0xFFFFu), len = int(g >> 16), me = i - f;
        int to = f;
#pragma unroll
        for (int j = 0; j < kSortThreshold; ++j) {
            const u32 other = keyOf(a[f + min(j, len - 1)]);
            to += j < len && (other < key || (other == key && j < me)) ? 1 : 0;
        }
        out[to] = v;
    }
    __syncthreads();
}

}  // namespace tb
}  // namespace ccb
