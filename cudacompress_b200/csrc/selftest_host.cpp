// selftest_host.cpp - host build of the table constructor in huffman_build.cuh,
// exported for the CPU unit tests (tests/test_table_build_host.py), which
// compare it with the oracle on many histograms.  Not part of the product
// library: it is built into _lib/libcc_selftest.so and loaded only by tests.
#include <algorithm>
#include <cstring>
#include <vector>
#include "heap_merge.cuh"
#include "huffman_build.cuh"

using namespace ccb;

namespace {

// heap_merge.cuh's warp as 32-element arrays over a bounds-checked memory.
struct LaneU { u32 v[32]; };
struct LaneB { bool v[32]; };

struct HostWarp {
    using U = LaneU;
    using B = LaneB;
    u8* mem;
    u32 bytes;
    bool* bad;
    template <class F> static U each(F f) { U r; for (u32 i = 0; i < 32; ++i) r.v[i] = f(i); return r; }
    template <class F> static B test(F f) { B r; for (u32 i = 0; i < 32; ++i) r.v[i] = f(i); return r; }
    U lane() const { return each([](u32 i) { return i; }); }
    U all(u32 x) const { return each([=](u32) { return x; }); }
    u32 first(const U& a) const { return a.v[0]; }
    B le(const U& a, const U& b) const { return test([&](u32 i) { return a.v[i] <= b.v[i]; }); }
    B lt(const U& a, const U& b) const { return test([&](u32 i) { return a.v[i] < b.v[i]; }); }
    B eq(const U& a, const U& b) const { return test([&](u32 i) { return a.v[i] == b.v[i]; }); }
    B nz(const U& a) const { return test([&](u32 i) { return a.v[i] != 0; }); }
    B both(const B& a, const B& b) const { return test([&](u32 i) { return a.v[i] && b.v[i]; }); }
    U sel(const B& c, const U& a, const U& b) const { return each([&](u32 i) { return c.v[i] ? a.v[i] : b.v[i]; }); }
    U min(const U& a, const U& b) const { return each([&](u32 i) { return std::min(a.v[i], b.v[i]); }); }
    U max(const U& a, const U& b) const { return each([&](u32 i) { return std::max(a.v[i], b.v[i]); }); }
    U sub(const U& a, const U& b) const { return each([&](u32 i) { return a.v[i] - b.v[i]; }); }
    U add(const U& a, const U& b) const { return each([&](u32 i) { return a.v[i] + b.v[i]; }); }
    U shr(const U& a, const U& n) const { return each([&](u32 i) { return a.v[i] >> n.v[i]; }); }
    U shr(const U& a, u32 n) const { return each([&](u32 i) { return a.v[i] >> n; }); }
    U shl(const U& a, u32 n) const { return each([&](u32 i) { return a.v[i] << n; }); }
    U shlv(const U& a, const U& n) const { return each([&](u32 i) { return a.v[i] << n.v[i]; }); }
    U min3(const U& a, const U& b, const U& c) const { return min(a, min(b, c)); }
    U below(const U& a) const { return each([&](u32 i) { return a.v[i] - 1u + (a.v[i] >> 31); }); }
    U andv(const U& a, const U& b) const { return each([&](u32 i) { return a.v[i] & b.v[i]; }); }
    U orv(const U& a, const U& b) const { return each([&](u32 i) { return a.v[i] | b.v[i]; }); }
    U xorv(const U& a, const U& b) const { return each([&](u32 i) { return a.v[i] ^ b.v[i]; }); }
    U lastSet(const U& m) const { return each([&](u32 i) { return m.v[i] ? 31u - u32(__builtin_clz(m.v[i])) : ~0u; }); }
    u32 ballot(const B& c) const { u32 m = 0; for (u32 i = 0; i < 32; ++i) m |= u32(c.v[i]) << i; return m; }
    u32 reduceMin(const U& a) const { return *std::min_element(a.v, a.v + 32); }
    U shfl(const U& a, const U& from) const { return each([&](u32 i) { return a.v[from.v[i] & 31u]; }); }
    void fence() const {}
    template <class T> T* at(u32 off) const {
        static u64 sink;
        if (u64(off) + sizeof(T) > bytes || off % sizeof(T)) { *bad = true; return reinterpret_cast<T*>(&sink); }
        return reinterpret_cast<T*>(mem + off);
    }
    template <u32 A> void ldPair(const U& o, U& x, U& y) const {
        for (u32 i = 0; i < 32; ++i) if ((A + o.v[i]) % 8) *bad = true;
        x = ld<A>(o);
        y = ld<A + 4u>(o);
    }
    template <u32 A> U ld(const U& o) const { return each([&](u32 i) { return *at<u32>(A + o.v[i]); }); }
    template <u32 A> u32 ldOne(u32 o) const { return *at<u32>(A + o); }
    template <u32 A> void st(const U& o, const U& x, const B& c) const {
        for (u32 i = 0; i < 32; ++i) if (c.v[i]) *at<u32>(A + o.v[i]) = x.v[i];
    }
    template <u32 A> void stAll(u32 o, u32 x) const { *at<u32>(A + o) = x; }
    template <u32 A> void stParent(const U& id2, u32 x) const { *at<u16>(A + id2.v[31]) = u16(x); }
};

}  // namespace

// The warp's merge loop over a heap of L leaves in a layout of kCap.
template <u32 kCap>
static bool warpMerge(const std::vector<u64>& heap, u32 L, u32* parents) {
    using At = hm::Layout<kCap>;
    std::vector<u64> area(At::kBytes / 8 + 1, 0xAAAAAAAAAAAAAAAAull);
    u8* m = reinterpret_cast<u8*>(area.data());
    u32* P = reinterpret_cast<u32*>(m);
    u32* I = reinterpret_cast<u32*>(m + At::kIds);
    u32* T = reinterpret_cast<u32*>(m + At::kTails);
    const u16* up = reinterpret_cast<const u16*>(m + At::kParents);
    const u32 D = hm::log2Floor(L);
    for (u32 i = 0; i < (2u << D); ++i) P[i] = hm::kInf;
    P[At::kNodes] = P[At::kNodes + 1] = hm::kInf;
    for (u32 i = 0; i < L; ++i) { P[i + 1] = u32(heap[i] >> 32); I[i + 1] = 2u * u32(heap[i]); }
    for (u32 k = L; k >= 1; --k) {
        const u32 c = 2 * k;
        T[k] = c > L ? 4u * (k << (D - hm::log2Floor(k))) : (c == L || P[c] < P[c + 1]) ? T[c] : T[c + 1];
    }
    bool bad = false;
    hm::Merge<HostWarp, kCap> merge(HostWarp{m, At::kBytes, &bad}, L);
    merge.run(L);
    for (u32 i = 0; i + 2 < 2 * L; ++i) parents[i] = up[i];
    return bad;
}

// Parent links of the tree over L >= 2 leaf probabilities, by the warp's merge
// loop in a layout of `cap` leaves (warpParents) and by the sequential
// libstdc++ replay (seqParents); 0, -1 after an access outside the layout's
// area, -2 for a capacity that is not built.
extern "C" int ccst_heap_merge(const u32* probs, u32 L, u32 cap, u32* warpParents, u32* seqParents) {
    std::vector<u64> heap(L);
    for (u32 i = 0; i < L; ++i) heap[i] = (u64(probs[i]) << 32) | i;
    std::vector<u64> seq(heap);
    std::vector<u32> par(2 * L, 0);
    hb::buildTree(seq.data(), par.data(), int(L));
    std::memcpy(seqParents, par.data(), sizeof(u32) * (2 * L - 2));
    hb::makeHeap(heap.data(), int(L), hb::ProbInvLess());
    if (L > cap) return -2;
    switch (cap) {
        case 256: return -int(warpMerge<256>(heap, L, warpParents));
        case 1024: return -int(warpMerge<1024>(heap, L, warpParents));
        case 2048: return -int(warpMerge<2048>(heap, L, warpParents));
        case 12288: return -int(warpMerge<12288>(heap, L, warpParents));
        default: return -2;
    }
}

extern "C" int ccst_huffman_build(const u32* hist, u32 bins, u32 symbolMax, u32 log2Max, u32* codewords,
                                  u32* lengths, u32* tableWords, u32 cap, u32* tableBits) {
    std::vector<u32> leafSym, leafProb;
    for (u32 s = 0; s < bins; ++s)
        if (hist[s]) { leafSym.push_back(s); leafProb.push_back(hist[s]); }
    int L = int(leafSym.size());
    for (u32 i = 0; i < bins; ++i) { codewords[i] = 0; lengths[i] = 0xFFFFFFFFu; }
    u32 lenCount[32] = {0};
    int maxLen = 0;
    std::vector<u32> sorted(L);
    if (L > 0) {
        std::vector<u64> heap(L);
        std::vector<u32> parent(2 * L);
        std::vector<u8> depth(2 * L);
        for (int i = 0; i < L; ++i) heap[i] = (u64(leafProb[i]) << 32) | u32(i);
        hb::buildTree(heap.data(), parent.data(), L);
        hb::nodeDepths(parent.data(), depth.data(), L);
        std::vector<u32> order(L);
        for (int i = 0; i < L; ++i) {
            order[i] = (u32(depth[i]) << 27) | u32(i);
            if (depth[i] > maxLen) maxLen = depth[i];
        }
        if (maxLen > 31) return -5;
        hb::introsort(order.data(), L, hb::LenLess());
        u32 code = 0, prevLen = 0;
        for (int k = 0; k < L; ++k) {
            u32 len = order[k] >> 27;
            u32 sym = leafSym[order[k] & hb::kLeafMask];
            if (k > 0) code = (code + 1) << (len - prevLen);
            prevLen = len;
            if (len) lenCount[len - 1]++;
            sorted[k] = sym;
            codewords[sym] = code;
            lengths[sym] = len;
        }
    }
    // serialization as HuffmanTable.cu:470-485
    std::vector<u32> w;
    u32 pos = 0;
    auto put = [&](u32 v, u32 n) {
        for (u32 b = 0; b < n; ++b, ++pos) {
            if (pos / 32 >= w.size()) w.push_back(0);
            if ((v >> (n - 1 - b)) & 1u) w[pos / 32] |= 1u << (31 - pos % 32);
        }
    };
    bool longSym = log2Max > 16;
    put(u32(maxLen), 5);
    for (int l = 0; l < maxLen; ++l) put(lenCount[l], log2Max);
    put(u32(L), log2Max);
    u32 symbolBits = requiredBits(symbolMax);
    put(symbolBits, longSym ? 5 : 4);
    for (int k = 0; k < L; ++k) put(sorted[k], symbolBits);
    *tableBits = pos;
    if (w.size() > cap) return -2;
    std::memcpy(tableWords, w.data(), w.size() * 4);
    return maxLen;
}
