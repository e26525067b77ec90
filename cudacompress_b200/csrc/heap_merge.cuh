// heap_merge.cuh - the merge loop of the Huffman tree construction
// (HuffmanTable.cu:507-529) on one warp, with exactly the element moves of
// libstdc++'s pop_heap / push_heap, so that ties are resolved as the
// reference's std::priority_queue resolves them.
//
// The loop is a chain: every merge pops two elements and pushes their sum,
// and a one-thread replay pays a dependent shared-memory load and a select
// per heap level (1640 cycles per merge at 2000 leaves, 1880 at 8000).  Here
// a lane holds a level, so an operation costs one round of loads whatever the
// depth.  Three facts make that exact:
//  * pop_heap moves the hole along the path of smaller children to a leaf and
//    sifts the last element v up from there.  The path's values ascend, so
//    the outcome is: path elements <= v move up one level, v stands below the
//    last of them.  The node of level d gets clamp(v, x[d], x[d+1]), x being
//    the old path.
//  * push_heap of c at position q shifts the ancestors of q that are > c down
//    one level: the node of level d gets clamp(c, e[d-1], e[d]).
//  * each node keeps the bottom end of its own path of smaller children
//    (its tail, a node number at the tree's full depth D: the path's node at
//    level d is tail >> (D - d)), so the next pop's path is known without
//    descending.  After an operation the tail of a path node is the tail of
//    the first sibling below it that became the smaller child, else the path
//    itself: for the root that is one minimum over the lanes' (level, tail).
//
// Measured on B200 (cycles per merge, one table alone on an SM): 457 at every
// size, where the one-thread replay took 1374 at 406 leaves, 1643 at 2012 and
// 1883 at 8192.  What bounds it is the chain of one operation - minimum over
// the lanes (24 cycles), pair loads (30 and up), clamp, compare - three times
// per merge: without the tails' upkeep it takes 365.  Nodes of 8 bytes, whose
// pair is one 16-byte load, took 574 (fewer instructions, but slower loads and
// stores); tails stored before the next operation's loads 619.
//
// Shared layout, nodes 1-based (node k's children are 2k and 2k + 1): the
// probabilities (a pair of children is one 8-byte load; node 0's is kInf), the
// ids and the tails, and the parent links.  Removing the last element leaves
// the tails of its ancestors that end in it pointing at a missing right child:
// every level therefore takes the smaller of the pair it loads, and a tail's
// last step - below which there are no elements - does not matter.
//
// W supplies the warp: lane vectors of 32-bit words and conditions, warp-wide
// minimum, ballot and shuffle, and shared-memory access (the device's own
// registers, or 32-element arrays with bounds checks in the host self-test).
#pragma once

#include "cc_common.cuh"

namespace ccb {
namespace hm {

constexpr u32 kMergeLeavesMax = 16384;  // ids and tails take 16 bits
constexpr u32 kInf = 0x7FFFFFFFu;       // probabilities and their sum are below it
constexpr u32 kKeyLevel = 18;           // a key: level << kKeyLevel | tail << 2
constexpr u32 kKeyTail = (1u << kKeyLevel) - 1u;
constexpr u32 kNoKey = 0x7Fu << kKeyLevel;   // | tail << 2: above every level's

CC_HD u32 log2Floor(u32 v) { return 31u - u32(__builtin_clz(v)); }

// Byte offsets of the arrays for a capacity of `leaves`.  Loads of missing
// nodes reach up to node 2^(D+1) - 1 < 2 leaves of each array: inside the
// whole area, their values unused.
struct Layout {
    u32 ids, tails, parents, bytes;
    CC_HD explicit Layout(u32 leaves) {
        const u32 n = (leaves + 3u) & ~1u;   // nodes 0 .. leaves, even
        ids = 4u * n;
        tails = ids + 2u * n;
        parents = tails + 2u * n;
        bytes = parents + 4u * n;
    }
};

template <class W>
struct Merge {
    using U = typename W::U;
    using B = typename W::B;

    W w;
    Layout at;
    u32 D;            // depth of the deepest level
    U level, sh, shChild;             // the lane's level; shifts from a key to byte offsets
    U pairMask, nodeMask, childMask;  // of a shifted key: 4 x the node's pair, 4 x node, 8 x node
    U outside, outsideChild;          // large where the lane has no node, or no children
    U deeper;         // mask of the lanes of deeper levels
    U upBound;        // the root has nothing above it
    B notTop;

    // An operation's loads.
    struct Loads {
        U px, py;     // the pair of the lane's node
        U nx, ny;     // pop: the pair below the node; push: nx the node above
        U ids;        // pop: the ids of that pair; push: the id of the node above
        U node4, sibTail;
        U child8;
        u32 tail4, v, idv;
    };
    // What its moves leave: whether the sibling is the smaller child now, its
    // tail, the lane's key and the path's end; the winners' ballot, and the
    // tails on their way to their array.  rootP, rootId: the root lane's
    // element.
    struct Path {
        U node4, sibTail, key, from, newTail;
        B holds, win;
        u32 tail4, winners;
    };
    U rootP, rootId;

    // The lanes run from the deepest level up (lane 31 is the root's), so that
    // the nearest winner below a level is a highest set bit.
    CC_HD Merge(W w_, u32 leavesCap, u32 L) : w(w_), at(leavesCap), D(log2Floor(L)) {
        level = w.sub(w.all(31u), w.lane());
        const B act = w.le(level, w.all(D));
        const B inner = w.lt(level, w.all(D));
        notTop = w.both(act, w.lt(w.all(0u), level));
        sh = w.sel(act, w.sub(w.all(D), level), w.all(31u));
        shChild = w.sel(inner, w.sub(w.all(D), w.add(level, w.all(1u))), w.all(31u));
        const U nodes = w.sel(act, w.sub(w.shlv(w.all(2u), w.sel(act, level, w.all(0u))), w.all(1u)), w.all(0u));
        nodeMask = w.shl(nodes, 2u);
        pairMask = w.andv(nodeMask, w.all(~7u));
        childMask = w.sel(inner, w.shl(nodes, 3u), w.all(0u));
        outside = w.sel(act, w.all(0u), w.all(1u << 30));
        outsideChild = w.sel(inner, w.all(0u), w.all(1u << 30));
        deeper = w.sub(w.shlv(w.all(1u), w.lane()), w.all(1u));
        upBound = w.sel(notTop, w.all(kInf), w.all(0u));
    }

    // The last element of a heap of n + 1.
    CC_HD void lastElement(Loads& l, u32 n) {
        l.v = w.ldOne32(4u * (n + 1));
        l.idv = w.ldOne16(at.ids + 2u * (n + 1));
    }

    // key: the previous operation's minimum.
    CC_HD void popLoads(Loads& l, u32 key) {
        const U t = w.shr(w.all(key), sh);
        const U pair4 = w.andv(t, pairMask);
        l.child8 = w.andv(w.shr(w.all(key), shChild), childMask);
        w.ldPair(pair4, l.px, l.py);
        w.ldPair(l.child8, l.nx, l.ny);
        l.node4 = w.andv(t, nodeMask);
        l.ids = w.ld16Pair(at.ids, w.shr(l.child8, 1u));
        l.sibTail = w.ld16(at.tails, w.xorv(w.shr(l.node4, 1u), w.all(2u)));
        l.tail4 = key & kKeyTail;
    }

    // The moves of a pop that leaves n elements.  fwdLevel / fwdTail4: the
    // tail of the node at which this path and the previous operation's part
    // (not stored yet); prev: that operation, whose tails are stored here.
    CC_HD void popMove(const Loads& l, u32 n, u32 fwdLevel, u32 fwdTail4, const Path& prev, Path& p) {
        const U n4 = w.all(4u * n);
        const U left4 = w.orv(w.andv(l.node4, w.all(~4u)), outside);
        const U kid4 = w.orv(l.child8, outsideChild);
        const U px = w.sel(w.le(left4, n4), l.px, w.all(kInf));
        const U py = w.sel(w.lt(left4, n4), l.py, w.all(kInf));
        const U nx = w.sel(w.le(kid4, n4), l.nx, w.all(kInf));
        const U ny = w.sel(w.lt(kid4, n4), l.ny, w.all(kInf));
        const U x = w.min(px, py), xn = w.min(nx, ny);
        const U v = w.all(l.v);
        const U y = w.max(x, w.min(v, xn));
        const B isLeft = w.lt(px, py);
        const U kk4 = w.add(left4, w.sel(isLeft, w.all(0u), w.all(4u)));
        const B moved = w.le(x, v);
        const U id = w.sel(w.le(xn, v), w.sel(w.lt(nx, ny), w.lo16(l.ids), w.hi16(l.ids)), w.all(l.idv));
        w.fence();
        w.st32(kk4, y, moved);
        w.st16(at.ids, w.shr(kk4, 1u), id, moved);
        tailsStore(prev);
        w.fence();
        rootP = y;
        rootId = id;
        // the sibling wins a left node's place on a tie too
        finish(l, n, y, w.sel(isLeft, w.sub(py, w.all(1u)), px), fwdLevel, fwdTail4, p);
    }

    CC_HD void finish(const Loads& l, u32 n, const U& y, const U& s, u32 fwdLevel, u32 fwdTail4, Path& p) {
        p.sibTail = w.sel(w.eq(level, w.all(fwdLevel)), w.all(fwdTail4), w.shl(l.sibTail, 2u));
        p.win = w.lt(s, y);
        p.key = w.sel(p.win, w.orv(w.shl(level, kKeyLevel), p.sibTail), w.all(kNoKey | l.tail4));
        p.node4 = l.node4;
        p.holds = w.le(w.orv(l.node4, outside), w.all(4u * n));
        p.tail4 = l.tail4;
    }

    // Loads of a push whose path ends in tail4 / 4.
    CC_HD void pushLoads(Loads& l, u32 tail4) {
        const U t = w.shr(w.all(tail4), sh);
        l.node4 = w.andv(t, nodeMask);
        const U up4 = w.andv(w.shr(t, 1u), w.shr(nodeMask, 1u));
        w.ldPair(w.andv(t, pairMask), l.px, l.py);
        l.nx = w.ld32(w.andv(up4, w.all(~3u)));
        l.ids = w.ld16(at.ids, w.andv(w.shr(up4, 1u), w.all(~1u)));
        l.sibTail = w.ld16(at.tails, w.xorv(w.shr(l.node4, 1u), w.all(2u)));
        l.tail4 = tail4;
    }

    // The moves of a push of c at position q.
    CC_HD void pushMove(const Loads& l, u32 q, u32 c, u32 id, u32 fwdLevel, u32 fwdTail4, const Path& prev, Path& p) {
        const U q4 = w.all(4u * q);
        const U node4 = w.orv(l.node4, outside);
        const B odd = w.nz(w.andv(l.node4, w.all(4u)));
        const B above = w.lt(node4, q4);   // held an element before the push; a left node: has a sibling
        const U e = w.sel(above, w.sel(odd, l.py, l.px), w.all(kInf));
        const U up = w.sel(w.both(notTop, w.le(node4, w.all(4u * q))), l.nx, upBound);
        const U cv = w.all(c);
        const U y = w.max(up, w.min(cv, e));
        const B moved = w.both(w.le(node4, q4), w.lt(cv, e));
        const U newId = w.sel(w.lt(cv, up), l.ids, w.all(id));
        w.fence();
        w.st32(node4, y, moved);
        w.st16(at.ids, w.shr(node4, 1u), newId, moved);
        tailsStore(prev);
        w.fence();
        rootP = y;
        rootId = w.sel(moved, newId, rootId);
        const U right = w.sel(above, w.sub(l.py, w.all(1u)), w.all(kInf));
        finish(l, q, y, w.sel(odd, l.px, right), fwdLevel, fwdTail4, p);
    }

    // Tails of an operation's path nodes, while the next operation waits for
    // its loads: the nearest winning sibling below each node, and its tail
    // (else the path's end).
    CC_HD void tailsFind(Path& p) {
        p.from = w.andv(w.all(p.winners), deeper);
        p.newTail = w.shfl(p.sibTail, w.lastSet(p.from));
    }
    CC_HD void tailsStore(const Path& p) {
        w.st16(at.tails, w.shr(p.node4, 1u), w.shr(w.sel(w.nz(p.from), p.newTail, w.all(p.tail4)), 2u), p.holds);
    }
    // The minimum over the keys after r.
    CC_HD u32 keyAfter(u32 r, const Path& p) {
        return w.reduceMin(w.sel(w.lt(w.all(r), p.key), p.key, w.all(kNoKey | p.tail4)));
    }

    // Merges the heap of L >= 2 elements (probability kInf at node 0; the
    // three arrays set up for nodes 1 .. L); writes the parent of every id but
    // the root's (2L - 2).
    CC_HD void run(u32 L) {
        Path pa, pb, pc;
        // an operation before the first: no winners, nothing to store
        pc.tail4 = 4u * w.ldOne16(at.tails + 2u);
        pc.node4 = w.all(0u);
        pc.sibTail = w.all(0u);
        pc.holds = w.lt(w.all(1u), w.all(0u));
        pc.winners = 0;
        pc.key = w.all(kNoKey | pc.tail4);
        rootP = w.all(w.ldOne32(4u));
        rootId = w.all(w.ldOne16(at.ids + 2u));
        u32 rc = kNoKey | pc.tail4;
        u32 next = L;
        u32 qDepth = D;   // depth of the push's position
        Loads l;
        lastElement(l, L - 1);
        for (u32 len = L; len > 1; --len, ++next) {
            const u32 q = len - 1;
            if (q < (1u << qDepth)) --qDepth;
            const u32 tailC = 4u * q << (D - qDepth);

            popLoads(l, rc);
            const u32 rc2 = keyAfter(rc, pc);
            tailsFind(pc);
            w.stParent(at.parents, rootId, next);
            U c = rootP;
            popMove(l, len - 1, rc >> kKeyLevel, rc2 & kKeyTail, pc, pa);
            lastElement(l, len - 2);
            const u32 ra = w.reduceMin(pa.key);
            pa.winners = w.ballot(pa.win);

            popLoads(l, ra);
            const u32 ra2 = keyAfter(ra, pa);
            w.stParent(at.parents, rootId, next);
            c = w.shfl(w.add(c, rootP), w.all(31u));
            tailsFind(pa);
            // the level at which the push's path leaves this pop's
            const u32 diff = (tailC ^ l.tail4) >> 2;
            const u32 h = diff ? D - log2Floor(diff) : 0x7Eu;
            popMove(l, len - 2, ra >> kKeyLevel, ra2 & kKeyTail, pa, pb);

            pushLoads(l, tailC);
            pb.winners = w.ballot(pb.win);
            const u32 rb2 = keyAfter((h << kKeyLevel) | kKeyTail, pb);
            tailsFind(pb);
            pushMove(l, q, w.first(c), next, h, rb2 & kKeyTail, pb, pc);
            lastElement(l, len - 2);
            rc = w.reduceMin(pc.key);
            pc.winners = w.ballot(pc.win);
        }
    }
};

#ifdef __CUDACC__
// The calling warp: a lane vector is the lane's own register; memory is the
// shared window from byte address `base`.
struct DeviceWarp {
    using U = u32;
    using B = bool;
    u32 base;
    __device__ __forceinline__ explicit DeviceWarp(const void* shared) : base(u32(__cvta_generic_to_shared(shared))) {}
    __device__ __forceinline__ u32 lane() const { return threadIdx.x & 31u; }
    __device__ __forceinline__ u32 all(u32 v) const { return v; }
    __device__ __forceinline__ u32 first(u32 v) const { return v; }
    __device__ __forceinline__ bool le(u32 a, u32 b) const { return a <= b; }
    __device__ __forceinline__ bool lt(u32 a, u32 b) const { return a < b; }
    __device__ __forceinline__ bool eq(u32 a, u32 b) const { return a == b; }
    __device__ __forceinline__ bool nz(u32 a) const { return a != 0; }
    __device__ __forceinline__ bool both(bool a, bool b) const { return a && b; }
    __device__ __forceinline__ u32 sel(bool c, u32 a, u32 b) const { return c ? a : b; }
    __device__ __forceinline__ u32 min(u32 a, u32 b) const { return a < b ? a : b; }
    __device__ __forceinline__ u32 max(u32 a, u32 b) const { return a > b ? a : b; }
    __device__ __forceinline__ u32 sub(u32 a, u32 b) const { return a - b; }
    __device__ __forceinline__ u32 add(u32 a, u32 b) const { return a + b; }
    __device__ __forceinline__ u32 shr(u32 a, u32 n) const { return a >> n; }
    __device__ __forceinline__ u32 shl(u32 a, u32 n) const { return a << n; }
    __device__ __forceinline__ u32 shlv(u32 a, u32 n) const { return a << n; }
    __device__ __forceinline__ u32 lo16(u32 a) const { return a & 0xFFFFu; }
    __device__ __forceinline__ u32 hi16(u32 a) const { return a >> 16; }
    __device__ __forceinline__ u32 andv(u32 a, u32 b) const { return a & b; }
    __device__ __forceinline__ u32 orv(u32 a, u32 b) const { return a | b; }
    __device__ __forceinline__ u32 xorv(u32 a, u32 b) const { return a ^ b; }
    __device__ __forceinline__ u32 lastSet(u32 m) const { return 31u - u32(__clz(int(m))); }
    __device__ __forceinline__ u32 ballot(bool c) const { return __ballot_sync(0xffffffffu, c); }
    __device__ __forceinline__ u32 reduceMin(u32 v) const { return __reduce_min_sync(0xffffffffu, v); }
    __device__ __forceinline__ u32 shfl(u32 v, u32 from) const { return __shfl_sync(0xffffffffu, v, int(from)); }
    __device__ __forceinline__ void fence() const { __syncwarp(); }
    __device__ __forceinline__ void ldPair(u32 off, u32& x, u32& y) const {
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(base + off) : "memory");
    }
    __device__ __forceinline__ u32 ld32(u32 off) const {
        u32 x;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(base + off) : "memory");
        return x;
    }
    __device__ __forceinline__ u32 ld16(u32 array, u32 off) const {
        u16 x;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(base + array + off) : "memory");
        return x;
    }
    __device__ __forceinline__ u32 ld16Pair(u32 array, u32 off) const { return ld32(array + off); }
    __device__ __forceinline__ u32 ldOne32(u32 off) const { return ld32(off); }
    __device__ __forceinline__ u32 ldOne16(u32 off) const { return ld16(0, off); }
    __device__ __forceinline__ void st32(u32 off, u32 v, bool c) const {
        asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u32 [%0], %1;\n}"
                     :: "r"(base + off), "r"(v), "r"(u32(c)) : "memory");
    }
    __device__ __forceinline__ void st16(u32 array, u32 off, u32 v, bool c) const {
        asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u16 [%0], %1;\n}"
                     :: "r"(base + array + off), "h"(u16(v)), "r"(u32(c)) : "memory");
    }
    // by the root's lane
    __device__ __forceinline__ void stParent(u32 array, u32 id, u32 v) const { st16(array, 2u * id, v, lane() == 31u); }
};
#endif

}  // namespace hm
}  // namespace ccb
