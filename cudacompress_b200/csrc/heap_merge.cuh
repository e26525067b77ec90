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
// Measured on B200 (cycles per merge, one table alone on an SM): 350 at every
// size, where a one-thread replay took 1374 at 406 leaves, 1643 at 2012 and
// 1883 at 8192.  What bounds it is one warp's chain of minimum over the lanes
// (24 cycles), pair loads (30 and up), clamp and compare, three times per
// merge, and in-order issue: whatever the next operation does not wait for -
// ids, tails, parents - is stored after the minimum is under way.  Tried:
// these stores before it 390; the new tail at the parting of two paths by a
// second minimum instead of in its lane 399; 16-bit ids and tails with
// comparisons instead of kInf nodes 457; nodes of 8 bytes, whose pair is one
// 16-byte load, 574; tails stored before the next operation's loads 619.  The
// loop's place among other code counts too: the same source took 350 to 377
// cycles as the code around it changed, and 370 as a function of its own.
//
// Shared layout, nodes 1-based (node k's children are 2k and 2k + 1), words:
// the probabilities (a pair of children is one 8-byte load), the ids, the
// tails, and 16-bit parent links.  Node 0 and every node without an element
// hold kInf, up to the last of the deepest level; lanes without a node (or
// without children) read a pair of kInf behind them.  Removing the last
// element leaves the tails of its ancestors that end in it pointing at a
// missing right child: every level therefore takes the smaller of the pair it
// loads, and a tail's last step - below which there are no elements - does not
// matter.
//
// W supplies the warp: lane vectors of 32-bit words and conditions, warp-wide
// minimum, ballot and shuffle, and shared-memory access (the device's own
// registers, or 32-element arrays with bounds checks in the host self-test).
#pragma once

#include "cc_common.cuh"

namespace ccb {
namespace hm {

constexpr u32 kInf = 0x80000000u;       // probabilities and their sum are below it
constexpr u32 kKeyLevel = 18;           // a key: level << kKeyLevel | tail << 2
constexpr u32 kKeyTail = (1u << kKeyLevel) - 1u;
constexpr u32 kNoKey = 0x7Fu << kKeyLevel;   // | tail << 2: above every level's

CC_HD constexpr u32 log2Floor(u32 v) { return 31u - u32(__builtin_clz(v)); }

// Byte offsets of the arrays for up to kCap leaves (ids and parents of 2 kCap
// nodes fit 16 bits).  Ids and tails are kept for kCap + 2 nodes; loads of
// missing nodes' reach at most kNodes words from their array's start, inside
// the area, and are not used.
template <u32 kCap>
struct Layout {
    static constexpr u32 kNodes = 2u << log2Floor(kCap);   // of the full tree
    static constexpr u32 kNone = 4u * kNodes;              // the pair without elements
    static constexpr u32 kIds = kNone + 8u;                // id x 2
    static constexpr u32 kTails = kIds + 4u * (kCap + 2u); // tail x 4
    static constexpr u32 kParents = kTails + 4u * (kCap + 2u);
    static constexpr u32 kBytes = kParents + 4u * kCap;
    static_assert(kCap % 2u == 0 && kCap <= 16384u, "pairs of ids are 8-byte aligned; a node id fits 15 bits");
    static_assert(kIds + 4u * kNodes <= kBytes && kTails + 4u * kNodes <= kBytes, "loads of missing nodes");
};

template <class W, u32 kCap>
struct Merge {
    using U = typename W::U;
    using B = typename W::B;
    using At = Layout<kCap>;

    W w;
    u32 D;            // depth of the deepest level
    U level, levelKey, sh, shChild;   // the lane's level; shifts from a key to byte offsets
    U pairMask, nodeMask, childMask;  // of a shifted key: 4 x the node's pair, 4 x node, 8 x node
    U none, noneChild;                // kNone where the lane has no node, or no children, else 0
    U deeper;         // mask of the lanes of deeper levels
    U upMask;         // the root has nothing above it

    // An operation's loads.
    struct Loads {
        U px, py;     // the pair of the lane's node
        U nx, ny;     // pop: the pair below the node; push: nx the node above
        U ix, iy;     // pop: the ids of that pair; push: ix the id of the node above
        U pair4, node4, sibTail;
        u32 tail4, v, idv;
    };
    // What its moves leave: whether the sibling is the smaller child now, its
    // tail, the lane's key and the path's end; the winners' ballot, and the
    // tails on their way to their array.
    struct Path {
        U node4, sibTail, key, newTail;
        B holds, win;
        u32 tail4, winners;
    };
    // An operation's moves: where, which id, whether.
    struct Store {
        U at4, id;
        B moved;
    };
    U rootP, rootId;   // the root's element, in its lane

    // The lanes run from the deepest level up (lane 31 is the root's), so that
    // the nearest winner below a level is a highest set bit.
    CC_HD Merge(W w_, u32 L) : w(w_), D(log2Floor(L)) {
        level = w.sub(w.all(31u), w.lane());
        levelKey = w.shl(level, kKeyLevel);
        const B act = w.le(level, w.all(D));
        const B inner = w.lt(level, w.all(D));
        sh = w.sel(act, w.sub(w.all(D), level), w.all(31u));
        shChild = w.sel(inner, w.sub(w.all(D), w.add(level, w.all(1u))), w.all(31u));
        const U nodes = w.sel(act, w.sub(w.shlv(w.all(2u), w.sel(act, level, w.all(0u))), w.all(1u)), w.all(0u));
        nodeMask = w.shl(nodes, 2u);
        pairMask = w.andv(nodeMask, w.all(~7u));
        childMask = w.sel(inner, w.shl(nodes, 3u), w.all(0u));
        none = w.sel(act, w.all(0u), w.all(At::kNone));
        noneChild = w.sel(inner, w.all(0u), w.all(At::kNone));
        deeper = w.sub(w.shlv(w.all(1u), w.lane()), w.all(1u));
        upMask = w.sel(w.eq(level, w.all(0u)), w.all(0u), w.all(~0u));
    }

    // Takes the last element out of a heap of n + 1.
    CC_HD void takeLast(Loads& l, u32 n) {
        l.v = w.template ldOne<0>(4u * (n + 1));
        l.idv = w.template ldOne<At::kIds>(4u * (n + 1));
        w.fence();
        w.template stAll<0>(4u * (n + 1), kInf);
        w.fence();
    }

    // key: the previous operation's minimum.
    CC_HD void popLoads(Loads& l, u32 key) {
        const U t = w.shr(w.all(key), sh);
        const U child8 = w.andv(w.shr(w.all(key), shChild), childMask);
        l.pair4 = w.orv(w.andv(t, pairMask), none);
        const U kids = w.orv(child8, noneChild);
        w.template ldPair<0>(l.pair4, l.px, l.py);
        w.template ldPair<0>(kids, l.nx, l.ny);
        l.node4 = w.andv(t, nodeMask);
        w.template ldPair<At::kIds>(child8, l.ix, l.iy);
        l.sibTail = w.template ld<At::kTails>(w.xorv(l.node4, w.all(4u)));
        l.tail4 = key & kKeyTail;
    }

    // The moves of a pop that leaves n elements.  prev: the previous
    // operation, whose tails are stored here; parting: the level at which this
    // path leaves its path (the sibling there is its node, with a new tail).
    CC_HD void popMove(const Loads& l, u32 n, u32 parting, const Path& prev, Path& p, Store& o) {
        const U v = w.all(l.v);
        const U x = w.min(l.px, l.py);
        const U y = w.max(x, w.min3(v, l.nx, l.ny));
        const B isLeft = w.lt(l.px, l.py);
        o.at4 = w.sel(isLeft, l.pair4, w.add(l.pair4, w.all(4u)));
        o.moved = w.le(x, v);
        w.fence();
        w.template st<0>(o.at4, y, o.moved);
        rootP = y;
        // the sibling wins a left node's place on a tie too
        finish(l, n, y, w.sel(isLeft, w.below(l.py), l.px), parting, prev, p);
        o.id = w.sel(w.le(w.min(l.nx, l.ny), v), w.sel(w.lt(l.nx, l.ny), l.ix, l.iy), w.all(l.idv));
    }
    // The ids of an operation's moves, and the tails of the one before.
    CC_HD void storeIds(const Store& o, const Path& prev) {
        w.template st<At::kIds>(o.at4, o.id, o.moved);
        tailsStore(prev);
        w.fence();
    }

    CC_HD void finish(const Loads& l, u32 n, const U& y, const U& s, u32 parting, const Path& prev, Path& p) {
        p.sibTail = w.sel(w.eq(level, w.all(parting)), prev.newTail, l.sibTail);
        p.win = w.lt(s, y);
        p.key = w.sel(p.win, w.orv(levelKey, p.sibTail), w.all(kNoKey | l.tail4));
        p.node4 = l.node4;
        p.holds = w.le(l.node4, w.all(4u * n));
        p.tail4 = l.tail4;
    }

    // Loads of a push whose path ends in tail4 / 4: the probabilities, and once
    // the pop's ids and tails are stored, the rest.
    CC_HD void pushValues(Loads& l, u32 tail4) {
        const U t = w.shr(w.all(tail4), sh);
        l.node4 = w.andv(t, nodeMask);
        l.pair4 = w.andv(t, pairMask);
        w.template ldPair<0>(w.orv(l.pair4, none), l.px, l.py);
        l.nx = w.template ld<0>(w.shr(l.pair4, 1u));
        l.tail4 = tail4;
    }
    CC_HD void pushRest(Loads& l) {
        l.ix = w.template ld<At::kIds>(w.shr(l.pair4, 1u));
        l.sibTail = w.template ld<At::kTails>(w.xorv(l.node4, w.all(4u)));
    }

    // The moves of a push of c at position q.
    CC_HD void pushMove(const Loads& l, u32 q, u32 c, u32 id, u32 parting, const Path& prev, Path& p, Store& o) {
        const B odd = w.nz(w.andv(l.node4, w.all(4u)));
        const U e = w.sel(odd, l.py, l.px);
        const U up = w.andv(l.nx, upMask);
        const U cv = w.all(c);
        const U y = w.max(up, w.min(cv, e));
        o.at4 = l.node4;
        o.moved = w.both(w.le(w.orv(l.node4, none), w.all(4u * q)), w.lt(cv, e));
        w.fence();
        w.template st<0>(o.at4, y, o.moved);
        rootP = y;
        finish(l, q, y, w.sel(odd, l.px, w.below(l.py)), parting, prev, p);
        o.id = w.sel(w.lt(cv, up), l.ix, w.all(id));
    }

    // Tails of an operation's path nodes, while the next operation waits for
    // its loads: the nearest winning sibling below each node, and its tail
    // (else the path's end).
    CC_HD void tailsFind(Path& p) {
        const U from = w.andv(w.all(p.winners), deeper);
        const U t = w.shfl(p.sibTail, w.lastSet(from));
        p.newTail = w.sel(w.nz(from), t, w.all(p.tail4));
    }
    CC_HD void tailsStore(const Path& p) {
        w.template st<At::kTails>(p.node4, p.newTail, p.holds);
    }
    // Merges the heap of L >= 2 elements (the arrays set up: ids and tails of
    // nodes 1 .. L, kInf at the others of the full tree and at kNone); writes
    // the parent of every id but the root's (2L - 2).
    CC_HD void run(u32 L) {
        Path pa, pb, pc;
        // an operation before the first: no winners, nothing to store
        pc.tail4 = w.template ldOne<At::kTails>(4u);
        pc.node4 = w.all(0u);
        pc.sibTail = w.all(0u);
        pc.holds = w.lt(w.all(1u), w.all(0u));
        pc.winners = 0;
        pc.newTail = w.all(pc.tail4);
        rootP = w.all(w.template ldOne<0>(4u));
        rootId = w.all(w.template ldOne<At::kIds>(4u));
        u32 rc = kNoKey | pc.tail4;
        u32 next = L;
        u32 qDepth = D;   // depth of the push's position
        Loads l;
        Store o;
        takeLast(l, L - 1);
        for (u32 len = L; len > 1; --len, ++next) {
            const u32 q = len - 1;
            if (q < (1u << qDepth)) --qDepth;
            const u32 tailC = 4u * q << (D - qDepth);

            popLoads(l, rc);
            tailsFind(pc);
            w.template stParent<At::kParents>(rootId, next);
            U c = rootP;
            popMove(l, len - 1, rc >> kKeyLevel, pc, pa, o);
            const u32 ra = w.reduceMin(pa.key);
            rootId = o.id;
            storeIds(o, pc);
            takeLast(l, len - 2);
            pa.winners = w.ballot(pa.win);

            popLoads(l, ra);
            tailsFind(pa);
            w.template stParent<At::kParents>(rootId, next);
            c = w.shfl(w.add(c, rootP), w.all(31u));
            // the level at which the push's path leaves this pop's
            const u32 diff = (tailC ^ l.tail4) >> 2;
            const u32 h = diff ? D - log2Floor(diff) : 0x7Eu;
            popMove(l, len - 2, ra >> kKeyLevel, pa, pb, o);
            w.fence();

            pushValues(l, tailC);
            pb.winners = w.ballot(pb.win);
            rootId = o.id;
            storeIds(o, pa);
            pushRest(l);
            tailsFind(pb);
            pushMove(l, q, w.first(c), 2u * next, h, pb, pc, o);
            rc = w.reduceMin(pc.key);
            pc.winners = w.ballot(pc.win);
            rootId = w.sel(o.moved, o.id, rootId);
            storeIds(o, pb);
            takeLast(l, len - 2);
        }
    }
};

#ifdef __CUDACC__
// The calling warp: a lane vector is the lane's own register; memory is the
// block's dynamic shared memory, whose address the compiler folds into the
// loads and stores.
struct DeviceWarp {
    using U = u32;
    using B = bool;
    __device__ __forceinline__ static unsigned char* mem() {
        extern __shared__ __align__(16) unsigned char dyn[];
        return dyn;
    }
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
    __device__ __forceinline__ u32 min3(u32 a, u32 b, u32 c) const { return __vimin3_u32(a, b, c); }
    __device__ __forceinline__ u32 max(u32 a, u32 b) const { return a > b ? a : b; }
    __device__ __forceinline__ u32 below(u32 a) const { return a - 1u + (a >> 31); }   // a - 1, kInf kept
    __device__ __forceinline__ u32 sub(u32 a, u32 b) const { return a - b; }
    __device__ __forceinline__ u32 add(u32 a, u32 b) const { return a + b; }
    __device__ __forceinline__ u32 shr(u32 a, u32 n) const { return a >> n; }
    __device__ __forceinline__ u32 shl(u32 a, u32 n) const { return a << n; }
    __device__ __forceinline__ u32 shlv(u32 a, u32 n) const { return a << n; }
    __device__ __forceinline__ u32 andv(u32 a, u32 b) const { return a & b; }
    __device__ __forceinline__ u32 orv(u32 a, u32 b) const { return a | b; }
    __device__ __forceinline__ u32 xorv(u32 a, u32 b) const { return a ^ b; }
    __device__ __forceinline__ u32 lastSet(u32 m) const { return 31u - u32(__clz(int(m))); }
    __device__ __forceinline__ u32 ballot(bool c) const { return __ballot_sync(0xffffffffu, c); }
    __device__ __forceinline__ u32 reduceMin(u32 v) const { return __reduce_min_sync(0xffffffffu, v); }
    __device__ __forceinline__ u32 shfl(u32 v, u32 from) const { return __shfl_sync(0xffffffffu, v, int(from)); }
    __device__ __forceinline__ void fence() const { __syncwarp(); }
    template <u32 kArray>
    __device__ __forceinline__ void ldPair(u32 off, u32& x, u32& y) const {
        const uint2 v = *reinterpret_cast<const uint2*>(mem() + kArray + off);
        x = v.x;
        y = v.y;
    }
    template <u32 kArray>
    __device__ __forceinline__ u32 ld(u32 off) const { return *reinterpret_cast<const u32*>(mem() + kArray + off); }
    template <u32 kArray>
    __device__ __forceinline__ u32 ldOne(u32 off) const { return ld<kArray>(off); }
    // Predicated stores are written out: as conditional statements they became
    // branches (541 instead of 390 cycles per merge then).
    __device__ __forceinline__ static u32 window() { return u32(__cvta_generic_to_shared(mem())); }
    template <u32 kArray>
    __device__ __forceinline__ void st(u32 off, u32 v, bool c) const {
        asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u32 [%0 + %3], %1;\n}"
                     :: "r"(window() + off), "r"(v), "r"(u32(c)), "n"(kArray) : "memory");
    }
    template <u32 kArray>
    __device__ __forceinline__ void stAll(u32 off, u32 v) const { *reinterpret_cast<u32*>(mem() + kArray + off) = v; }
    // by the root's lane; id2: the id x 2
    template <u32 kArray>
    __device__ __forceinline__ void stParent(u32 id2, u32 v) const {
        asm volatile("{\n.reg .pred p;\nsetp.eq.u32 p, %2, 31;\n@p st.shared.u16 [%0 + %3], %1;\n}"
                     :: "r"(window() + id2), "h"(u16(v)), "r"(lane()), "n"(kArray) : "memory");
    }
};
#endif

}  // namespace hm
}  // namespace ccb
