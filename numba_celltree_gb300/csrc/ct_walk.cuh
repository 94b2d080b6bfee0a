// ct_walk.cuh -- tree traversals by a warp over a queue of nodes.
//
// A traversal with one thread per query is a chain of dependent node loads in
// which each lane of a warp is at another node, and the longest query of a
// warp holds the others up (9 to 12 of 32 lanes active).  Here a warp takes a
// few queries and keeps their open nodes, in traversal order, in a queue in
// shared memory.  Every round takes 32 of them, one per lane, loads their
// records at once and replaces each node by its children to visit (none, one
// or two, in the order they are visited) or by itself when it is terminal.
// The queue is therefore always the list of nodes still to be reported, in
// the order of the depth-first walk, and what is reported and its order are
// the walk's.
//
// A queue of at most WALK_FULL nodes is expanded as a whole, level by level.
// Above that, leading terminal nodes are reported first and a round's worth
// of leading nodes is expanded, or as many as keep WALK_RESERVE places free,
// at least one.  So the queue grows past WALK_CAP - WALK_RESERVE nodes only while one
// leading node at a time is expanded: that is the depth-first walk, whose
// open nodes are at most one per level below the node it began with (126
// levels), and its terminal nodes are reported as they come to the head.
// The queue never overflows.
#pragma once

#include "ct_common.cuh"

constexpr int WALK_CAP = 512;      // nodes per queue (two per warp)
constexpr int WALK_WARPS = 4;      // warps per block, at most and by default
constexpr int WALK_BLOCKS = 8;     // such blocks per SM (28 KB of shared memory each)
// Queries per warp, at most.  More (16, 32, let in a few at a time) fill the
// rounds of tiny queries better but leave fewer warps, and the heavy ones of
// a batch end later: 250k boxes of very different sizes 33.5 -> 34.2 -> 35.6
// ms, 1M segments 9.8 -> 10.2 -> 11.1 ms.
constexpr int WALK_Q = 8;
constexpr int WALK_RESERVE = 130;  // more than the deepest stacked tree's levels
constexpr int WALK_FULL = (WALK_CAP - WALK_RESERVE) / 2;  // a queue that may double

// item: node, and query (low byte: WALK_QMASK) with flags and depth
constexpr unsigned WALK_QMASK = 0x1fu, WALK_TERM = 0x20u, WALK_WHOLE = 0x40u;

enum { WALK_DROP = 0, WALK_OPEN = 1, WALK_LEAF = 2, WALK_ALL = 3 };

struct WalkBuf {
    int node[2][WALK_CAP];
    unsigned short meta[2][WALK_CAP];
};

// A warp's shared memory: its queue, the queries, results reported of each.
template <class Query, class Count>
struct WalkShared {
    WalkBuf buf;
    Query query[WALK_Q];
    Count count[WALK_Q];
};

// Puts the first nodes (-1: none) of the warp's queries (lane = query) into
// the queue; returns their number.
__device__ __forceinline__ int walk_begin(WalkBuf& B, int start, int lane) {
    const unsigned b = __ballot_sync(0xffffffffu, start >= 0);
    if (start >= 0) {
        const int p = __popc(b & ((1u << lane) - 1u));
        B.node[0][p] = start;
        B.meta[0][p] = (unsigned short)lane;
    }
    __syncwarp();
    return __popc(b);
}

template <class Policy>
__device__ __forceinline__ void walk_report(Policy& pol, const int* node, const unsigned short* meta, int m, int lane) {
    for (int k = lane; k - lane < m; k += 32) {
        const bool have = k < m;
        pol.emit(have ? node[k] : -1, have ? (unsigned)meta[k] : 0u, have);
    }
}

// Runs the queue B.node[0][0 .. n) to its end.  `pol.visit(node, query, depth,
// &first, &second)` gives WALK_DROP, WALK_OPEN (children, -1: not visited),
// WALK_LEAF or WALK_ALL (terminal); `pol.emit(node, meta, have)` reports the
// lanes' terminal nodes, in lane order.  `rounds`: bound on the rounds.
template <class Policy>
__device__ __forceinline__ void walk(Policy& pol, WalkBuf& B, int n, int lane, int64_t rounds, unsigned int* err) {
    const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
    int cur = 0, head = 0, open = n;
    while (n > 0) {
        if (open == 0) {
            walk_report(pol, B.node[cur] + head, B.meta[cur] + head, n, lane);
            return;
        }
        if (--rounds < 0) {
            if (lane == 0) set_error(err, CT_DEVERR_LOOP);
            return;
        }
        if (n > WALK_FULL) {
            int lead = 0;
            for (; lead < n; lead += 32) {
                const bool term = lead + lane < n && (B.meta[cur][head + lead + lane] & WALK_TERM);
                const unsigned b = __ballot_sync(FULL, !term);
                if (b) {
                    lead = min(n, lead + __ffs(b) - 1);
                    break;
                }
            }
            if (lead > 0) {
                walk_report(pol, B.node[cur] + head, B.meta[cur] + head, lead, lane);
                head += lead;
                n -= lead;
            }
        }
        const int w = n <= WALK_FULL ? n : min(n, max(1, min(32, WALK_CAP - n - WALK_RESERVE)));
        int nn = 0;
        open = 0;
        for (int base = 0; base < n; base += 32) {
            const int k = base + lane;
            const bool have = k < n;
            int v = -1, first = -1, second = -1;
            unsigned m = WALK_TERM;
            if (have) {
                v = B.node[cur][head + k];
                m = B.meta[cur][head + k];
            }
            unsigned mo = m;
            if (have) {
                first = v;
                if (!(m & WALK_TERM) && k < w) {
                    const int kind = pol.visit(v, (int)(m & WALK_QMASK), (int)(m >> 8), &first, &second);
                    if (kind == WALK_DROP) first = second = -1;
                    if (kind == WALK_OPEN) mo = m + 0x100u;
                    if (kind == WALK_LEAF || kind == WALK_ALL) {
                        first = v;
                        second = -1;
                        mo = m | WALK_TERM | (kind == WALK_ALL ? WALK_WHOLE : 0u);
                    }
                }
            }
            const unsigned b1 = __ballot_sync(FULL, first >= 0), b2 = __ballot_sync(FULL, second >= 0);
            const unsigned bo = __ballot_sync(FULL, first >= 0 && !(mo & WALK_TERM));
            int p = nn + __popc(b1 & lt) + __popc(b2 & lt);
            if (first >= 0) {
                B.node[cur ^ 1][p] = first;
                B.meta[cur ^ 1][p] = (unsigned short)mo;
                p++;
            }
            if (second >= 0) {
                B.node[cur ^ 1][p] = second;
                B.meta[cur ^ 1][p] = (unsigned short)mo;
            }
            nn += __popc(b1) + __popc(b2);
            open += __popc(bo) + __popc(b2);
        }
        __syncwarp();
        cur ^= 1;
        head = 0;
        n = nn;
    }
}

// Rank of each lane's results within its query: lanes hold items of
// consecutive queries in order; `emitted[q]` counts what the query has
// reported before and is raised by this call's.
template <typename C>
__device__ __forceinline__ C walk_rank(int q, C c, bool have, int lane, C* emitted) {
    const unsigned FULL = 0xffffffffu;
    C incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const C t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    const C excl = incl - c;
    const int qp = __shfl_up_sync(FULL, q, 1), qn = __shfl_down_sync(FULL, q, 1);
    const unsigned heads = __ballot_sync(FULL, lane == 0 || qp != q);
    const int h = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    const C before = __shfl_sync(FULL, excl, h);
    const C done = have ? emitted[q] : 0;
    __syncwarp();
    if (have && (lane == 31 || qn != q)) emitted[q] = done + incl - before;
    __syncwarp();
    return done + excl - before;
}
