// ct_multi.cu -- multi-result queries, per-pair kernels, barycentric weights
// and node-bound diagnostics.
//
// Multi-result queries (locate_boxes query.py:177-289, _locate_edges
// query.py:357-533) are rebuilt as count -> exclusive scan -> write: the
// count and write kernels run the same traversal, so the write pass knows
// each query's output offset.  Results come out query-major and, within a
// query, in traversal order -- exactly upstream's concatenated order.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "ct_common.cuh"
#include "ct_clip.cuh"
#include "ct_geom.cuh"
#include "ct_internal.h"
#include "ct_locf.cuh"
#include "ct_walk.cuh"

extern "C" size_t ct_radix_pass_workspace_size(void);
extern "C" int ct_radix_pass(const unsigned* kin, const int* iin, int64_t n, int32_t shift, unsigned* kout, int* iout,
                             void* ws, size_t ws_bytes, void* stream);

namespace ctm {

struct TreeQ {
    const float4* nf;    // packed node meta: z = child / ptr, w = -1 - dim / size
    const double2* nd;   // Lmax, Rmin
    const double2* poly; // leaf-ordered polygons (K per cell)
    const uint8_t* plen;
    const int64_t* bbi;
    const double* bb;    // bb_coords (cell order)
    unsigned int* err;
    int64_t n_nodes;
    dbox bbox;
    int K;
    int box_warps, seg_warps;  // warps per block of the walks by warps
    bool finite;  // all node bounds and cell boxes finite: order comparisons on integer keys
    // box index (ct_pack_box_index; null when not built)
    const double4* bbl;        // cell boxes in leaf order
    const struct NodeBox* nbx; // per node: bounding box of its cells (float32 frame, outward) and leaf range
    const int* lstart;         // per leaf position: first position of its leaf
    double ox, oy;             // float32 frame origin
    const int* parent;         // node parents (trees deeper than the stacks are walked through them)
    // float32 leaf data (ct_locf.cuh) for the filters of the segment test
    const float4* polyf;
    const uint8_t* plen32;
    int S4;
    float dabs;                // float64 rounding of absolute coordinates
    // line filter of the segment traversal (null bbl32: off)
    const float4* bbl32;       // cell boxes in leaf order, float32 frame, rounded outward
    float fX, fY;              // largest |x - ox|, |y - oy| over the tree's bbox
    double babs;               // largest |coordinate| of the tree's bbox
    double mext;               // 2^-37 x the tree's largest extent + 2^-47
};

// Bounding box of a node's cells in the float32 frame of the tree (x - ox,
// y - oy rounded outward) and the node's range of leaf positions.  32 bytes.
struct NodeBox {
    float xmin, xmax, ymin, ymax;
    int ptr, size, pad0, pad1;
};

// x < y for finite (or infinite, non-NaN) doubles as one 64-bit integer
// comparison of order-preserving keys (-0.0 and +0.0 share a key, as they
// compare equal): the comparisons of the box and segment traversals run on
// the integer pipes instead of GB300's narrow float64 pipe.
__device__ __forceinline__ bool not_nan(double x) {
    return ((unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull) <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool is_fin(double x) {
    return ((unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull) < 0x7ff0000000000000ull;
}

__device__ __forceinline__ int na(const float4& q) { return __float_as_int(q.z); }
__device__ __forceinline__ int nb(const float4& q) { return __float_as_int(q.w); }

constexpr int STK = 128;  // traversal stack (tree depth + 2 must fit; checked on the host)

// bb_coords of the cell at leaf position j: from the leaf-ordered copy of the
// box index when it is built, else through bb_indices
__device__ __forceinline__ dbox leaf_box(const TreeQ& T, int64_t j) {
    if (T.bbl) {
        double4 c4 = T.bbl[j];
        dbox b;
        b.xmin = c4.x;
        b.xmax = c4.y;
        b.ymin = c4.z;
        b.ymax = c4.w;
        return b;
    }
    return load_box(T.bb + 4 * T.bbi[j]);
}

// ---------------------------------------------------------------------------
// locate_box query.py:177-244
// ---------------------------------------------------------------------------
// A subtree wholly inside a query box whose cells the writing pass leaves to
// k_box_jobs: its output offset, the query box and its leaf range.
struct BoxJob {
    int64_t out, box;
    int ptr, size, pad0, pad1;
};
constexpr int BOX_JOB_MIN = 8;  // default: smaller subtrees are written in line

// One thread per box: large batches of boxes of a few cells each (query faces;
// boxes whose sizes were looked at), whose neighbouring lanes take the same
// path in mesh order or spatial order -- 1M faces on 500k cells 0.38 ms, by
// warps (below) 0.6 ms -- and, with DEEP, trees deeper than the warps' walk
// takes.
template <bool WRITE, bool DEEP>
__global__ void __launch_bounds__(256) k_boxes(TreeQ T, const double4* __restrict__ boxes, int64_t n,
                                               const int* __restrict__ order, int64_t* __restrict__ cnt_or_off,
                                               int64_t* __restrict__ ii, int64_t* __restrict__ jj,
                                               BoxJob* __restrict__ jobs = nullptr,
                                               unsigned long long* __restrict__ njobs = nullptr, int64_t job_cap = 0,
                                               int job_min = BOX_JOB_MIN, int* __restrict__ spec = nullptr,
                                               int spec_cap = 0, const int64_t* __restrict__ spec_cnt = nullptr) {
    int64_t tq = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tq >= n) return;
    // queries in work order (similar work in one warp); results by query index
    int64_t i = order ? (int64_t)order[tq] : tq;
    // writing pass after a speculative count: boxes whose pairs all fit the
    // per-box scratch were written from it (k_boxes_spec_emit)
    if (WRITE && spec_cnt && spec_cnt[i] <= spec_cap) return;
    int* sp_out = (!WRITE && spec) ? spec + i * (int64_t)spec_cap : nullptr;
    double4 q4 = boxes[i];
    dbox box;
    box.xmin = q4.x;
    box.xmax = q4.y;
    box.ymin = q4.z;
    box.ymax = q4.w;
    int64_t count = 0;
    int64_t base = WRITE ? cnt_or_off[i] : 0;
    // key path: every value non-NaN, so the order comparisons equal the
    // float64 ones (NaN boxes keep the float64 comparisons)
    const bool keys = T.finite && not_nan(box.xmin) && not_nan(box.xmax) && not_nan(box.ymin) && not_nan(box.ymax);
    const unsigned long long kx0 = fkey(box.xmin), kx1 = fkey(box.xmax), ky0 = fkey(box.ymin), ky1 = fkey(box.ymax);
    // box index: a node whose cells' bounding box lies strictly inside the
    // query box has every cell overlapping it (boxes_intersect is strict and
    // cell.xmax >= node.xmin > box.xmin, ...); the traversal would visit all
    // of it.  The query box in the float32 frame is rounded inward, the node
    // boxes outward, so a float32 "strictly inside" implies the float64 one.
    // A node whose cells' bounding box lies strictly beyond a side of the
    // query box has no overlapping cell (boxes_intersect needs
    // box.xmin < cell.xmax <= node.xmax, ...): its subtree is skipped.  The
    // query box rounded outward, the node boxes outward: since x -> fl(x - o)
    // is monotonic, node.xmax_f32 < float_rd(fl(box.xmin - o)) implies
    // node.xmax < box.xmin.  Skipped subtrees hold no result, so the output
    // and its order are unchanged.
    const bool idx = keys && T.nbx != nullptr;
    float qx0 = 0.0f, qx1 = 0.0f, qy0 = 0.0f, qy1 = 0.0f;
    float ox0 = 0.0f, ox1 = 0.0f, oy0 = 0.0f, oy1 = 0.0f;
    if (idx) {
        qx0 = __double2float_ru(box.xmin - T.ox);
        qx1 = __double2float_rd(box.xmax - T.ox);
        qy0 = __double2float_ru(box.ymin - T.oy);
        qy1 = __double2float_rd(box.ymax - T.oy);
        ox0 = __double2float_rd(box.xmin - T.ox);
        ox1 = __double2float_ru(box.xmax - T.ox);
        oy0 = __double2float_rd(box.ymin - T.oy);
        oy1 = __double2float_ru(box.ymax - T.oy);
    }
    if (boxes_intersect(box, T.bbox)) {
        // depth-first walk: a stack, or (DEEP, trees deeper than the stack)
        // the parent links -- down to the child that would be popped first,
        // back up to the parent to find the sibling still to visit
        int st[DEEP ? 1 : STK];
        int sp = 1;
        st[0] = 0;
        int dv = 0, from = -1;
        bool down = true;
        int64_t budget = DEEP ? 2 * T.n_nodes + 2 : T.n_nodes;
        while (DEEP ? dv >= 0 : sp > 0) {
            if (--budget < 0) {
                set_error(T.err, CT_DEVERR_LOOP);
                break;
            }
            const int v = DEEP ? dv : st[--sp];
            bool terminal = false;
            // the node's three records loaded together (one memory round trip
            // per visited node instead of a chain of three)
            const float4 q = T.nf[v];
            const double2 nd_v = T.nd[v];
            NodeBox nbv;
            if (idx && (!DEEP || down)) nbv = T.nbx[v];
            if (!DEEP || down) {
                if (idx) {
                    if (nbv.xmax < ox0 || nbv.xmin > ox1 || nbv.ymax < oy0 || nbv.ymin > oy1) {
                        terminal = true;  // no cell below overlaps the box
                    } else if (qx0 < nbv.xmin && nbv.xmax < qx1 && qy0 < nbv.ymin && nbv.ymax < qy1) {
                        // the whole subtree, in upstream's visiting order: right
                        // child first, i.e. leaves by decreasing position, each
                        // leaf's cells by increasing position
                        int64_t jk = -1;
                        if (WRITE && jobs && nbv.size >= job_min) {
                            jk = (int64_t)atomicAdd(njobs, 1ull);
                            if (jk < job_cap) {
                                BoxJob J;
                                J.out = base + count;
                                J.box = i;
                                J.ptr = nbv.ptr;
                                J.size = nbv.size;
                                J.pad0 = J.pad1 = 0;
                                jobs[jk] = J;
                            } else {
                                jk = -1;  // no room (cannot happen with the sized buffer): write in line
                            }
                        }
                        if ((WRITE && jk < 0) || (sp_out && count < spec_cap)) {
                            int qq = nbv.ptr + nbv.size;
                            int64_t c = count;
                            while (qq > nbv.ptr && (WRITE || c < spec_cap)) {
                                int s = T.lstart[qq - 1];
                                if (s < nbv.ptr || s >= qq) {  // corrupt index: stop rather than loop
                                    set_error(T.err, CT_DEVERR_LOOP);
                                    break;
                                }
                                for (int j = s; j < qq; j++) {
                                    if (WRITE) {
                                        ii[base + c] = i;
                                        jj[base + c] = T.bbi[j];
                                    } else if (c < spec_cap) {
                                        sp_out[c] = (int)T.bbi[j];
                                    }
                                    c++;
                                }
                                qq = s;
                            }
                        }
                        count += nbv.size;
                        terminal = true;
                    }
                }
                if (!terminal) {
                    int b = nb(q);
                    if (b >= 0) {
                        int ptr = na(q);
                        for (int j = ptr; j < ptr + b; j++) {
                            dbox lb = leaf_box(T, j);
                            // boxes_intersect geometry_utils.py:292-300
                            bool hit = keys ? (kx0 < fkey(lb.xmax) && fkey(lb.xmin) < kx1 && ky0 < fkey(lb.ymax) &&
                                               fkey(lb.ymin) < ky1)
                                            : boxes_intersect(box, lb);
                            if (hit) {
                                if (WRITE) {
                                    ii[base + count] = i;
                                    jj[base + count] = T.bbi[j];
                                } else if (sp_out && count < spec_cap) {
                                    sp_out[count] = (int)T.bbi[j];
                                }
                                count++;
                            }
                        }
                        terminal = true;
                    }
                }
            }
            int first = -1, second = -1;
            if (!terminal) {
                int dim = -1 - nb(q);
                const double2 d = nd_v;
                bool left, right;
                if (keys) {
                    left = (dim ? ky0 : kx0) <= fkey(d.x);
                    right = (dim ? ky1 : kx1) >= fkey(d.y);
                } else {
                    double bmin = dim ? box.ymin : box.xmin, bmax = dim ? box.ymax : box.xmax;
                    left = bmin <= d.x;
                    right = bmax >= d.y;
                }
                // pushed left, then right: the right child is visited first
                int child = na(q);
                first = right ? child + 1 : (left ? child : -1);
                second = (left && right) ? child : -1;
            }
            if (DEEP) {
                int next = terminal ? -1 : (down ? first : ((from == first) ? second : -1));
                from = dv;
                if (next >= 0) {
                    dv = next;
                    down = true;
                } else {
                    dv = T.parent[dv];
                    down = false;
                }
            } else if (!terminal) {
                if (sp + 2 > STK) {
                    set_error(T.err, CT_DEVERR_STACK);
                    break;
                }
                if (second >= 0) st[sp++] = second;
                if (first >= 0) st[sp++] = first;
            }
        }
    }
    if (!WRITE) cnt_or_off[i] = count;
}

// ---------------------------------------------------------------------------
// Box queries by warps (ct_walk.cuh): counts, with `spec` the first spec_cap
// cells of every box (in output order) as well, or with WRITE the pairs at
// the boxes' offsets.  The tests of a node and of a cell are those of
// k_boxes, whose comments give the reasons.  A terminal node is a leaf
// or a subtree wholly inside the box; the outputs of 32 of them are numbered
// through and shared out over the lanes, so pairs are written coalesced
// however they are spread over nodes.
//
// A thread per box was bound by its chain of node loads and by the largest
// box of its warp (9 of 32 lanes active).  250k boxes of 0.1 to 50 m on 5M
// cells: counting 4.6 -> 2.6 ms, writing 6.8 -> 4.6 ms; 10k small boxes on 80k
// cells 117 -> 37 us.
// ---------------------------------------------------------------------------
struct WalkBox {  // 88 bytes: an odd number of 8-byte words, so lanes of different queries hit different banks
    unsigned long long kx0, kx1, ky0, ky1;
    float qx0, qx1, qy0, qy1;  // the box in the float32 frame, rounded inward
    float ox0, ox1, oy0, oy1;  // and outward
    int64_t base, id;
    bool keys, idx;
};
static_assert(sizeof(WalkBox) == 88, "see above");

// A terminal node of a box's walk with pairs, kept by the counting pass: the
// box (top bit: the whole subtree lies inside it), the rank of the first pair
// within the box (top bit: a leaf of more than 32 cells), the first leaf
// position, and the leaf's overlapping cells as bits or the number of cells.
// A whole subtree of more than two parts of `part` cells is kept in parts
// that begin at leaves: a warp of k_box_records takes 32 records, and one
// warp alone would write the pairs of a box around the mesh (one box around
// 5M cells 183 ms, in parts 0.85).  The writing pass leaves whole subtrees
// to k_box_records in the same form, where it has the room.
struct BoxRecs {
    int4* rec;
    unsigned long long* count;   // records the counting pass asked for (null: there was none)
    unsigned long long* pushed;  // records of the writing pass
    int64_t cap;
    int part;  // of the writing pass (of the counting pass: REC_PART)
    uint8_t* inside;  // optional, per pair: the cell lies in a subtree inside the box
};
constexpr int REC_FLAG = (int)0x80000000u;
constexpr int REC_PART = 256;

// The outputs of the lanes' terminal nodes (`share` each), 32 at a time:
// put(box, output index, leaf position) per lane; whole subtrees give their
// leaves by decreasing position, each leaf's cells by increasing position.
template <class Id, class Put>
__device__ __forceinline__ void box_outputs(const TreeQ& T, int lane, int64_t share, int64_t at, Id id, int ptr,
                                            int size, unsigned hit, bool all, const Put& put) {
    const unsigned FULL = 0xffffffffu;
    int64_t incl = share;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    const int64_t excl = incl - share, total = __shfl_sync(FULL, incl, 31);
    for (int64_t t0 = 0; t0 < total; t0 += 32) {
        const int64_t t = t0 + lane;
        int k = 0;  // the node of output t: the last one that starts at or before it
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            if (__shfl_sync(FULL, excl, k + o) <= t) k += o;
        const int64_t o = t - __shfl_sync(FULL, excl, k);
        const int kp = __shfl_sync(FULL, ptr, k), ks = __shfl_sync(FULL, size, k);
        unsigned kh = __shfl_sync(FULL, hit, k);
        const int64_t ka = __shfl_sync(FULL, at, k);
        const Id ki = __shfl_sync(FULL, id, k);
        const bool kall = __shfl_sync(FULL, (int)all, k) != 0;
        if (t >= total) continue;
        int j;
        if (kall) {
            const int end = kp + ks, q = end - 1 - (int)o;
            const int s0 = T.lstart[q];
            if (s0 < kp || s0 > q) {  // corrupt index: leave the slot, report
                set_error(T.err, CT_DEVERR_LOOP);
                continue;
            }
            int e = q + 1;
            while (e < end && T.lstart[e] == s0) e++;
            j = s0 + (e - 1 - q);
        } else {
            for (int z = (int)o; z > 0; z--) kh &= kh - 1u;
            j = kp + __ffs(kh) - 1;
        }
        put(ki, ka + o, j, kall);
    }
}

enum { BOX_COUNT = 0, BOX_WRITE = 1, BOX_RECORD = 2 };  // BOX_COUNT: with the scratch, if there is one

template <int MODE>
struct BoxWalk {
    static constexpr bool WRITE = MODE == BOX_WRITE;
    const TreeQ& T;
    const double4* boxes;
    const WalkBox* Q;
    int64_t* emitted;
    int lane;
    int64_t *ii, *jj;
    int* spec;
    int spcap;
    BoxRecs recs;

    __device__ __forceinline__ int visit(int v, int qi, int, int* first, int* second) const {
        const WalkBox& S = Q[qi];
        const float4 q = T.nf[v];
        const double2 d = T.nd[v];
        if (S.idx) {
            const float4 b = *reinterpret_cast<const float4*>(T.nbx + v);  // xmin, xmax, ymin, ymax
            if (b.y < S.ox0 || b.x > S.ox1 || b.w < S.oy0 || b.z > S.oy1) return WALK_DROP;
            if (S.qx0 < b.x && b.y < S.qx1 && S.qy0 < b.z && b.w < S.qy1) return WALK_ALL;
        }
        if (nb(q) >= 0) return WALK_LEAF;
        const int dim = -1 - nb(q);
        bool left, right;
        if (S.keys) {
            left = (dim ? S.ky0 : S.kx0) <= fkey(d.x);
            right = (dim ? S.ky1 : S.kx1) >= fkey(d.y);
        } else {
            const double4 b = boxes[S.id];
            left = (dim ? b.z : b.x) <= d.x;
            right = (dim ? b.w : b.y) >= d.y;
        }
        // the right child is visited first
        const int child = na(q);
        *first = right ? child + 1 : (left ? child : -1);
        *second = (left && right) ? child : -1;
        return *first >= 0 ? WALK_OPEN : WALK_DROP;
    }

    // boxes_intersect geometry_utils.py:292-300
    __device__ __forceinline__ bool overlaps(const WalkBox& S, int j) const {
        const dbox b = leaf_box(T, j);
        return S.keys ? (S.kx0 < fkey(b.xmax) && fkey(b.xmin) < S.kx1 && S.ky0 < fkey(b.ymax) && fkey(b.ymin) < S.ky1)
                      : boxes_intersect(load_box(reinterpret_cast<const double*>(boxes + S.id)), b);
    }

    __device__ __forceinline__ void put(int64_t at, int64_t id, int64_t rank, int j) const {
        if (WRITE) {
            ii[at + rank] = id;
            jj[at + rank] = T.bbi[j];
        } else if (rank < spcap) {
            spec[at + rank] = (int)T.bbi[j];
        }
    }

    // Keeps `parts` records of each lane's node r (of a whole subtree, or one);
    // whether the lane's fit.  `whole`: all of a lane's or none.
    __device__ __forceinline__ bool keep_records(unsigned long long* count, int parts, bool whole, int4 r) const {
        const unsigned FULL = 0xffffffffu;
        const unsigned some = __ballot_sync(FULL, parts > 0), many = __ballot_sync(FULL, parts > 1);
        if (!some) return false;
        int before = __popc(some & ((1u << lane) - 1u)), total = __popc(some);
        if (many) {
            int incl = parts;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            before = incl - parts;
            total = __shfl_sync(FULL, incl, 31);
        }
        unsigned long long first = 0;
        if (lane == 0) first = atomicAdd(count, (unsigned long long)total);
        first = __shfl_sync(FULL, first, 0) + (unsigned)before;
        const unsigned long long cap = (unsigned long long)recs.cap;
        const bool fits = first + (unsigned)parts <= cap;
        if (parts == 1 && fits) recs.rec[first] = r;
        for (unsigned m = many; m; m &= m - 1u) {
            const int src = __ffs(m) - 1, k = __shfl_sync(FULL, parts, src);
            const unsigned long long at = __shfl_sync(FULL, first, src);
            const int id = __shfl_sync(FULL, r.x, src), rank = __shfl_sync(FULL, r.y, src);
            const int ptr = __shfl_sync(FULL, r.z, src), end = ptr + __shfl_sync(FULL, r.w, src);
            const int part = MODE == BOX_RECORD ? REC_PART : recs.part;
            const bool none = whole && at + (unsigned)k > cap;  // slots before the end get no cells
            for (int t = lane; t < k && at + (unsigned)t < cap; t += 32) {
                int p0 = ptr, p1 = end;
                if (t > 0) p0 = max(ptr, min(T.lstart[ptr + t * part], ptr + t * part));
                if (t + 1 < k) p1 = max(p0, min(T.lstart[ptr + (t + 1) * part], end));
                recs.rec[at + (unsigned)t] = none ? make_int4(id, 0, ptr, 0) : make_int4(id, rank + (end - p1), p0, p1 - p0);
            }
        }
        return parts > 0 && fits;
    }

    __device__ __forceinline__ void emit(int v, unsigned meta, bool have) const {
        const unsigned FULL = 0xffffffffu;
        const int qi = have ? (int)(meta & WALK_QMASK) : -1;
        const WalkBox& S = Q[have ? qi : 0];
        const bool all = have && (meta & WALK_WHOLE) != 0;
        int ptr = 0, size = 0;
        unsigned hit = 0;  // the overlapping ones of a leaf's first 32 cells
        int64_t c = 0;
        if (all) {
            const int4 r = reinterpret_cast<const int4*>(T.nbx + v)[1];
            ptr = r.x;
            size = r.y;
            c = size;
        } else if (have) {
            const float4 q = T.nf[v];
            ptr = na(q);
            size = nb(q);
            for (int k = 0; k < size; k++)
                if (overlaps(S, ptr + k)) {
                    if (k < 32) hit |= 1u << k;
                    c++;
                }
        }
        const int64_t rank = walk_rank<int64_t>(qi, c, have, lane, emitted);
        if (MODE == BOX_RECORD) {
            const int parts = c == 0 ? 0 : all && c >= 2 * REC_PART ? (int)c / REC_PART : 1;
            keep_records(recs.count, parts, false,
                         make_int4((int)S.id | (all ? REC_FLAG : 0), (int)rank | (!all && size > 32 ? REC_FLAG : 0), ptr,
                                   all || size > 32 ? size : (int)hit));
            return;
        }
        if (!WRITE && !spec) return;
        const int64_t at = have ? S.base : 0;
        const int64_t id = have ? S.id : 0;
        int64_t share = WRITE ? c : min(c, max((int64_t)0, (int64_t)spcap - rank));
        if (WRITE && recs.rec) {  // whole subtrees to k_box_records
            const int parts = all && c >= recs.part ? (int)c / recs.part : 0;
            if (keep_records(recs.pushed, parts, true, make_int4((int)id | REC_FLAG, (int)rank, ptr, size))) share = 0;
        }
        if (!all && size > 32) {  // a large leaf: its own lane
            int64_t r = rank;
            for (int k = 0; k < size && share > 0; k++)
                if (overlaps(S, ptr + k)) put(at, id, r++, ptr + k);
            share = 0;
        }
        box_outputs(T, lane, share, at + rank, id, ptr, size, hit, all, [&](int64_t i, int64_t k, int j, bool whole) {
            if (WRITE) {
                ii[k] = i;
                jj[k] = T.bbi[j];
                if (recs.inside) recs.inside[k] = whole;
            } else {
                spec[k] = (int)T.bbi[j];
            }
        });
    }
};

template <int MODE>
__global__ void __launch_bounds__(32 * WALK_WARPS, WALK_BLOCKS) k_box_walk(TreeQ T, const double4* __restrict__ boxes, int64_t n,
                                                              const int* __restrict__ order, int per_warp,
                                                              int64_t* __restrict__ cnt_or_off,
                                                              int64_t* __restrict__ ii, int64_t* __restrict__ jj,
                                                              int* __restrict__ spec, int spcap,
                                                              const int64_t* __restrict__ spec_cnt, BoxRecs recs) {
    constexpr bool WRITE = MODE == BOX_WRITE;
    if (WRITE && recs.count && *recs.count <= (unsigned long long)recs.cap) return;  // written from the records
    extern __shared__ __align__(16) unsigned char walk_smem[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    WalkShared<WalkBox, int64_t>& S0 = reinterpret_cast<WalkShared<WalkBox, int64_t>*>(walk_smem)[wi];
    const int64_t t0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + wi) * per_warp;
    if (t0 >= n) return;
    const bool valid = lane < per_warp && t0 + lane < n;
    int64_t i = 0;
    bool start = false;
    if (valid) {
        i = order ? (int64_t)order[t0 + lane] : t0 + lane;
        // writing after a count with scratch: boxes whose pairs all fit it
        // were written from it (k_boxes_spec_emit)
        if (!(WRITE && spec_cnt && spec_cnt[i] <= spcap)) {
            const double4 q4 = boxes[i];
            dbox b;
            b.xmin = q4.x;
            b.xmax = q4.y;
            b.ymin = q4.z;
            b.ymax = q4.w;
            start = boxes_intersect(b, T.bbox);
            if (start) {
                WalkBox& S = S0.query[lane];
                S.keys = T.finite && not_nan(b.xmin) && not_nan(b.xmax) && not_nan(b.ymin) && not_nan(b.ymax);
                S.kx0 = fkey(b.xmin);
                S.kx1 = fkey(b.xmax);
                S.ky0 = fkey(b.ymin);
                S.ky1 = fkey(b.ymax);
                S.idx = S.keys && T.nbx != nullptr;
                const double x0 = b.xmin - T.ox, x1 = b.xmax - T.ox, y0 = b.ymin - T.oy, y1 = b.ymax - T.oy;
                S.qx0 = __double2float_ru(x0);
                S.qx1 = __double2float_rd(x1);
                S.qy0 = __double2float_ru(y0);
                S.qy1 = __double2float_rd(y1);
                S.ox0 = __double2float_rd(x0);
                S.ox1 = __double2float_ru(x1);
                S.oy0 = __double2float_rd(y0);
                S.oy1 = __double2float_ru(y1);
                S.id = i;
                S.base = WRITE ? cnt_or_off[i] : i * (int64_t)spcap;
            }
        }
    }
    if (lane < WALK_Q) S0.count[lane] = 0;
    const int nq = walk_begin(S0.buf, start ? 0 : -1, lane);
    BoxWalk<MODE> pol{T, boxes, S0.query, S0.count, lane, ii, jj, spec, spcap, recs};
    walk(pol, S0.buf, nq, lane, (int64_t)per_warp * (T.n_nodes + 1), T.err);
    __syncwarp();
    if (!WRITE && valid) cnt_or_off[i] = S0.count[lane];
}

// The pairs of the counting pass's records (of the writing pass's, when those
// did not all fit), a warp per 32 of them: no second walk (91M pairs of 250k
// boxes: 1.20 ms, the walk again 4.45).
__global__ void __launch_bounds__(256) k_box_records(TreeQ T, const double4* __restrict__ boxes, BoxRecs recs,
                                                     const int64_t* __restrict__ off, int64_t* __restrict__ ii,
                                                     int64_t* __restrict__ jj) {
    const int lane = threadIdx.x & 31;
    const unsigned long long cap = (unsigned long long)recs.cap, asked = recs.count ? *recs.count : cap + 1;
    // not all were kept: the boxes have been walked again, but for these
    const int64_t n = (int64_t)(asked <= cap ? asked : min(*recs.pushed, cap));
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    auto put = [&](int i, int64_t k, int j, bool whole) {
        ii[k] = i;
        jj[k] = T.bbi[j];
        if (recs.inside) recs.inside[k] = whole;
    };
    for (int64_t r0 = 32 * (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); r0 < n; r0 += 32 * warps) {
        const bool have = r0 + lane < n;
        const int4 r = have ? recs.rec[r0 + lane] : make_int4(0, 0, 0, 0);
        const bool all = have && r.x < 0, big = have && r.y < 0;
        const int id = r.x & ~REC_FLAG;
        int64_t at = have ? off[id] + (r.y & ~REC_FLAG) : 0;
        if (big) {  // a large leaf: its own lane
            const dbox b = load_box(reinterpret_cast<const double*>(boxes + id));
            int64_t k = at;
            for (int c = 0; c < r.w; c++)
                if (boxes_intersect(b, leaf_box(T, r.z + c))) put(id, k++, r.z + c, false);
        }
        const int64_t share = !have || big ? 0 : all ? r.w : __popc((unsigned)r.w);
        box_outputs(T, lane, share, at, id, r.z, all ? r.w : 0, all ? 0u : (unsigned)r.w, all, put);
    }
}

// The cells of each deferred subtree, one warp per subtree, in upstream's
// visiting order (leaves by decreasing position, each leaf's cells by
// increasing position): output o takes reversed position q = end - 1 - o,
// whose leaf [s, e) contributes position s + (e - 1 - q).  Writes and the
// bb_indices reads are coalesced across the warp.
__global__ void __launch_bounds__(256) k_box_jobs(const BoxJob* __restrict__ jobs,
                                                  const unsigned long long* __restrict__ njobs,
                                                  int64_t job_cap, const int* __restrict__ lstart,
                                                  const int64_t* __restrict__ bbi, int64_t* __restrict__ ii,
                                                  int64_t* __restrict__ jj, unsigned int* __restrict__ err) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t nj = (int64_t)min(*njobs, (unsigned long long)job_cap);
    for (int64_t k = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < nj; k += warps) {
        const BoxJob J = jobs[k];
        const int end = J.ptr + J.size;
        bool bad = false;
        for (int o = lane; o < J.size; o += 32) {
            const int q = end - 1 - o;
            const int s0 = lstart[q];
            int e = q + 1;
            while (e < end && lstart[e] == s0) e++;
            const int p = s0 + (e - 1 - q);
            if (s0 < J.ptr || s0 > q) {  // corrupt index: leave the slot, report
                bad = true;
                continue;
            }
            ii[J.out + o] = J.box;
            jj[J.out + o] = bbi[p];
        }
        if (bad) set_error(err, CT_DEVERR_LOOP);
    }
}

// Pairs of the boxes whose count fits the speculative scratch: four lanes a
// box, so that the writes of a box's pairs are contiguous and only slots that
// hold a pair are looked at (a thread per slot, with a division for its box:
// 1M boxes of 3.4 pairs 56 -> 31 us).
__global__ void __launch_bounds__(256) k_boxes_spec_emit(const int64_t* __restrict__ cnt,
                                                         const int64_t* __restrict__ off, int64_t n,
                                                         const int* __restrict__ spec, int cap,
                                                         int64_t* __restrict__ ii, int64_t* __restrict__ jj) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 4 * n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t >> 2, m = cnt[i], o = off[i];
        if (m > cap) continue;
        for (int64_t c = t & 3; c < m; c += 4) {
            ii[o + c] = i;
            jj[o + c] = spec[i * (int64_t)cap + c];
        }
    }
}

// Candidates of the segments whose count fits the counting pass's scratch
// (or the work items': item_seg), 16 lanes a segment (1M segments of some 60
// candidates: 339 -> 117 us).
__global__ void __launch_bounds__(256) k_edge_spec_emit(const int64_t* __restrict__ cnt,
                                                        const int64_t* __restrict__ off, int64_t n,
                                                        const int* __restrict__ item_seg,
                                                        const int* __restrict__ spec, int cap, int* __restrict__ cseg,
                                                        int* __restrict__ cpos) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 16 * n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t >> 4, m = cnt[i], o = off[i];
        if (m > cap) continue;
        const int s = item_seg ? item_seg[i] : (int)i;
        for (int64_t c = t & 15; c < m; c += 16) {
            cseg[o + c] = s;
            cpos[o + c] = spec[i * (int64_t)cap + c];
        }
    }
}

// ---------------------------------------------------------------------------
// locate_edge query.py:357-455 with compute_edge_edge_intersect (292-306,
// mode 0) or compute_edge_face_intersect (309-328, mode 1)
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// locate_edge (query.py:357-455) in two phases: the traversal collects
// candidate (segment, cell) pairs in upstream traversal order; one thread per
// candidate then runs the float64 cell test.  Clipping inside the traversal
// would run with a few lanes of a warp active (every segment's traversal
// differs); per candidate it runs with full warps.  Phase 1 drops only the
// cells that the cell test's own first step (Cohen-Sutherland's
// shared-outcode reject, an exact order comparison) rejects.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cs_code_keys(unsigned long long kx, unsigned long long ky, unsigned long long x0,
                                            unsigned long long x1, unsigned long long y0, unsigned long long y1) {
    int p = CS_INSIDE;
    if (kx < x0) p |= CS_LEFT;
    else if (kx > x1) p |= CS_RIGHT;
    if (ky < y0) p |= CS_LOWER;
    else if (ky > y1) p |= CS_UPPER;
    return p;
}

// Line filter of the segment traversal (no upstream counterpart).  A cell
// whose box the segment's line misses by more than a margin m cannot be a
// result: Cohen-Sutherland (cohen_sutherland.py:32-101) then rejects it --
// each clipping step puts an endpoint on a box edge line at most a few
// float64 roundings (of the coordinates' magnitude C) off the line, so every
// point it computes stays outside the box, on the side the exact algorithm's
// does, and the exact algorithm rejects a segment that misses the box (a
// segment whose line meets the box beyond an endpoint shares an outcode bit
// and is rejected by the outcode test) -- and for edge trees
// lines_intersect (geometry_utils.py:361-418) finds both tree edge
// endpoints strictly on one side of the segment's line and not within its
// tolerance (1e-12 of the edge length) of it.  m = 2^-40 C (C: the largest
// |coordinate| of the segment and the tree's bbox) + 2^-37 x the tree's
// extent + 2^-47 covers both by orders of magnitude.  The test runs in
// float32 in the tree's frame on node boxes and cell boxes rounded outward:
// f = n . (corner - a) at the corner nearest the line's side, against a
// bound on the float32 and conversion errors (2^-19 of the products'
// magnitudes plus the frame magnitudes) plus m |n|.  Pruning only removes
// cells that produce no result, so results and their order are unchanged.
struct LineF {
    float ax, ay, nx, ny, K, em;
    bool on;
};

__device__ __forceinline__ LineF line_filter(const TreeQ& T, dpt a, dpt b, dpt V, bool keys) {
    LineF L;
    L.on = keys && T.bbl32 != nullptr;
    L.ax = L.ay = L.nx = L.ny = L.K = L.em = 0.0f;
    if (!L.on) return L;
    L.ax = __double2float_rn(a.x - T.ox);
    L.ay = __double2float_rn(a.y - T.oy);
    L.nx = __double2float_rn(-V.y);
    L.ny = __double2float_rn(V.x);
    const float anx = fabsf(L.nx), any = fabsf(L.ny);
    L.K = __fadd_ru(__fmul_ru(anx, __fadd_ru(fabsf(L.ax), T.fX)), __fmul_ru(any, __fadd_ru(fabsf(L.ay), T.fY)));
    const double C = fmax(fmax(fmax(fabs(a.x), fabs(a.y)), fmax(fabs(b.x), fabs(b.y))), T.babs);
    const float m = __double2float_ru(__dadd_ru(__dmul_ru(C, 0x1p-40), T.mext));
    L.em = __fmul_ru(__fmul_ru(m, __fadd_ru(anx, any)), 1.0f + 0x1p-18f);
    // a non-finite term switches the filter off (its comparisons would be false anyway)
    L.on = isfinite(L.K) && isfinite(L.em) && isfinite(L.ax) && isfinite(L.ay);
    return L;
}

// Whether the segment's line surely misses the float32 box (frame of the tree).
__device__ __forceinline__ bool line_misses(const LineF& L, float x0, float x1, float y0, float y1) {
    const float px = L.nx > 0.0f ? x0 : x1, qx = L.nx > 0.0f ? x1 : x0;
    const float py = L.ny > 0.0f ? y0 : y1, qy = L.ny > 0.0f ? y1 : y0;
    const float dpx = __fsub_rn(px, L.ax), dpy = __fsub_rn(py, L.ay);
    const float dqx = __fsub_rn(qx, L.ax), dqy = __fsub_rn(qy, L.ay);
    const float t1 = __fmul_rn(L.nx, dpx), t2 = __fmul_rn(L.ny, dpy);
    const float u1 = __fmul_rn(L.nx, dqx), u2 = __fmul_rn(L.ny, dqy);
    const float fmin = __fadd_rn(t1, t2), fmax_ = __fadd_rn(u1, u2);
    const float emin = __fadd_ru(__fmul_ru(__fadd_ru(__fadd_ru(fabsf(t1), fabsf(t2)), L.K), 0x1p-19f),
                                 __fadd_ru(L.em, 0x1p-100f));
    const float emax = __fadd_ru(__fmul_ru(__fadd_ru(__fadd_ru(fabsf(u1), fabsf(u2)), L.K), 0x1p-19f),
                                 __fadd_ru(L.em, 0x1p-100f));
    return fmin > emin || fmax_ < -emax;
}

// Segment a -> b against the cells of leaf `v` (nf q): the candidates that
// Cohen-Sutherland's shared-outcode test does not reject (mode 1), or every
// cell (mode 0), counted and, with WRITE, written at cseg / cj[base + count].
template <bool WRITE, int MODE>
__device__ __forceinline__ void edge_leaf(const TreeQ& T, float4 q, dpt a, dpt b, bool keys, unsigned long long kax,
                                          unsigned long long kay, unsigned long long kbx, unsigned long long kby,
                                          int64_t i, int64_t base, int64_t& count, int* __restrict__ cseg,
                                          int* __restrict__ cj, int spcap = 0) {
    int ptr = na(q), bq = nb(q);
    for (int j = ptr; j < ptr + bq; j++) {
        bool cand = true;
        if (MODE == 1) {
            dbox bx = leaf_box(T, j);
            int k1, k2;
            if (keys) {
                unsigned long long x0 = fkey(bx.xmin), x1 = fkey(bx.xmax), y0 = fkey(bx.ymin), y1 = fkey(bx.ymax);
                k1 = cs_code_keys(kax, kay, x0, x1, y0, y1);
                k2 = cs_code_keys(kbx, kby, x0, x1, y0, y1);
            } else {
                k1 = cs_code(a, bx);
                k2 = cs_code(b, bx);
            }
            cand = (k1 & k2) == 0;
        }
        if (cand) {
            if (WRITE) {
                cseg[base + count] = (int)i;
                cj[base + count] = j;
            } else if (count < spcap) {
                cj[count] = j;  // counting pass: the segment's scratch row
            }
            count++;
        }
    }
}

// Children of internal node v the segment's traversal enters (locate_edge
// query.py:410-441): `first` is visited first (the right child when both).
__device__ __forceinline__ void edge_children(const TreeQ& T, double2 nd, float4 q, dpt a, dpt b, dpt V, bool keys,
                                              unsigned long long kax, unsigned long long kay,
                                              unsigned long long kbx, unsigned long long kby, int* first,
                                              int* second) {
    int dim = -1 - nb(q);
    double dx = dim ? V.y : V.x;
    bool left, right;
    if (keys) {
        unsigned long long ka = dim ? kay : kax, kb = dim ? kby : kbx;
        bool pos = dx > 0.0;
        left = fkey(nd.x) >= (pos ? ka : kb);
        right = fkey(nd.y) <= (pos ? kb : ka);
    } else {
        double an = dim ? a.y : a.x, bn = dim ? b.y : b.x;
        double dx_left, dx_right;
        if (dx > 0.0) {
            dx_left = nd.x - an;
            dx_right = nd.y - bn;
        } else {
            dx_left = nd.x - bn;
            dx_right = nd.y - an;
        }
        left = dx_left >= 0.0;
        right = dx_right <= 0.0;
        if (dx > 0.0) {
            if (left) left = (dx_left / dx) >= 0.0;
            if (right) right = (dx_right / dx) <= 1.0;
        } else if (dx < 0.0) {
            if (left) left = (1.0 - (dx_left / dx)) >= 0.0;
            if (right) right = (1.0 - (dx_right / dx)) <= 1.0;
        }
    }
    // pushed left, then right: the right child is visited first
    int child = na(q);
    *first = right ? child + 1 : (left ? child : -1);
    *second = (left && right) ? child : -1;
}

struct EdgeKeys {
    bool keys;
    unsigned long long kax, kay, kbx, kby;
};

__device__ __forceinline__ EdgeKeys edge_keys(const TreeQ& T, dpt a, dpt b) {
    dpt V = vsub(b, a);
    EdgeKeys k;
    k.keys = T.finite && is_fin(a.x) && is_fin(a.y) && is_fin(b.x) && is_fin(b.y) && is_fin(V.x) && is_fin(V.y);
    k.kax = fkey(a.x);
    k.kay = fkey(a.y);
    k.kbx = fkey(b.x);
    k.kby = fkey(b.y);
    return k;
}

// ---------------------------------------------------------------------------
// The traversal by warps (ct_walk.cuh): one task per segment from the root,
// or one per work item (segment, node) of a cut traversal.  With ITEMS it
// stops `cut` levels below the root (and at leaves above) and reports those
// nodes instead of their candidates: the cut splits a long segment's
// traversal into subtrees whose candidate lists, concatenated in this order,
// are the traversal's.  Counts per task, or with WRITE the candidates (nodes)
// at their offsets.
//
// Bound by reading the nodes (90 B each) where the segments come in no order;
// 8 tasks per warp fill the rounds of short segments.  The two cut
// passes and the two item passes of 1000 segments across a mesh of 5M cells:
// 1.73 -> 0.72 ms; 1M short segments uncut: 7.0 ms as with one thread per
// segment.
// ---------------------------------------------------------------------------
struct WalkSeg {  // 88 bytes, as WalkBox
    unsigned long long kax, kay, kbx, kby;
    LineF lf;
    int seg;
    int64_t base;
    bool keys, posx, posy;
    int64_t pad;
};

template <int MODE, bool ITEMS, bool WRITE>
struct SegWalk {
    const TreeQ& T;
    const double4* segs;
    const WalkSeg* Q;
    int* emitted;
    int lane, cut;
    int *out_seg, *out_val;  // WRITE: at the task's offset; else the scratch rows
    int spcap;

    __device__ __forceinline__ int visit(int v, int qi, int depth, int* first, int* second) const {
        const WalkSeg& S = Q[qi];
        // the node's records loaded together (one round trip per node)
        const float4 q = T.nf[v];
        const double2 nd = T.nd[v];
        if (S.lf.on) {
            const float4 nbx = *reinterpret_cast<const float4*>(T.nbx + v);
            if (line_misses(S.lf, nbx.x, nbx.y, nbx.z, nbx.w)) return WALK_DROP;
        }
        if (nb(q) >= 0 || (ITEMS && depth >= cut)) return WALK_LEAF;
        if (S.keys) {
            const int dim = -1 - nb(q);
            const bool pos = dim ? S.posy : S.posx;
            const unsigned long long ka = dim ? S.kay : S.kax, kb = dim ? S.kby : S.kbx;
            const bool left = fkey(nd.x) >= (pos ? ka : kb), right = fkey(nd.y) <= (pos ? kb : ka);
            const int child = na(q);
            *first = right ? child + 1 : (left ? child : -1);
            *second = (left && right) ? child : -1;
        } else {
            const double4 s4 = segs[S.seg];
            const dpt a = mkp(s4.x, s4.y), b = mkp(s4.z, s4.w);
            edge_children(T, nd, q, a, b, vsub(b, a), false, 0, 0, 0, 0, first, second);
        }
        return *first >= 0 ? WALK_OPEN : WALK_DROP;
    }

    // whether the cell at leaf position j is a candidate of segment S (as
    // edge_leaf)
    __device__ __forceinline__ bool candidate(const WalkSeg& S, int j) const {
        if (S.lf.on) {
            const float4 c = T.bbl32[j];
            if (line_misses(S.lf, c.x, c.y, c.z, c.w)) return false;
        }
        if (MODE == 0) return true;
        const dbox bx = leaf_box(T, j);
        if (S.keys) {
            const unsigned long long x0 = fkey(bx.xmin), x1 = fkey(bx.xmax), y0 = fkey(bx.ymin), y1 = fkey(bx.ymax);
            return (cs_code_keys(S.kax, S.kay, x0, x1, y0, y1) & cs_code_keys(S.kbx, S.kby, x0, x1, y0, y1)) == 0;
        }
        const double4 s4 = segs[S.seg];
        return (cs_code(mkp(s4.x, s4.y), bx) & cs_code(mkp(s4.z, s4.w), bx)) == 0;
    }

    __device__ __forceinline__ void put(const WalkSeg& S, int rank, int val) const {
        if (WRITE) {
            out_seg[S.base + rank] = S.seg;
            out_val[S.base + rank] = val;
        } else if (rank < spcap) {
            out_val[S.base + rank] = val;  // counting pass: the segment's scratch row
        }
    }

    __device__ __forceinline__ void emit(int v, unsigned meta, bool have) const {
        const int qi = have ? (int)(meta & WALK_QMASK) : -1;
        const WalkSeg& S = Q[have ? qi : 0];
        int ptr = 0, size = 0, c = have ? 1 : 0;
        unsigned hit = 0;  // the first 32 cells of the leaf
        if (!ITEMS) {
            c = 0;
            if (have) {
                const float4 q = T.nf[v];
                ptr = na(q);
                size = nb(q);
            }
            for (int k = 0; k < size; k++)
                if (candidate(S, ptr + k)) {
                    if (k < 32) hit |= 1u << k;
                    c++;
                }
        }
        int r = walk_rank<int>(qi, c, have, lane, emitted);
        if (ITEMS) {
            if (have) put(S, r, v);
        } else if (c > 0 && (WRITE || spcap > 0)) {
            for (unsigned h = hit; h; h &= h - 1u) put(S, r++, ptr + __ffs(h) - 1);
            for (int k = 32; k < size; k++)
                if (candidate(S, ptr + k)) put(S, r++, ptr + k);
        }
    }
};

template <int MODE, bool ITEMS, bool WRITE>
__global__ void __launch_bounds__(32 * WALK_WARPS, WALK_BLOCKS) k_edge_walk(
    TreeQ T, const double4* __restrict__ segs, int64_t n, const int* __restrict__ order,
    const int* __restrict__ item_seg, const int* __restrict__ item_node, int cut, int per_warp,
    int64_t* __restrict__ cnt_or_off, int* __restrict__ out_seg, int* __restrict__ out_val, int spcap,
    const int64_t* __restrict__ spec_cnt) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    WalkShared<WalkSeg, int>& S0 = reinterpret_cast<WalkShared<WalkSeg, int>*>(walk_smem)[wi];
    const int64_t t0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + wi) * per_warp;
    if (t0 >= n) return;
    const bool valid = lane < per_warp && t0 + lane < n;
    int64_t row = 0;
    int start = -1;
    if (valid) {
        const int64_t k = t0 + lane;
        const int64_t i = item_seg ? (int64_t)item_seg[k] : order ? (int64_t)order[k] : k;
        row = item_seg ? k : i;
        // written already: the candidates fit the counting pass's scratch
        if (!(WRITE && spec_cnt && spec_cnt[row] <= spcap)) {
            const double4 s4 = segs[i];
            const dpt a = mkp(s4.x, s4.y), b = mkp(s4.z, s4.w);
            if (item_node) {
                start = item_node[k];
            } else {  // segments that miss the tree's bbox have none
                dpt c, d;
                const int r = cohen_sutherland(a, b, T.bbox, &c, &d);
                if (r < 0) set_error(T.err, CT_DEVERR_LOOP);
                if (r == 1) start = 0;
            }
            if (start >= 0) {
                const dpt V = vsub(b, a);
                const EdgeKeys K = edge_keys(T, a, b);
                WalkSeg& S = S0.query[lane];
                S.kax = K.kax;
                S.kay = K.kay;
                S.kbx = K.kbx;
                S.kby = K.kby;
                S.lf = line_filter(T, a, b, V, K.keys);
                S.keys = K.keys;
                S.posx = V.x > 0.0;
                S.posy = V.y > 0.0;
                S.seg = (int)i;
                S.base = WRITE ? cnt_or_off[row] : row * (int64_t)spcap;
            }
        }
    }
    if (lane < WALK_Q) S0.count[lane] = 0;
    const int nq = walk_begin(S0.buf, start, lane);
    SegWalk<MODE, ITEMS, WRITE> pol{T, segs, S0.query, S0.count, lane, cut, out_seg, out_val, spcap};
    walk(pol, S0.buf, nq, lane, (int64_t)per_warp * (T.n_nodes + 1), T.err);
    __syncwarp();
    if (!WRITE && valid) cnt_or_off[row] = S0.count[lane];
}

// Trees deeper than the walk's reserve: one thread per segment through the
// parent links (see k_boxes).
// spcap > 0: in the counting pass cj is a scratch of spcap entries per
// segment that keeps its first candidates; in the writing pass spec_cnt
// holds the counts and segments whose candidates fit were copied from the
// scratch (k_edge_spec_emit), so they return at once.
template <bool WRITE, int MODE>
__global__ void __launch_bounds__(128) k_edge_cands_deep(TreeQ T, const double4* __restrict__ segs, int64_t n,
                                                         const int* __restrict__ order,
                                                         int64_t* __restrict__ cnt_or_off, int* __restrict__ cseg,
                                                         int* __restrict__ cj, int spcap = 0,
                                                         const int64_t* __restrict__ spec_cnt = nullptr) {
    int64_t tq = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tq >= n) return;
    int64_t i = order ? (int64_t)order[tq] : tq;
    if (WRITE && spec_cnt && spec_cnt[i] <= spcap) return;
    if (!WRITE && spcap > 0) cj += i * (int64_t)spcap;
    double4 s4 = segs[i];
    dpt a = mkp(s4.x, s4.y), b = mkp(s4.z, s4.w);
    int64_t count = 0;
    int64_t base = WRITE ? cnt_or_off[i] : 0;
    dpt c, d;
    int r = cohen_sutherland(a, b, T.bbox, &c, &d);
    if (r < 0) set_error(T.err, CT_DEVERR_LOOP);
    if (r == 1) {
        const dpt V = vsub(b, a);
        const EdgeKeys K = edge_keys(T, a, b);
        int dv = 0, from = -1;
        bool down = true;
        int64_t budget = 2 * T.n_nodes + 2;
        while (dv >= 0) {
            if (--budget < 0) {
                set_error(T.err, CT_DEVERR_LOOP);
                break;
            }
            const int v = dv;
            float4 q = T.nf[v];
            int first = -1, second = -1;
            const bool terminal = nb(q) >= 0;
            if (terminal && down)
                edge_leaf<WRITE, MODE>(T, q, a, b, K.keys, K.kax, K.kay, K.kbx, K.kby, i, base, count, cseg, cj,
                                       WRITE ? 0 : spcap);
            if (!terminal)
                edge_children(T, T.nd[v], q, a, b, V, K.keys, K.kax, K.kay, K.kbx, K.kby, &first, &second);
            int next = terminal ? -1 : (down ? first : ((from == first) ? second : -1));
            from = dv;
            if (next >= 0) {
                dv = next;
                down = true;
            } else {
                dv = T.parent[dv];
                down = false;
            }
        }
    }
    if (!WRITE) cnt_or_off[i] = count;
}

// Per segment: the offset and count of its candidates, from its items'
// (items are segment-major; a segment's items are [ioff[s], ioff[s] + icnt[s])).
__global__ void k_seg_from_items(const int64_t* __restrict__ ioff, const int64_t* __restrict__ icnt, int64_t n,
                                 const int64_t* __restrict__ item_coff, const int64_t* __restrict__ item_ccnt,
                                 int64_t n_items, int64_t* __restrict__ coff, int64_t* __restrict__ ccnt) {
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k0 = ioff[s], k1 = k0 + icnt[s];
        const int64_t total = n_items > 0 ? item_coff[n_items - 1] + item_ccnt[n_items - 1] : 0;
        const int64_t c0 = k0 < n_items ? item_coff[k0] : total;
        const int64_t c1 = k1 < n_items ? item_coff[k1] : total;
        coff[s] = c0;
        ccnt[s] = c1 - c0;
    }
}

// Sign of the cross product (v - a) x s used by Cyrus-Beck's crossing walk
// (cyrus_beck.py:162-180: ksi / eta) decided in float32 in the cell's local
// frame: -1 / +1 when sure (then also nonzero), 0 when the float64 product
// must be computed.  dv, da: float32 local coordinates of v and a (error ev
// per component), sf: float32 s with error es.  The float64 value is
// fl(fl(U.x * s.y) - fl(U.y * s.x)) with U = fl(v - a): within
// 3.0001 u (|U.x||s.y| + |U.y||s.x|) (u = 2^-53) of the exact product of the
// float64 inputs, so a float32 margin above that bound plus the float32
// error fixes its sign.
__device__ __forceinline__ int cb_sign32(float2 dv, float2 da, float ev, float2 sf, float es) {
    const float u24 = 5.9604644775390625e-08f;
    float ux = dv.x - da.x, uy = dv.y - da.y;
    float eu = 2.0f * ev + u24 * fmaxf(fabsf(ux), fabsf(uy));
    float M = fmaxf(fabsf(ux), fabsf(uy)) + eu;
    float Ns = fabsf(sf.x) + fabsf(sf.y) + 2.0f * es;
    float est = ux * sf.y - uy * sf.x;
    float thr = 1.02f * (2.0f * es * M + Ns * eu + 4.0f * u24 * Ns * M + 3.3307e-16f * Ns * M) + 1e-37f;
    if (!(fabsf(est) > thr)) return 0;
    return est > 0.0f ? 1 : -1;
}

// cyrus_beck_line_polygon_clip (cyrus_beck.py:133-241) with its float64
// decisions screened in float32: the two point_in_polygon_or_on_edge tests by
// the certified leaf filter (ct_locf.cuh), the crossing walk's signs by
// cb_sign32; undecided ones run in float64.  The intersection parameters and
// clipped points are the float64 computations of cyrus_beck().
template <int KT>
__device__ __forceinline__ bool cyrus_beck_f32(dpt a, dpt b, const dpt* poly, int length, double tol,
                                               const float4* __restrict__ cellf, int len32, float dabs, dpt* c,
                                               dpt* d) {
    *c = mkp(dnan(), dnan());
    *d = *c;
    dpt s = vsub(b, a);
    if (s.x == 0 && s.y == 0) return false;
    float tolf = (float)tol;
    if ((double)tolf < tol) tolf = nextafterf(tolf, INFINITY);
    PtSplit Pa = split_point(a.x, a.y), Pb = split_point(b.x, b.y);
    int ra = leaf_filter_local<KT>(Pa, dabs, tolf, cellf, len32);
    int rb = leaf_filter_local<KT>(Pb, dabs, tolf, cellf, len32);
    bool a_inside = (ra == LF_UNSURE) ? pip_or_edge(a, poly, length, tol) : (ra == LF_INSIDE);
    bool b_inside = (rb == LF_UNSURE) ? pip_or_edge(b, poly, length, tol) : (rb == LF_INSIDE);
    if (a_inside && b_inside) {
        *c = a;
        *d = b;
        return true;
    }
    // float32 local coordinates of a and s (frame: the cell's first vertex)
    float da_x, da_y, ea, db_x, db_y, eb;
    local_delta(Pa, cellf[0], &da_x, &da_y, &ea);
    local_delta(Pb, cellf[0], &db_x, &db_y, &eb);
    const float u24 = 5.9604644775390625e-08f;
    const float ed = fmaxf(ea, eb) + dabs;
    const float2 da = make_float2(da_x, da_y);
    const float2 sf = make_float2(db_x - da_x, db_y - da_y);
    const float es = 2.0f * ed + 2.0f * u24 * fmaxf(fabsf(sf.x), fabsf(sf.y));
    const float2* rel = reinterpret_cast<const float2*>(cellf + 1);
    // poly[i] in the local frame: vertex 0 at the origin, the others as their
    // stored float32 offsets (rounded by 2^-24 of their size)
    float vmax = 0.0f;
    for (int i = 1; i < len32 && i < KT; i++) vmax = fmaxf(vmax, fmaxf(fabsf(rel[i - 1].x), fabsf(rel[i - 1].y)));
    const float ev = ed + u24 * vmax + dabs;
    // the float32 cell lists the same vertices as poly unless repeated ones were dropped
    const bool use32 = (len32 == length);
    int i0 = -1, i1 = -1, i = 0, k = 0;
    int sk = use32 ? cb_sign32(make_float2(0.0f, 0.0f), da, ev, sf, es) : 0;
    bool ksi64 = sk == 0;
    double ksi = ksi64 ? crossp(vsub(poly[0], a), s) : 0.0;
    while (i < length && k < 2) {
        const int in = (i + 1) % length;
        int se = use32 ? cb_sign32(in == 0 ? make_float2(0.0f, 0.0f) : rel[in - 1], da, ev, sf, es) : 0;
        const bool eta64 = se == 0;
        const double eta = eta64 ? crossp(vsub(poly[in], a), s) : 0.0;
        const bool ksi_neg = ksi64 ? (ksi < 0.0) : (sk < 0);
        const bool eta_neg = eta64 ? (eta < 0.0) : (se < 0);
        if (ksi_neg != eta_neg) {
            if (k == 0) i0 = i;
            else i1 = i;
            k++;
        } else if (ksi64 && eta64 && ksi == 0.0 && eta == 0.0) {
            bool r = cb_collinear(a, b, poly[i], poly[in], c, d);
            if (!r) {
                *c = mkp(dnan(), dnan());
                *d = *c;
            }
            return r;
        }
        ksi = eta;
        sk = se;
        ksi64 = eta64;
        i++;
    }
    if (k == 0) return false;
    // intersections cyrus_beck.py:46-63 (Python index -1 wraps)
    int j0 = i0 < 0 ? i0 + length : i0, j1 = i1 < 0 ? i1 + length : i1;
    dpt v0 = poly[j0], v01 = poly[(i0 + 1) % length];
    dpt v1 = poly[j1], v11 = poly[((i1 + 1) % length + length) % length];
    bool e0, e1;
    double t0 = cb_param(a, s, v0, v01, &e0);
    double t1 = cb_param(a, s, v1, v11, &e1);
    if (e1) {
        double t = t0;
        t0 = t1;
        t1 = t;
    }
    if (t0 == t1) {
        if (a_inside && t1 != 0.0) t0 = 0.0;
        else if (b_inside && t0 != 1.0) t1 = 1.0;
        else return false;
    }
    if (t1 < t0) {
        double t = t0;
        t0 = t1;
        t1 = t;
    }
    bool valid0 = t0 >= 0 && t0 < 1;
    bool valid1 = t1 > 0 && t1 <= 1;
    if (valid0 && valid1) {
        *c = mkp(a.x + t0 * s.x, a.y + t0 * s.y);
        *d = mkp(a.x + t1 * s.x, a.y + t1 * s.y);
        return true;
    } else if (valid0) {
        *c = mkp(a.x + t0 * s.x, a.y + t0 * s.y);
        *d = b;
        return true;
    } else if (valid1) {
        *c = a;
        *d = mkp(a.x + t1 * s.x, a.y + t1 * s.y);
        return true;
    }
    return false;
}

// ---------------------------------------------------------------------------
// Cohen-Sutherland's verdict in float32 intervals (no upstream counterpart)
// ---------------------------------------------------------------------------
// cohen_sutherland() above is replayed in the cell's local frame (the float32
// cell: its first vertex split hi + lo, the other vertices as offsets) on
// intervals with directed rounding.  Every interval encloses the float64 value
// upstream's code computes at that step: inputs enclose the exact local
// coordinates, each operation's result is widened by the float64 rounding of
// that operation (2^-51 of its magnitude, plus 2^-50 of the largest absolute
// coordinate where the result is an absolute coordinate).  When every outcode
// test and every dx == dy == 0 test is decided for the whole interval, the
// float64 run takes the same path, so its verdict is known: 1 accept, 0
// reject; -1 when any test is undecided (the caller runs the float64 clip).
// Only the verdict is used: upstream overwrites the clipped points with
// Cyrus-Beck's.
struct FI {
    float lo, hi;
};
__device__ __forceinline__ FI fi_sub(FI a, FI b) { return FI{__fsub_rd(a.lo, b.hi), __fsub_ru(a.hi, b.lo)}; }
__device__ __forceinline__ FI fi_add(FI a, FI b) { return FI{__fadd_rd(a.lo, b.lo), __fadd_ru(a.hi, b.hi)}; }
__device__ __forceinline__ FI fi_mul(FI a, FI b) {
    const float l = fminf(fminf(__fmul_rd(a.lo, b.lo), __fmul_rd(a.lo, b.hi)),
                          fminf(__fmul_rd(a.hi, b.lo), __fmul_rd(a.hi, b.hi)));
    const float h = fmaxf(fmaxf(__fmul_ru(a.lo, b.lo), __fmul_ru(a.lo, b.hi)),
                          fmaxf(__fmul_ru(a.hi, b.lo), __fmul_ru(a.hi, b.hi)));
    return FI{l, h};
}
// b must exclude 0
__device__ __forceinline__ FI fi_div(FI a, FI b) {
    const float l = fminf(fminf(__fdiv_rd(a.lo, b.lo), __fdiv_rd(a.lo, b.hi)),
                          fminf(__fdiv_rd(a.hi, b.lo), __fdiv_rd(a.hi, b.hi)));
    const float h = fmaxf(fmaxf(__fdiv_ru(a.lo, b.lo), __fdiv_ru(a.lo, b.hi)),
                          fmaxf(__fdiv_ru(a.hi, b.lo), __fdiv_ru(a.hi, b.hi)));
    return FI{l, h};
}
__device__ __forceinline__ bool fi_ok(FI a) { return isfinite(a.lo) && isfinite(a.hi) && a.lo <= a.hi; }
__device__ __forceinline__ bool fi_has0(FI a) { return !(a.lo > 0.0f || a.hi < 0.0f); }
// float64 rounding of one operation: 2^-51 of the result's magnitude, plus
// `w` (2^-50 of the largest absolute coordinate) for absolute coordinates
__device__ __forceinline__ FI fi_round(FI a, float w) {
    const float e = __fadd_ru(__fmul_ru(fmaxf(fabsf(a.lo), fabsf(a.hi)), 0x1p-51f), w + 0x1p-126f);
    return FI{__fsub_rd(a.lo, e), __fadd_ru(a.hi, e)};
}

// Outcode of an interval point (-1: undecided); a coordinate set to a box
// side (tag >= 0) is exactly that side.
__device__ __forceinline__ int fi_code(FI x, FI y, int tx, int ty, const FI* B) {
    int p = 0;
    if (tx < 0) {
        if (x.hi < B[0].lo) p |= CS_LEFT;
        else if (x.lo >= B[0].hi && x.lo > B[1].hi) p |= CS_RIGHT;
        else if (!(x.lo >= B[0].hi && x.hi <= B[1].lo)) return -1;
    }
    if (ty < 0) {
        if (y.hi < B[2].lo) p |= CS_LOWER;
        else if (y.lo >= B[2].hi && y.lo > B[3].hi) p |= CS_UPPER;
        else if (!(y.lo >= B[2].hi && y.hi <= B[3].lo)) return -1;
    }
    return p;
}

__device__ __forceinline__ int cs_f32(dpt a, dpt b, const dbox& box, const float4* __restrict__ cellf, int len32,
                                      float dabs) {
    // non-finite endpoints and cells of fewer than two distinct vertices
    // (no float32 frame) take the float64 clip
    if (!(is_fin(a.x) && is_fin(a.y) && is_fin(b.x) && is_fin(b.y)) || len32 < 2) return -1;
    // the exact tests on the inputs, as upstream
    if (g_eq_finite(a.x, b.x) && g_eq_finite(a.y, b.y)) return 0;
    int k1 = cs_code(a, box), k2 = cs_code(b, box);
    if ((k1 | k2) == 0) return 1;
    if ((k1 & k2) != 0) return 0;
    // local frame: intervals of the endpoints and the box sides
    const PtSplit Pa = split_point(a.x, a.y), Pb = split_point(b.x, b.y);
    float ax, ay, ea, bx, by, eb;
    local_delta(Pa, cellf[0], &ax, &ay, &ea);
    local_delta(Pb, cellf[0], &bx, &by, &eb);
    const float2* rel = reinterpret_cast<const float2*>(cellf + 1);
    float x0 = 0.0f, x1 = 0.0f, y0 = 0.0f, y1 = 0.0f, vmax = 0.0f;
    for (int i = 1; i < len32 && i < 8; i++) {
        const float2 r = rel[i - 1];
        x0 = fminf(x0, r.x);
        x1 = fmaxf(x1, r.x);
        y0 = fminf(y0, r.y);
        y1 = fmaxf(y1, r.y);
        vmax = fmaxf(vmax, fmaxf(fabsf(r.x), fabsf(r.y)));
    }
    // stored offsets: float32 roundings of the float64 differences
    const float ev = __fadd_ru(__fmul_ru(vmax, 0x1p-22f), dabs + 0x1p-126f);
    const float ep = fmaxf(ea, eb) + dabs + 0x1p-126f;
    FI B[4] = {FI{__fsub_rd(x0, ev), __fadd_ru(x0, ev)}, FI{__fsub_rd(x1, ev), __fadd_ru(x1, ev)},
               FI{__fsub_rd(y0, ev), __fadd_ru(y0, ev)}, FI{__fsub_rd(y1, ev), __fadd_ru(y1, ev)}};
    FI Ax{__fsub_rd(ax, ep), __fadd_ru(ax, ep)}, Ay{__fsub_rd(ay, ep), __fadd_ru(ay, ep)};
    FI Bx{__fsub_rd(bx, ep), __fadd_ru(bx, ep)}, By{__fsub_rd(by, ep), __fadd_ru(by, ep)};
    int tax = -1, tay = -1, tbx = -1, tby = -1;
    // 2^-50 of the largest absolute coordinate of the segment and the cell
    const float C = fmaxf(fmaxf(fmaxf(fabsf(Pa.xh), fabsf(Pa.yh)), fmaxf(fabsf(Pb.xh), fabsf(Pb.yh))),
                          fmaxf(fabsf(cellf[0].x), fabsf(cellf[0].z)) + vmax);
    const float w = __fmul_ru(__fmul_ru(C, 1.0f + 0x1p-20f), 0x1p-50f);
    if (!(fi_ok(Ax) && fi_ok(Ay) && fi_ok(Bx) && fi_ok(By) && isfinite(w))) return -1;
    for (int iter = 0; iter < 8; iter++) {
        if ((k1 | k2) == 0) return 1;
        if ((k1 & k2) != 0) return 0;
        const int opt = k1 ? k1 : k2;
        const FI DX = fi_round(fi_sub(Bx, Ax), 0.0f), DY = fi_round(fi_sub(By, Ay), 0.0f);
        FI x, y;
        int tx = -1, ty = -1;
        if (opt & (CS_UPPER | CS_LOWER)) {
            if (fi_has0(DY)) return -1;
            const int side = (opt & CS_UPPER) ? 3 : 2;
            const FI t = fi_round(fi_div(fi_round(fi_mul(DX, fi_round(fi_sub(B[side], Ay), 0.0f)), 0.0f), DY), 0.0f);
            x = fi_round(fi_add(Ax, t), w);
            y = B[side];
            ty = side;
        } else {
            if (fi_has0(DX)) return -1;
            const int side = (opt & CS_RIGHT) ? 1 : 0;
            const FI t = fi_round(fi_div(fi_round(fi_mul(DY, fi_round(fi_sub(B[side], Ax), 0.0f)), 0.0f), DX), 0.0f);
            y = fi_round(fi_add(Ay, t), w);
            x = B[side];
            tx = side;
        }
        if (!(fi_ok(x) && fi_ok(y))) return -1;
        if (opt == k1) {
            Ax = x;
            Ay = y;
            tax = tx;
            tay = ty;
            k1 = fi_code(Ax, Ay, tax, tay, B);
            if (k1 < 0) return -1;
        } else {
            Bx = x;
            By = y;
            tbx = tx;
            tby = ty;
            k2 = fi_code(Bx, By, tbx, tby, B);
            if (k2 < 0) return -1;
        }
        // dx == 0 and dy == 0: equal coordinates are certain when both were
        // set to the same box side, unequal when the intervals are disjoint
        const bool xeq = tax >= 0 && tax == tbx, yeq = tay >= 0 && tay == tby;
        const bool xne = Ax.hi < Bx.lo || Bx.hi < Ax.lo, yne = Ay.hi < By.lo || By.hi < Ay.lo;
        if (xeq && yeq) return 0;
        if (!(xne || yne)) return -1;
    }
    return -1;
}

// The test of one candidate as upstream runs it (compute_edge_face_intersect
// query.py:309-328): Cohen-Sutherland against the cell's box, then
// Cyrus-Beck.
__device__ __noinline__ bool edge_face_general(const TreeQ& T, dpt a, dpt b, int j, dpt* c, dpt* d) {
    dbox bx = leaf_box(T, j);
    int rr = -1;
    if (T.polyf && T.K <= 8) rr = cs_f32(a, b, bx, T.polyf + (size_t)j * T.S4, (int)T.plen32[j], T.dabs);
    if (rr < 0) {
        rr = cohen_sutherland(a, b, bx, c, d);
        if (rr < 0) set_error(T.err, CT_DEVERR_LOOP);
    }
    *c = *d = mkp(dnan(), dnan());
    if (rr != 1) return false;
    const dpt* poly = reinterpret_cast<const dpt*>(T.poly + (size_t)j * T.K);
    int len = T.plen ? (int)T.plen[j] : T.K;
    double tol = pmax(CT_MIN_TOLERANCE, CT_TOLERANCE_FACTOR * pmax(bx.xmax - bx.xmin, bx.ymax - bx.ymin));
    if (T.polyf && T.K <= 8)
        return cyrus_beck_f32<8>(a, b, poly, len, tol, T.polyf + (size_t)j * T.S4, (int)T.plen32[j], T.dabs, c, d);
    return cyrus_beck(a, b, poly, len, tol, c, d);
}

// compute_intersection cyrus_beck.py:26-43 with products and quotient on the
// integer pipes
__device__ __forceinline__ double cb_param_sf(dpt a, dpt s, double2 v0, double2 v1, bool* bad) {
    const dpt si = mkp(v0.x - a.x, v0.y - a.y);
    const dpt n = mkp(sf_value(sf_bits(v1.y - v0.y) ^ 0x8000000000000000ull), v1.x - v0.x);
    const double n_si = sf_mul(n.x, si.x, bad) + sf_mul(n.y, si.y, bad);
    const double k = sf_mul(n.x, s.x, bad) + sf_mul(n.y, s.y, bad);
    return sf_div(n_si, k, bad);
}

// The same verdict and points for cells of at most 8 vertices without repeated
// ones, with every decision certain in float32; -1 when one is not.
//
// The decisions, in coordinates relative to the cell's first vertex O (float64
// differences truncated to float: error ed; stored vertex offsets: ev0):
//   * the side of every vertex of the segment's line (Cyrus-Beck's walk): as
//     cb_sign32;
//   * whether an endpoint lies in the cell: not when it is beyond the cell's
//     box by more than the errors and the tolerance, else by the leaf filter;
//   * Cohen-Sutherland's verdict, needed only when Cyrus-Beck hits: accept
//     when the middle X of the clipped part lies inside the box by more than
//     its error, the box's, and 2^-46 of the largest coordinate.  (Each of
//     its clipping steps moves an endpoint along the segment to a box side
//     with a few roundings, at most 2^-48 of the largest coordinate in all,
//     and never past X, so no step sees both endpoints beyond one side.)
// Running Cohen-Sutherland's replay first, and Cyrus-Beck's parts in their
// own branches, kept 16 of 32 lanes busy; here nearly every candidate runs
// the same straight code: sides, then the two parameters and points in
// float64 for those whose line crosses the cell.  37M candidates of 1M short
// segments: 15.8 -> 3.1 ms.  No branch that part
// of a warp takes contains an exit: with exits there the lanes rejoin only at
// the function's end (12 instead of 23 of 32 lanes active, 5.1 ms).
__device__ __forceinline__ int edge_face_fast(const TreeQ& T, dpt a, dpt b, int j, dpt* c, dpt* d) {
    const float u24 = 5.9604644775390625e-08f;
    const int len = T.plen ? (int)T.plen[j] : T.K;
    if (len < 3 || (int)T.plen32[j] != len) return -1;
    const double2* poly = T.poly + (size_t)j * T.K;
    const float2* rel = reinterpret_cast<const float2*>(T.polyf + (size_t)j * T.S4 + 1);
    const double2 O = poly[0];
    const dpt s = vsub(b, a);
    const float2 da = make_float2(cl_float(a.x - O.x), cl_float(a.y - O.y));
    const float2 db = make_float2(cl_float(b.x - O.x), cl_float(b.y - O.y));
    const float2 sf = make_float2(cl_float(s.x), cl_float(s.y));
    const float smax = cl_max2(sf), m = fmaxf(fmaxf(cl_max2(da), cl_max2(db)), smax);
    const float om = fmaxf(fabsf(cl_float(O.x)), fabsf(cl_float(O.y)));
    if (!(m < 1e15f && om < 1e25f) || !(smax > 0.0f)) return -1;
    const float ed = 2.01f * u24 * m + 1e-37f, es = 2.01f * u24 * smax + 1e-37f;
    // box of the cell, and sides of its vertices
    float x0 = 0.0f, x1 = 0.0f, y0 = 0.0f, y1 = 0.0f;
    for (int i = 1; i < len; i++) {
        const float2 r = rel[i - 1];
        x0 = fminf(x0, r.x);
        x1 = fmaxf(x1, r.x);
        y0 = fminf(y0, r.y);
        y1 = fmaxf(y1, r.y);
    }
    const float vmax = fmaxf(fmaxf(-x0, x1), fmaxf(-y0, y1));
    const float ev0 = 2.0f * u24 * vmax + T.dabs, ev = ed + ev0;
    const float Ns = fabsf(sf.x) + fabsf(sf.y) + 2.0f * es;
    const float k1 = 1.03f * (2.0f * es + 5.2f * u24 * Ns);
    const float k0 = 1.03f * (2.0f * ev * (2.0f * es + 4.2f * u24 * Ns) + 2.0f * ev * Ns) + 1e-37f;
    unsigned neg = 0;
    bool sure = true;
    for (int i = 0; i < len; i++) {
        const float2 r = i ? rel[i - 1] : make_float2(0.0f, 0.0f);
        const float ux = r.x - da.x, uy = r.y - da.y;
        const float est = __fmaf_rn(ux, sf.y, -(uy * sf.x));
        sure = sure && fabsf(est) > __fmaf_rn(fabsf(ux) + fabsf(uy), k1, k0);
        neg |= (est < 0.0f ? 1u : 0u) << i;
    }
    if (!sure) return -1;
    // crossing at i: vertices i and i + 1 on different sides
    unsigned cross = (neg ^ ((neg >> 1) | (neg << (len - 1)))) & ((1u << len) - 1u);
    // endpoints in the cell
    const float tolf = fmaxf(1.01e-15f, 1.01e-12f * fmaxf(x1 - x0 + 2.0f * ev0, y1 - y0 + 2.0f * ev0));
    const float g = 1.01f * (ed + ev0 + 3.0f * tolf + 2.0f * u24 * vmax);
    int fa = LF_OUTSIDE, fb = LF_OUTSIDE;
    if (da.x >= x0 - g && da.x <= x1 + g && da.y >= y0 - g && da.y <= y1 + g)
        fa = leaf_filter_joined(da.x, da.y, ed, T.dabs, tolf, rel, len);
    if (db.x >= x0 - g && db.x <= x1 + g && db.y >= y0 - g && db.y <= y1 + g)
        fb = leaf_filter_joined(db.x, db.y, ed, T.dabs, tolf, rel, len);
    if (fa == LF_UNSURE || fb == LF_UNSURE) return -1;
    *c = a;
    *d = b;
    float ta = 0.0f, tb = 1.0f;
    bool valid0 = true, valid1 = true, known = true;
    const bool both = fa == LF_INSIDE && fb == LF_INSIDE;
    if (!both && !cross) return 0;
    if (!both) {
        const int i0 = __ffs(cross) - 1, i1 = __ffs(cross & (cross - 1u)) - 1;
        bool bad = false;
        const double p = cb_param_sf(a, s, poly[i0], poly[i0 + 1 < len ? i0 + 1 : 0], &bad);
        const double q = cb_param_sf(a, s, poly[i1], poly[i1 + 1 < len ? i1 + 1 : 0], &bad);
        // the order of the parameters and their ranges on their bits
        const unsigned long long kp = fkey(p), kq = fkey(q);
        const double t0 = kp < kq ? p : q, t1 = kp < kq ? q : p;
        const unsigned long long k0_ = kp < kq ? kp : kq, k1_ = kp < kq ? kq : kp;
        const unsigned long long zero = 0x8000000000000000ull, one = 0xbff0000000000000ull;  // fkey(0), fkey(1)
        valid0 = k0_ >= zero && k0_ < one;
        valid1 = k1_ > zero && k1_ <= one;
        bool b0 = false, b1 = false;
        const double x = sf_mul(t0, s.x, &b0), y = sf_mul(t0, s.y, &b0);
        const double z = sf_mul(t1, s.x, &b1), w = sf_mul(t1, s.y, &b1);
        known = !bad && kp != kq && !(valid0 && b0) && !(valid1 && b1);
        if (valid0) {
            *c = mkp(a.x + x, a.y + y);
            ta = cl_float(t0);
        }
        if (valid1) {
            *d = mkp(a.x + z, a.y + w);
            tb = cl_float(t1);
        }
    }
    if (!known) return -1;
    if (!(valid0 || valid1)) return 0;
    const float tm = 0.5f * (ta + tb);
    const float2 X = make_float2(__fmaf_rn(tm, sf.x, da.x), __fmaf_rn(tm, sf.y, da.y));
    const float mg = 1.05f * (ed + es + 5.0f * u24 * smax + 2.0f * u24 * cl_max2(X) + 2.0f * ev0 +
                              1.5e-14f * (om + 2.0f * m));
    return X.x > x0 + mg && X.x < x1 - mg && X.y > y0 + mg && X.y < y1 - mg ? 1 : -1;
}

__device__ __noinline__ bool edge_edge_general(dpt a, dpt b, dpt p, dpt q, dpt* c) {
    return lines_intersect(a, b, p, q, &c->x, &c->y);
}

// lines_intersect (geometry_utils.py:318-418) of a -> b and p -> q when its
// decisions are certain in float32: 1 a crossing at c, 0 none, -1 unsure.
// With U = q - p, V = b - a, D = a - p (float64 differences truncated to
// float, 2 u of each) the four left_of tests are the signs of U x D,
// U x (D + V), V x D and V x (U - D) (upstream's rounded products are off by
// 2^-53 of theirs).  If both pairs differ the segments cross properly, so
// upstream's overlap tests hold; it then only asks whether they are parallel
// within its tolerance.  Otherwise it returns false unless p and q both lie
// within the tolerance of a -> b's line.  The crossing itself is computed as
// upstream does, products and quotient on the integer pipes.  The float64
// unit bounded the plain form (60 instructions of 20 cycles per warp): 2.5M
// candidates of 100k cross-sections of a network 272 -> 95 us.
__device__ __forceinline__ int edge_edge_fast(dpt a, dpt b, dpt p, dpt q, dpt* c) {
    const float u24 = 5.9604644775390625e-08f;
    const dpt U = vsub(q, p), V = vsub(b, a), D = vsub(a, p);
    const float2 u = make_float2(cl_float(U.x), cl_float(U.y)), v = make_float2(cl_float(V.x), cl_float(V.y));
    const float2 d = make_float2(cl_float(D.x), cl_float(D.y));
    const float mu = fabsf(u.x) + fabsf(u.y), mv = fabsf(v.x) + fabsf(v.y), md = fabsf(d.x) + fabsf(d.y);
    if (!(mu < 1e15f && mv < 1e15f && md < 1e15f)) return -1;
    const float2 e = make_float2(d.x + v.x, d.y + v.y), g = make_float2(u.x - d.x, u.y - d.y);
    const float c1 = __fmaf_rn(u.x, d.y, -(u.y * d.x)), c2 = __fmaf_rn(u.x, e.y, -(u.y * e.x));
    const float c3 = __fmaf_rn(v.x, d.y, -(v.y * d.x)), c4 = __fmaf_rn(v.x, g.y, -(v.y * g.x));
    const float den = __fmaf_rn(v.x, u.y, -(v.y * u.x));
    const float tu = 12.0f * u24 * mu + 2.4e-38f, tv = 12.0f * u24 * mv + 2.4e-38f, f = 1e-36f;
    // tolerance 1e-12 of U's larger component, at least 1e-15; times |V|
    const float tol = 1.02f * fmaxf(1e-15f, 1e-12f * (fmaxf(fabsf(u.x), fabsf(u.y)) + 2.4e-38f)) * (mv + 2.4e-38f);
    const bool s12 = fabsf(c1) > tu * md + f * mu + f && fabsf(c2) > tu * (md + mv) + f * mu + f;
    const bool s34 = fabsf(c3) > tv * md + tol + f * mv + f && fabsf(c4) > tv * (mu + md) + tol + f * mv + f;
    // the pair known to lie on one side settles a miss, if p or q is clear of
    // the tolerance as well
    const bool clear = fabsf(c3) > tv * md + tol + f * mv + f || fabsf(c4) > tv * (mu + md) + tol + f * mv + f;
    if (clear && s12 && (c1 > 0.0f) == (c2 > 0.0f)) return 0;
    if (s34 && (c3 < 0.0f) == (c4 > 0.0f)) return 0;
    if (!(s12 && s34) || !(fabsf(den) > tv * mu + tol + f * mv + f)) return -1;
    bool bad = false;
    const dpt R = mkp(sf_value(sf_bits(D.x) ^ 0x8000000000000000ull), sf_value(sf_bits(D.y) ^ 0x8000000000000000ull));
    const double denom = sf_mul(V.x, U.y, &bad) - sf_mul(V.y, U.x, &bad);
    const double t = sf_div(sf_mul(R.x, U.y, &bad) - sf_mul(R.y, U.x, &bad), denom, &bad);
    const double x = sf_mul(t, V.x, &bad), y = sf_mul(t, V.y, &bad);
    if (bad) return -1;
    *c = mkp(a.x + x, a.y + y);
    return 1;
}

// The cell test of every candidate (compute_edge_face_intersect
// query.py:309-328 / compute_edge_edge_intersect 292-306).
template <int MODE, typename KeepT>
__global__ void __launch_bounds__(128) k_edge_test(TreeQ T, const double4* __restrict__ segs,
                                                   const int* __restrict__ cseg, const int* __restrict__ cj,
                                                   int64_t nc, KeepT* __restrict__ keep, double4* __restrict__ xy) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nc; t += (int64_t)gridDim.x * blockDim.x) {
        double4 s4 = segs[cseg[t]];
        dpt a = mkp(s4.x, s4.y), b = mkp(s4.z, s4.w);
        int j = cj[t];
        dpt c, d;
        bool hit;
        if (MODE == 0) {
            double2 p0 = T.poly[(size_t)j * 2], p1 = T.poly[(size_t)j * 2 + 1];
            const dpt p = mkp(p0.x, p0.y), q = mkp(p1.x, p1.y);
            c = mkp(dnan(), dnan());
            const int r = edge_edge_fast(a, b, p, q, &c);
            hit = r < 0 ? edge_edge_general(a, b, p, q, &c) : r == 1;
            d = c;
        } else {
            int r = -1;
            if (T.polyf && T.K <= 8) r = edge_face_fast(T, a, b, j, &c, &d);
            hit = r < 0 ? edge_face_general(T, a, b, j, &c, &d) : r == 1;
        }
        keep[t] = hit ? 1 : 0;
        if (MODE == 1 && !hit) c = d = mkp(dnan(), dnan());
        xy[t] = make_double4(c.x, c.y, d.x, d.y);
    }
}

// Diagnostics of the segment test's float32 certificates (tests only): per
// pair, upstream's float64 Cohen-Sutherland verdict (1 accept, 0 reject, -1
// loop cap), the float32 interval verdict (cs_f32: 1, 0, -1 undecided) and
// whether the traversal's line filter surely misses the cell's box (1/0; 0
// when the filter is off).
__global__ void k_cs_certificates(TreeQ T, const double4* __restrict__ segs, const int* __restrict__ cseg,
                                  const int* __restrict__ cj, int64_t nc, int8_t* __restrict__ out) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nc; t += (int64_t)gridDim.x * blockDim.x) {
        double4 s4 = segs[cseg[t]];
        dpt a = mkp(s4.x, s4.y), b = mkp(s4.z, s4.w);
        const int j = cj[t];
        dbox bx = leaf_box(T, j);
        dpt c, d;
        out[3 * t] = (int8_t)cohen_sutherland(a, b, bx, &c, &d);
        out[3 * t + 1] = (int8_t)((T.polyf && T.K <= 8)
                                      ? cs_f32(a, b, bx, T.polyf + (size_t)j * T.S4, (int)T.plen32[j], T.dabs)
                                      : -1);
        const EdgeKeys K = edge_keys(T, a, b);
        const LineF LF = line_filter(T, a, b, vsub(b, a), K.keys);
        int miss = 0;
        if (LF.on) {
            const float4 q = T.bbl32[j];
            miss = line_misses(LF, q.x, q.y, q.z, q.w) ? 1 : 0;
        }
        out[3 * t + 2] = (int8_t)miss;
    }
}

// Hits in candidate order (segment-major, traversal order within a segment),
// and every segment's hit offset and count.
__global__ void k_edge_compact(const int64_t* __restrict__ keep, const int64_t* __restrict__ pos, int64_t nc,
                               const int* __restrict__ cseg, const int* __restrict__ cj,
                               const int64_t* __restrict__ bbi, const double4* __restrict__ xy_c,
                               int64_t* __restrict__ ii, int64_t* __restrict__ jj, double4* __restrict__ xy) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nc; t += (int64_t)gridDim.x * blockDim.x) {
        if (!keep[t]) continue;
        int64_t p = pos[t];
        ii[p] = cseg[t];
        jj[p] = bbi[cj[t]];
        xy[p] = xy_c[t];
    }
}

__global__ void k_edge_seg_counts(const int64_t* __restrict__ coff, const int64_t* __restrict__ ccnt,
                                  const int64_t* __restrict__ keep, const int64_t* __restrict__ pos, int64_t nc,
                                  int64_t n, int64_t* __restrict__ off, int64_t* __restrict__ cnt) {
    const int64_t total = nc > 0 ? pos[nc - 1] + keep[nc - 1] : 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c0 = coff[i], c1 = c0 + ccnt[i];
        int64_t p0 = c0 < nc ? pos[c0] : total, p1 = c1 < nc ? pos[c1] : total;
        off[i] = p0;
        cnt[i] = p1 - p0;
    }
}

// ---------------------------------------------------------------------------
// exclusive scan of int64 counts
// ---------------------------------------------------------------------------
constexpr int SCAN_T = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_T * SCAN_ITEMS;

// Block-wide exclusive scan; every thread receives the block total in *total.
__device__ __forceinline__ int64_t block_exclusive_scan(int64_t v, int64_t* total) {
    __shared__ int64_t warp_sums[SCAN_T / 32];
    __shared__ int64_t block_total;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int64_t t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t s = lane < SCAN_T / 32 ? warp_sums[lane] : 0;
        int64_t y = s;
        for (int o = 1; o < 32; o <<= 1) {
            int64_t t = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += t;
        }
        if (lane < SCAN_T / 32) warp_sums[lane] = y - s;
        if (lane == SCAN_T / 32 - 1) block_total = y;
    }
    __syncthreads();
    int64_t r = x - v + warp_sums[w];
    *total = block_total;
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(const int64_t* __restrict__ in, int64_t n, int64_t* __restrict__ sums) {
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int64_t s = 0;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + (int64_t)k * SCAN_T + threadIdx.x;
        if (i < n) s += in[i];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ int64_t ws[SCAN_T / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int k = 0; k < SCAN_T / 32; k++) t += ws[k];
        sums[blockIdx.x] = t;
    }
}

// single block: exclusive scan of the block sums in place, total at sums[nb]
// (eight sums per thread and step: 45k sums in 22 steps of a barrier chain
// instead of 174, 140 -> 44 us)
__global__ void k_scan_sums(int64_t* sums, int64_t nblocks) {
    constexpr int IPT = 8;
    int64_t carry = 0;
    for (int64_t base = 0; base < nblocks; base += SCAN_T * IPT) {
        const int64_t i = base + (int64_t)threadIdx.x * IPT;
        int64_t v[IPT], s = 0, tot;
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            v[k] = i + k < nblocks ? sums[i + k] : 0;
            s += v[k];
        }
        int64_t ex = block_exclusive_scan(s, &tot) + carry;
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            if (i + k < nblocks) sums[i + k] = ex;
            ex += v[k];
        }
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[nblocks] = carry;
}

__global__ void k_scan_down(const int64_t* __restrict__ in, int64_t n, const int64_t* __restrict__ sums,
                            int64_t* __restrict__ out) {
    int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    int64_t v[SCAN_ITEMS];
    int64_t s = 0;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    int64_t tot;
    int64_t ex = block_exclusive_scan(s, &tot) + sums[blockIdx.x];
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int64_t i = base + k;
        if (i < n) out[i] = ex;
        ex += v[k];
    }
}

// ---------------------------------------------------------------------------
// per-segment stable sort by t (sort_intersections_by_edge
// geometry_utils.py:564-574: np.lexsort((t, ii)), NaN last)
// ---------------------------------------------------------------------------

// sortable key of t: NaN greatest, otherwise the float order
__device__ __forceinline__ unsigned long long tkey(double t) {
    unsigned long long b = (unsigned long long)__double_as_longlong(t);
    if ((b & 0x7fffffffffffffffull) > 0x7ff0000000000000ull) return ~0ull;
    return fkey(t);
}

__global__ void k_tkeys(const double4* __restrict__ segs, const int64_t* __restrict__ ii,
                        const double4* __restrict__ xy, int64_t total, unsigned long long* __restrict__ key,
                        int64_t* __restrict__ idx) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= total) return;
    double4 s = segs[ii[r]];
    double4 c = xy[r];
    double abx = s.z - s.x, aby = s.w - s.y;
    double acx = c.x - s.x, acy = c.y - s.y;
    double t = acx * abx + acy * aby;
    key[r] = tkey(t);
    idx[r] = r;
}

template <typename I>
__device__ __forceinline__ bool kless(unsigned long long ka, I ia, unsigned long long kb, I ib) {
    return ka < kb || (ka == kb && ia < ib);
}

constexpr int SORT_T = 128;
constexpr int SORT_SMEM = 1024;  // 2 x 1024 x (8 + 8) B = 32 KB static shared memory

// One block per segment: stable sort of (key, idx) pairs of the segment by
// bottom-up merging; (key, idx) pairs are unique, so each element's output
// rank is its rank in its own run plus the number of smaller elements in the
// partner run (binary search).  Small segments are sorted in shared memory,
// large ones in global memory (A/B ping-pong); the result lands in `idx_out`.
// Segments of more than WARP_SORT_MAX results (listed by k_segsort_warp).
__global__ void __launch_bounds__(SORT_T) k_segsort(const int64_t* __restrict__ off, const int64_t* __restrict__ cnt,
                                                    const int* __restrict__ list,
                                                    const unsigned long long* __restrict__ nlist,
                                                    unsigned long long* __restrict__ kA, int64_t* __restrict__ iA,
                                                    unsigned long long* __restrict__ kB, int64_t* __restrict__ iB,
                                                    int64_t* __restrict__ idx_out) {
    __shared__ unsigned long long sk[2][SORT_SMEM];
    __shared__ int64_t si[2][SORT_SMEM];
    const int64_t nl = (int64_t)*nlist;
    for (int64_t li = blockIdx.x; li < nl; li += gridDim.x) {
    __syncthreads();
    const int64_t sgi = list[li];
    int64_t c = cnt[sgi], o = off[sgi];
    bool smem = c <= SORT_SMEM;
    unsigned long long* k0 = smem ? sk[0] : kA + o;
    int64_t* i0 = smem ? si[0] : iA + o;
    unsigned long long* k1 = smem ? sk[1] : kB + o;
    int64_t* i1 = smem ? si[1] : iB + o;
    if (smem) {
        for (int64_t t = threadIdx.x; t < c; t += blockDim.x) {
            sk[0][t] = kA[o + t];
            si[0][t] = iA[o + t];
        }
    }
    __syncthreads();
    for (int64_t w = 1; w < c; w <<= 1) {
        for (int64_t t = threadIdx.x; t < c; t += blockDim.x) {
            int64_t run = t / w;
            int64_t r0 = (run ^ 1) * w;  // partner run start
            bool left = (run & 1) == 0;
            int64_t own0 = run * w;
            int64_t pair0 = left ? own0 : r0;
            unsigned long long mk = k0[t];
            int64_t mi = i0[t];
            int64_t plo = r0, phi = min(r0 + w, c);
            if (plo > c) plo = c;
            int64_t lo = plo, hi = phi;  // count partner elements smaller than (mk, mi)
            while (lo < hi) {
                int64_t mid = (lo + hi) >> 1;
                if (kless(k0[mid], i0[mid], mk, mi)) lo = mid + 1;
                else hi = mid;
            }
            int64_t dst = pair0 + (t - own0) + (lo - plo);
            k1[dst] = mk;
            i1[dst] = mi;
        }
        __syncthreads();
        unsigned long long* tk = k0;
        k0 = k1;
        k1 = tk;
        int64_t* ti = i0;
        i0 = i1;
        i1 = ti;
    }
    for (int64_t t = threadIdx.x; t < c; t += blockDim.x) idx_out[o + t] = i0[t];
    }
}

// One warp per segment: bitonic sort of up to 32 x E (key, idx) pairs in
// registers (element r * 32 + lane in register r of the lane; pads sort
// last).  (key, idx) pairs are unique, so the order is the stable sort's.
constexpr int WARP_SORT_MAX = 128;

template <int E, typename I>
__device__ __forceinline__ void warp_bitonic(unsigned long long (&k)[E], I (&x)[E], int lane) {
    const unsigned FULL = 0xffffffffu;
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
        for (int j = size >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int rj = j >> 5;
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const int rp = r ^ rj;
                    if (rp > r) {
                        const bool asc = ((r * 32 + lane) & size) == 0;
                        const bool less_rp = kless(k[rp], x[rp], k[r], x[r]);
                        if (asc ? less_rp : !less_rp) {
                            const unsigned long long tk = k[r];
                            k[r] = k[rp];
                            k[rp] = tk;
                            const I tx = x[r];
                            x[r] = x[rp];
                            x[rp] = tx;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const unsigned long long pk = __shfl_xor_sync(FULL, k[r], j);
                    const I px = __shfl_xor_sync(FULL, x[r], j);
                    const bool asc = ((r * 32 + lane) & size) == 0;
                    const bool lower = (lane & j) == 0;
                    const bool pless = kless(pk, px, k[r], x[r]);
                    if ((lower == asc) ? pless : !pless) {
                        k[r] = pk;
                        x[r] = px;
                    }
                }
            }
        }
    }
}

template <int E>
__device__ __forceinline__ void warp_sort_segment(const unsigned long long* __restrict__ kA,
                                                  const int64_t* __restrict__ iA, int64_t o, int64_t c, int lane,
                                                  int64_t* __restrict__ idx_out) {
    unsigned long long k[E];
    int64_t x[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int64_t e = r * 32 + lane;
        k[r] = e < c ? kA[o + e] : ~0ull;
        x[r] = e < c ? iA[o + e] : INT64_MAX;
    }
    warp_bitonic(k, x, lane);
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int64_t e = r * 32 + lane;
        if (e < c) idx_out[o + e] = x[r];
    }
}

// Segments of up to WARP_SORT_MAX results sorted by a warp each; longer ones
// are listed for k_segsort.
__global__ void __launch_bounds__(256) k_segsort_warp(const int64_t* __restrict__ off,
                                                      const int64_t* __restrict__ cnt, int64_t nseg,
                                                      const unsigned long long* __restrict__ kA,
                                                      const int64_t* __restrict__ iA, int64_t* __restrict__ idx_out,
                                                      int* __restrict__ list, unsigned long long* __restrict__ nlist) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t sgi = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); sgi < nseg; sgi += warps) {
        const int64_t c = cnt[sgi], o = off[sgi];
        if (c <= 0) continue;
        if (c == 1) {
            if (lane == 0) idx_out[o] = iA[o];
        } else if (c <= 32) {
            warp_sort_segment<1>(kA, iA, o, c, lane, idx_out);
        } else if (c <= 64) {
            warp_sort_segment<2>(kA, iA, o, c, lane, idx_out);
        } else if (c <= WARP_SORT_MAX) {
            warp_sort_segment<4>(kA, iA, o, c, lane, idx_out);
        } else if (lane == 0) {
            list[atomicAdd(nlist, 1ull)] = (int)sgi;
        }
    }
}

__global__ void k_gather_results(const int64_t* __restrict__ perm, int64_t total, const int64_t* __restrict__ jj_in,
                                 const double4* __restrict__ xy_in, int64_t* __restrict__ jj_out,
                                 double4* __restrict__ xy_out) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= total) return;
    int64_t s = perm[r];
    jj_out[r] = jj_in[s];
    xy_out[r] = xy_in[s];
}

// ---------------------------------------------------------------------------
// From the tested candidates to the results: every segment's hits counted,
// and, with the offsets known, each segment's hits sorted by t and written in
// place at once (segments of up to 128 hits by a warp, longer ones by a
// block).  The candidates may be grouped by segments in another order than
// the results (`order`: result segment of candidate segment s).  Against
// compacting the hits, then keys, sort and gather as passes over all results
// (31M hits of 1M segments: 2.6 ms) this reads the hits once and writes the
// results once (1.3 ms).
// ---------------------------------------------------------------------------
// Hits of every segment: eight lanes a segment, the warp together for those
// of more than 256 candidates (a warp per segment and 32 candidates at a time:
// 1M segments 177 -> 80 us, 1000 sections 48 -> 35).
__global__ void __launch_bounds__(256) k_hit_counts(const uint8_t* __restrict__ keep,
                                                    const int64_t* __restrict__ coff,
                                                    const int64_t* __restrict__ ccnt, const int* __restrict__ order,
                                                    int64_t n, int64_t* __restrict__ counts,
                                                    unsigned long long* __restrict__ longest) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const int64_t groups = ((int64_t)gridDim.x * blockDim.x) >> 3;
    int64_t most = 0;
    // (the same number of rounds in all lanes of a warp)
    for (int64_t s0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4; s0 < n; s0 += groups) {
        const int64_t s = s0 + (lane >> 3);
        int64_t c0 = 0, m = 0, c = 0;
        if (s < n) {
            c0 = coff[s];
            m = ccnt[s];
        }
        if (m <= 256)
            for (int64_t k = sub; k < m; k += 8) c += keep[c0 + k] != 0;
        for (unsigned w = __ballot_sync(FULL, m > 256 && sub == 0); w; w &= w - 1u) {
            const int src = __ffs(w) - 1;
            const int64_t wc0 = __shfl_sync(FULL, c0, src), wm = __shfl_sync(FULL, m, src);
            int64_t x = 0;
            for (int64_t k = lane; k < wm; k += 128) {
                int h = keep[wc0 + k] != 0;
#pragma unroll
                for (int u = 1; u < 4; u++) h += k + 32 * u < wm && keep[wc0 + k + 32 * u] != 0;
                x += h;
            }
            x += __shfl_xor_sync(FULL, x, 16);
            x += __shfl_xor_sync(FULL, x, 8);
            if ((lane >> 3) == (src >> 3)) c = x;  // summed over its eight lanes below
        }
        for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o, 8);
        most = max(most, c);
        if (sub == 0 && s < n) counts[order ? (int64_t)order[s] : s] = c;
    }
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(FULL, most, o));
    if (lane == 0 && most > 0) atomicMax(longest, (unsigned long long)most);
}

struct HitSort {
    const double4* segs;   // in candidate order
    const int* order;
    const uint8_t* keep;
    const int* cj;
    const int64_t* bbi;
    const double4* xy_c;
    const int64_t *coff, *ccnt, *counts, *offsets;
    int64_t *ii, *jj;
    double4* xy;
};

// sort key of candidate r of a segment from a with direction ab
__device__ __forceinline__ unsigned long long hit_key(const HitSort& H, int64_t r, double4 s) {
    const double2 c = *reinterpret_cast<const double2*>(H.xy_c + r);
    const double abx = s.z - s.x, aby = s.w - s.y;
    const double acx = c.x - s.x, acy = c.y - s.y;
    return tkey(acx * abx + acy * aby);
}

__device__ __forceinline__ void hit_write(const HitSort& H, int64_t out, int64_t seg, int64_t r) {
    H.ii[out] = seg;
    H.jj[out] = H.bbi[H.cj[r]];
    H.xy[out] = H.xy_c[r];
}

template <int E>
__device__ __forceinline__ void hit_sort_warp(const HitSort& H, const unsigned long long* sk, const unsigned* si,
                                              int c, int64_t o, int64_t i, int64_t c0, int lane) {
    unsigned long long k[E];
    unsigned x[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int e = r * 32 + lane;
        k[r] = e < c ? sk[e] : ~0ull;
        x[r] = e < c ? si[e] : ~0u;
    }
    warp_bitonic(k, x, lane);
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int e = r * 32 + lane;
        if (e < c) hit_write(H, o + e, i, c0 + x[r]);
    }
}

__global__ void __launch_bounds__(256) k_finish_warp(HitSort H, int64_t n, int* __restrict__ list,
                                                     unsigned long long* __restrict__ nlist) {
    __shared__ unsigned long long keys[8][WARP_SORT_MAX];
    __shared__ unsigned idx[8][WARP_SORT_MAX];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long* sk = keys[w];
    unsigned* si = idx[w];
    const int64_t warps = (int64_t)gridDim.x * 8;
    for (int64_t s = (int64_t)blockIdx.x * 8 + w; s < n; s += warps) {
        const int64_t i = H.order ? (int64_t)H.order[s] : s;
        const int64_t c = H.counts[i];
        if (c == 0) continue;
        if (c > WARP_SORT_MAX) {
            if (lane == 0) list[atomicAdd(nlist, 1ull)] = (int)s;
            continue;
        }
        const int64_t c0 = H.coff[s], m = H.ccnt[s], o = H.offsets[i];
        const double4 sg = H.segs[s];
        int have = 0;
        for (int64_t k = 0; k < m; k += 32) {
            const bool hit = k + lane < m && H.keep[c0 + k + lane];
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                const int p = have + __popc(b & ((1u << lane) - 1u));
                sk[p] = hit_key(H, c0 + k + lane, sg);
                si[p] = (unsigned)(k + lane);
            }
            have += __popc(b);
        }
        __syncwarp();
        if (c <= 32) hit_sort_warp<1>(H, sk, si, (int)c, o, i, c0, lane);
        else if (c <= 64) hit_sort_warp<2>(H, sk, si, (int)c, o, i, c0, lane);
        else hit_sort_warp<4>(H, sk, si, (int)c, o, i, c0, lane);
        __syncwarp();
    }
}

constexpr int FIN_T = 256;
constexpr int FIN_SMEM = 8 * WARP_SORT_MAX;  // hits a block sorts in shared memory

// c (<= FIN_SMEM) pairs in (k[0], x[0]): sorted by warps in runs of 128, then
// merged by ranks; returns the buffer (0 / 1) that holds the result.
__device__ __forceinline__ int block_sort(unsigned long long (*k)[FIN_SMEM], unsigned (*x)[FIN_SMEM], int c) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int b0 = w * WARP_SORT_MAX;
    if (b0 < c) {
        unsigned long long kr[4];
        unsigned xr[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int e = b0 + r * 32 + lane;
            kr[r] = e < c ? k[0][e] : ~0ull;
            xr[r] = e < c ? x[0][e] : ~0u;
        }
        warp_bitonic(kr, xr, lane);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int e = b0 + r * 32 + lane;
            if (e < c) {
                k[0][e] = kr[r];
                x[0][e] = xr[r];
            }
        }
    }
    __syncthreads();
    int cur = 0;
    for (int wd = WARP_SORT_MAX; wd < c; wd <<= 1) {
        for (int t = threadIdx.x; t < c; t += FIN_T) {
            const int run = t / wd, own = run * wd, plo = min((run ^ 1) * wd, c), phi = min(plo + wd, c);
            const unsigned long long mk = k[cur][t];
            const unsigned mx = x[cur][t];
            int lo = plo, hi = phi;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (kless(k[cur][mid], x[cur][mid], mk, mx)) lo = mid + 1;
                else hi = mid;
            }
            const int dst = (run & ~1) * wd + (t - own) + (lo - plo);
            k[cur ^ 1][dst] = mk;
            x[cur ^ 1][dst] = mx;
        }
        __syncthreads();
        cur ^= 1;
    }
    return cur;
}

// Longer segments (listed), one block each: hits collected in any order (the
// (key, candidate) pairs are unique), sorted in shared memory up to FIN_SMEM,
// else in sorted runs of that many merged by ranks in global memory (gk / gx:
// two buffers of `total` pairs).
__global__ void __launch_bounds__(FIN_T) k_finish_block(HitSort H, const int* __restrict__ list,
                                                        const unsigned long long* __restrict__ nlist, int64_t total,
                                                        unsigned long long* __restrict__ gk,
                                                        unsigned* __restrict__ gx) {
    __shared__ unsigned long long k[2][FIN_SMEM];
    __shared__ unsigned x[2][FIN_SMEM];
    __shared__ unsigned long long fill;
    const int lane = threadIdx.x & 31;
    const int64_t nl = (int64_t)*nlist;
    for (int64_t li = blockIdx.x; li < nl; li += gridDim.x) {
        const int64_t s = list[li], i = H.order ? (int64_t)H.order[s] : s;
        const int64_t c = H.counts[i], c0 = H.coff[s], m = H.ccnt[s], o = H.offsets[i];
        const bool small = c <= FIN_SMEM;
        const double4 sg = H.segs[s];
        __syncthreads();
        if (threadIdx.x == 0) fill = 0;
        __syncthreads();
        for (int64_t t0 = 0; t0 < m; t0 += FIN_T) {
            const int64_t t = t0 + threadIdx.x;
            const bool hit = t < m && H.keep[c0 + t];
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            unsigned long long p = 0;
            if (lane == 0 && b) p = atomicAdd(&fill, (unsigned long long)__popc(b));
            p = __shfl_sync(0xffffffffu, p, 0) + __popc(b & ((1u << lane) - 1u));
            if (hit) {
                const unsigned long long key = hit_key(H, c0 + t, sg);
                if (small) {
                    k[0][p] = key;
                    x[0][p] = (unsigned)t;
                } else {
                    gk[o + p] = key;
                    gx[o + p] = (unsigned)t;
                }
            }
        }
        __syncthreads();
        if (small) {
            const int cur = block_sort(k, x, (int)c);
            for (int t = threadIdx.x; t < c; t += FIN_T) hit_write(H, o + t, i, c0 + x[cur][t]);
            continue;
        }
        for (int64_t r0 = 0; r0 < c; r0 += FIN_SMEM) {
            const int rc = (int)min((int64_t)FIN_SMEM, c - r0);
            for (int t = threadIdx.x; t < rc; t += FIN_T) {
                k[0][t] = gk[o + r0 + t];
                x[0][t] = gx[o + r0 + t];
            }
            __syncthreads();
            const int cur = block_sort(k, x, rc);
            for (int t = threadIdx.x; t < rc; t += FIN_T) {
                gk[o + r0 + t] = k[cur][t];
                gx[o + r0 + t] = x[cur][t];
            }
            __syncthreads();
        }
        unsigned long long *ka = gk + o, *kb = gk + total + o;
        unsigned *xa = gx + o, *xb = gx + total + o;
        for (int64_t wd = FIN_SMEM; wd < c; wd <<= 1) {
            for (int64_t t = threadIdx.x; t < c; t += FIN_T) {
                const int64_t run = t / wd, own = run * wd, plo = min((run ^ 1) * wd, c), phi = min(plo + wd, c);
                const unsigned long long mk = ka[t];
                const unsigned mx = xa[t];
                int64_t lo = plo, hi = phi;
                while (lo < hi) {
                    const int64_t mid = (lo + hi) >> 1;
                    if (kless(ka[mid], xa[mid], mk, mx)) lo = mid + 1;
                    else hi = mid;
                }
                const int64_t dst = (run & ~(int64_t)1) * wd + (t - own) + (lo - plo);
                kb[dst] = mk;
                xb[dst] = mx;
            }
            __syncthreads();
            unsigned long long* tk = ka;
            ka = kb;
            kb = tk;
            unsigned* tx = xa;
            xa = xb;
            xb = tx;
        }
        for (int64_t t = threadIdx.x; t < c; t += FIN_T) hit_write(H, o + t, i, c0 + xa[t]);
    }
}

// ---------------------------------------------------------------------------
// per-pair kernels
// ---------------------------------------------------------------------------

__device__ __forceinline__ int load_poly(const double* __restrict__ v, const int64_t* __restrict__ faces, int K,
                                         int64_t f, dpt* out) {
    return gather_polygon(v, faces + f * K, K, out);
}

// Float32 filter of polygons_intersect (separating_axis.py:17-75).
//
// For the axis of edge p -> q the upstream test compares float64
// projections v . n with n = (p.y - q.y, q.x - p.x) (both float64).  Each
// projection is within D = 2u(1+u) |v|max (|n.x| + |n.y|) (u = 2^-53) of the
// exact projection on that same n, so a comparison of a maximum with a
// minimum whose exact values differ by more than 2D has the float64 outcome
// of the exact one.  Here the projections are evaluated in float32 in a frame
// at the first vertex of a (each coordinate split exactly into float hi + lo,
// as the leaf filter does), within E of the exact ones (error terms of the
// local coordinates, of n and of the float32 dot products).  An axis whose
// two comparisons clear 2(D + E) is decided: separating or not.  Any
// decided separating axis makes the answer false (upstream stops at the
// first separating axis, but the answer is the same boolean); all axes
// decided and none separating makes it true; otherwise the float64 test runs.
// Returns 0 / 1 for a decided answer, 2 when undecided.
template <int KA, int KB>
__device__ __forceinline__ int sat_filter(const dpt* a, int la, const dpt* b, int lb) {
    constexpr int KM = KA + KB;
    const float u32 = 5.9604644775390625e-08f;  // 2^-24
    float dx[KM], dy[KM];
    float vmax = 0.0f, dmax = 0.0f, ed = 0.0f;
    PtSplit O = split_point(a[0].x, a[0].y);
    bool finite = true;
#pragma unroll
    for (int j = 0; j < KM; j++) {
        if (j < KA ? j < la : (j - KA) < lb) {
            dpt v = j < KA ? a[j] : b[j - KA];
            finite = finite && g_finite(v.x) && g_finite(v.y);
            PtSplit P = split_point(v.x, v.y);
            float4 o = make_float4(O.xh, O.xl, O.yh, O.yl);
            float e;
            local_delta(P, o, &dx[j], &dy[j], &e);
            ed = fmaxf(ed, e);
            dmax = fmaxf(dmax, fmaxf(fabsf(dx[j]), fabsf(dy[j])));
            vmax = fmaxf(vmax, fmaxf(fabsf(P.xh), fabsf(P.yh)));
        } else {
            dx[j] = dy[j] = 0.0f;
        }
    }
    if (!finite) return 2;
    vmax *= 1.0000003f;
    dmax += ed;
    bool undecided = false;
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const int base = side ? KA : 0, len = side ? lb : la;
        const int KS = side ? KB : KA;
#pragma unroll
        for (int i = 0; i < KS; i++) {
            if (i >= len) break;
            const int ip = (i == 0) ? base + len - 1 : base + i - 1, iq = base + i;
            dpt p = side ? b[ip - KA] : a[ip], q = side ? b[iq - KA] : a[iq];
            if (g_zero_edge(p, q)) continue;  // norm == (0, 0): upstream skips the axis
            float nx = dy[ip] - dy[iq], ny = dx[iq] - dx[ip];
            float nm = fabsf(nx) + fabsf(ny);
            float en = 2.0f * ed + 2.0f * u32 * fmaxf(fabsf(nx), fabsf(ny));
            float mina = 3.0e38f, maxa = -3.0e38f, minb = 3.0e38f, maxb = -3.0e38f;
#pragma unroll
            for (int j = 0; j < KM; j++) {
                if (j < KA ? j < la : (j - KA) < lb) {
                    float pr = dx[j] * nx + dy[j] * ny;
                    if (j < KA) {
                        mina = fminf(mina, pr);
                        maxa = fmaxf(maxa, pr);
                    } else {
                        minb = fminf(minb, pr);
                        maxb = fmaxf(maxb, pr);
                    }
                }
            }
            float E = ed * nm + 2.0f * dmax * en + 4.0f * u32 * dmax * (nm + 2.0f * en);
            float D = 2.2204461e-16f * 1.0001f * vmax * (nm + 2.0f * en);
            float thr = 2.03f * (E + D) + 1e-37f;
            float d1 = maxa - minb, d2 = maxb - mina;
            bool sure1 = fabsf(d1) * (1.0f - 4.0f * u32) > thr, sure2 = fabsf(d2) * (1.0f - 4.0f * u32) > thr;
            // separating for sure: one comparison surely false
            if ((sure1 && d1 < 0.0f) || (sure2 && d2 < 0.0f)) return 0;
            if (!(sure1 && sure2)) undecided = true;
        }
    }
    return undecided ? 2 : 1;
}

// polygons_intersect separating_axis.py:58-75
__global__ void k_sat(const double* __restrict__ va, const int64_t* __restrict__ fa, int Ka,
                      const double* __restrict__ vb, const int64_t* __restrict__ fb, int Kb,
                      const int64_t* __restrict__ ia, const int64_t* __restrict__ ib, int64_t n,
                      uint8_t* __restrict__ out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dpt a[CT_MAX_N_VERTEX], b[CT_MAX_N_VERTEX];
    int la = load_poly(va, fa, Ka, ia[i], a);
    int lb = load_poly(vb, fb, Kb, ib[i], b);
    int r = 2;
    if (Ka <= 4 && Kb <= 4) r = sat_filter<4, 4>(a, la, b, lb);
    else if (Ka <= 8 && Kb <= 8) r = sat_filter<8, 8>(a, la, b, lb);
    if (r == 2) r = (int)(separating_axes(a, la, b, lb) && separating_axes(b, lb, a, la));
    out[i] = (uint8_t)r;
}

// One pair's area by the general clip (polygons in local memory).
__device__ __noinline__ double clip_pair_general(const double4* __restrict__ boxes, const double* __restrict__ va,
                                                 const int64_t* __restrict__ fa, int Ka, int64_t ia,
                                                 const double* __restrict__ vb, const int64_t* __restrict__ fb,
                                                 int Kb, int64_t ib, unsigned int* __restrict__ err) {
    dpt a[CT_MAX_N_VERTEX], b[CT_MAX_N_VERTEX];
    dpt A[CT_CLIP_MAX], B[CT_CLIP_MAX];
    int la = 4;
    if (boxes) {
        const double4 q = boxes[ia];
        a[0] = mkp(q.x, q.z);
        a[1] = mkp(q.y, q.z);
        a[2] = mkp(q.y, q.w);
        a[3] = mkp(q.x, q.w);
    } else {
        la = load_poly(va, fa, Ka, ia, a);
    }
    int lb = load_poly(vb, fb, Kb, ib, b);
    bool of = false;
    const double area = clip_area_conv(a, la, b, lb, A, B, &of);
    if (of) set_error(err, CT_DEVERR_CLIP);
    return area;
}

// area_of_intersection sutherland_hodgman.py:151-168 (subject: face of a,
// clipper: face of b) and, with `boxes`, box_area_of_intersection 171-187
// (subject: the box).
// `order`: NULL, or a permutation of the pairs (processing order only:
// pairs of equal polygon lengths side by side, so a warp's lanes run the
// same number of clip edges; results stay at their pair's index).
__global__ void k_clip_area(const double4* __restrict__ boxes, const double* __restrict__ va,
                            const int64_t* __restrict__ fa, int Ka, const double* __restrict__ vb,
                            const int64_t* __restrict__ fb, int Kb, const int64_t* __restrict__ ia,
                            const int64_t* __restrict__ ib, int64_t n, const int* __restrict__ order,
                            double* __restrict__ out, unsigned int* __restrict__ err) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int64_t i = order ? (int64_t)order[t] : t;
    out[i] = clip_pair_general(boxes, va, fa, Ka, ia[i], vb, fb, Kb, ib[i], err);
}

// The same for polygons of at most CL_SLOTS (subject) and KT (clipper)
// vertices: ct_clip.cuh, the general clip where it does not apply.
template <int KT, bool BOX>
__global__ void __launch_bounds__(CL_THREADS) k_clip_area_small(
    const double4* __restrict__ boxes, const double2* __restrict__ va, const int64_t* __restrict__ fa, int Ka,
    const double2* __restrict__ vb, const int64_t* __restrict__ fb, int Kb, const int64_t* __restrict__ ia,
    const int64_t* __restrict__ ib, int64_t n, const int* __restrict__ order, double* __restrict__ out,
    unsigned int* __restrict__ err) {
    __shared__ ClipCols<KT> S;
    const int tid = threadIdx.x;
    const int64_t t = (int64_t)blockIdx.x * CL_THREADS + tid;
    if (t >= n) return;
    const int64_t i = order ? (int64_t)order[t] : t;
    const int64_t ja = ia[i], jb = ib[i];
    int64_t kb[KT];
    int lb = Kb;
#pragma unroll
    for (int k = 0; k < KT; k++) kb[k] = k < Kb ? fb[jb * Kb + k] : CT_FILL_VALUE;
#pragma unroll
    for (int k = KT - 1; k >= 3; k--)
        if (k < Kb && kb[k] == CT_FILL_VALUE) lb = k;
    int la = 4;
    if (BOX) {
        const double4 q = boxes[ja];
        S.v[0][tid] = make_double2(q.x, q.z);
        S.v[1][tid] = make_double2(q.y, q.z);
        S.v[2][tid] = make_double2(q.y, q.w);
        S.v[3][tid] = make_double2(q.x, q.w);
    } else {
        const int64_t* face = fa + ja * Ka;
        la = polygon_length(face, Ka);
        for (int k = 0; k < la; k++) S.v[k][tid] = va[face[k]];
    }
#pragma unroll
    for (int k = 0; k < KT; k++)
        if (k < lb) S.c[k][tid] = vb[kb[k]];
    double area;
    if (!clip_area_small<KT, BOX>(S, tid, la, lb, &area))
        area = clip_pair_general(boxes, (const double*)va, fa, Ka, ja, (const double*)vb, fb, Kb, jb, err);
    out[i] = area;
}

__global__ void k_face_lengths(const int64_t* __restrict__ faces, int K, int64_t n, uint8_t* __restrict__ length) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        length[i] = (uint8_t)polygon_length(faces + i * K, K);
}

// The classes of (box, face) pairs from the faces' lengths, a byte each: for
// batches with many pairs per face, whose rows are read from DRAM for every
// pair otherwise (91M pairs on 5M faces 1.65 -> 0.42 ms).
__global__ void __launch_bounds__(256) k_box_pair_keys(const uint8_t* __restrict__ length,
                                                       const int64_t* __restrict__ ib,
                                                       const uint8_t* __restrict__ inside, int64_t n,
                                                       unsigned* __restrict__ key) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
        int64_t b[4];
        int l[4];
#pragma unroll
        for (int u = 0; u < 4; u++) b[u] = ib[min(i0 + u * step, n - 1)];
#pragma unroll
        for (int u = 0; u < 4; u++) l[u] = 2 * min((int)length[b[u]] - 3, 7) + (inside && inside[min(i0 + u * step, n - 1)] ? 1 : 0);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i0 + u * step < n) key[i0 + u * step] = (unsigned)l[u];
    }
}

// 6-bit class of a pair: the polygon lengths (3 .. 10) of its two faces
// (fa NULL: boxes, length 4)
__global__ void k_pair_keys(const int64_t* __restrict__ fa, int Ka, const int64_t* __restrict__ ia,
                            const int64_t* __restrict__ fb, int Kb, const int64_t* __restrict__ ib, int64_t n,
                            unsigned* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int la = fa ? polygon_length(fa + ia[i] * Ka, Ka) : 4;
        int lb = polygon_length(fb + ib[i] * Kb, Kb);
        key[i] = (unsigned)(min(la - 3, 7) * 8 + min(lb - 3, 7));
    }
}

// Compaction of pairs: keep those of area > 0 (celltree.py:183, 268) or of a
// set flag, in order.  Bound by memory: a tile's kept pairs are counted, the
// tiles' counts summed, and the tiles written from the areas read again (a
// keep array, its scan and the writes by both moved 8 GB for 91M pairs, 1.8 ms;
// now 5 GB, 0.85 ms).
constexpr int KEEP_T = 256, KEEP_ROUNDS = 8, KEEP_TILE = KEEP_T * KEEP_ROUNDS;
constexpr int KEEP_DIRECT = 1024;  // tiles whose counts a block sums itself, without a scan before

__device__ __forceinline__ bool kept(const double* __restrict__ area, const uint8_t* __restrict__ flag, int64_t i,
                                     int64_t n) {
    return i < n && (area ? area[i] > 0 : flag[i] != 0);
}

__global__ void __launch_bounds__(KEEP_T) k_keep_count(const double* __restrict__ area,
                                                       const uint8_t* __restrict__ flag, int64_t n,
                                                       int64_t* __restrict__ counts) {
    const int64_t base = (int64_t)blockIdx.x * KEEP_TILE + threadIdx.x;
    bool k[KEEP_ROUNDS];
#pragma unroll
    for (int r = 0; r < KEEP_ROUNDS; r++) k[r] = kept(area, flag, base + r * KEEP_T, n);
    int c = 0;
#pragma unroll
    for (int r = 0; r < KEEP_ROUNDS; r++) c += __syncthreads_count(k[r]);
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

// `sums`: the tiles' counts, or with `scanned` the kept pairs before each.
__global__ void __launch_bounds__(KEEP_T) k_compact(const double* __restrict__ area, const uint8_t* __restrict__ flag,
                                                    int64_t n, const int64_t* __restrict__ sums, bool scanned,
                                                    const int64_t* __restrict__ ii, const int64_t* __restrict__ jj,
                                                    int64_t* __restrict__ ii_out, int64_t* __restrict__ jj_out,
                                                    double* __restrict__ vals_out, int64_t* __restrict__ total) {
    __shared__ int wsum[KEEP_T / 32];
    __shared__ int64_t part[KEEP_T / 32];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t b = blockIdx.x, base = b * KEEP_TILE + w * (32 * KEEP_ROUNDS) + lane;  // a warp's pairs in a row
    double v[KEEP_ROUNDS];
    unsigned m[KEEP_ROUNDS];
    int64_t i[KEEP_ROUNDS], j[KEEP_ROUNDS];
    int mine = 0;
#pragma unroll
    for (int r = 0; r < KEEP_ROUNDS; r++) {
        const int64_t p = base + r * 32;
        v[r] = area && p < n ? area[p] : 0.0;
        m[r] = __ballot_sync(FULL, area ? p < n && v[r] > 0 : kept(area, flag, p, n));
        mine += __popc(m[r]);
    }
#pragma unroll
    for (int r = 0; r < KEEP_ROUNDS; r++) {
        const bool k = (m[r] >> lane) & 1u;
        i[r] = k ? ii[base + r * 32] : 0;
        j[r] = k ? jj[base + r * 32] : 0;
    }
    int64_t before = 0;
    if (!scanned) {
        for (int64_t k = threadIdx.x; k < b; k += KEEP_T) before += sums[k];
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(FULL, before, o);
    }
    if (lane == 0) {
        wsum[w] = mine;
        part[w] = before;
    }
    __syncthreads();
    int64_t at = scanned ? sums[b] : 0;
    for (int k = 0; k < KEEP_T / 32; k++) {
        if (!scanned) at += part[k];
        if (k < w) at += wsum[k];
    }
    if (total && b == gridDim.x - 1 && w == KEEP_T / 32 - 1 && lane == 0) *total = at + mine;
#pragma unroll
    for (int r = 0; r < KEEP_ROUNDS; r++) {
        if ((m[r] >> lane) & 1u) {
            const int64_t p = at + __popc(m[r] & ((1u << lane) - 1u));
            ii_out[p] = i[r];
            jj_out[p] = j[r];
            if (vals_out) vals_out[p] = v[r];
        }
        at += __popc(m[r]);
    }
}

// ---------------------------------------------------------------------------
// barycentric weights (barycentric_triangle.py:46-64,
// barycentric_wachspress.py:88-107)
// ---------------------------------------------------------------------------
__device__ __noinline__ void bary_general(double2 pp, int64_t f, const double* __restrict__ v,
                                          const int64_t* __restrict__ faces, int K, double tol,
                                          double* __restrict__ w) {
    const dpt p = mkp(pp.x, pp.y);
    const int64_t* face = faces + f * K;
    if (K > 3) {
        dpt poly[CT_MAX_N_VERTEX];
        double ww[CT_MAX_N_VERTEX];
        int len = gather_polygon(v, face, K, poly);
        for (int k = 0; k < K; k++) ww[k] = 0.0;
        wachspress(poly, len, p, ww, K, tol);
        for (int k = 0; k < K; k++) w[k] = ww[k];
    } else {
        double ww[3];
        tri_weights(mkp(v[2 * face[0]], v[2 * face[0] + 1]), mkp(v[2 * face[1]], v[2 * face[1] + 1]),
                    mkp(v[2 * face[2]], v[2 * face[2] + 1]), p, ww);
        w[0] = ww[0];
        w[1] = ww[1];
        w[2] = ww[2];
    }
}

__global__ void k_barycentric(const double2* __restrict__ pts, const int64_t* __restrict__ fidx, int64_t n,
                              const double* __restrict__ v, const int64_t* __restrict__ faces, int K, int KW,
                              double tol, double* __restrict__ out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* w = out + i * KW;
    const int64_t f = fidx[i];
    if (f == -1) {
        for (int k = 0; k < KW; k++) w[k] = 0.0;
        return;
    }
    bary_general(pts[i], f, v, faces, K, tol, w);
}

// |u x v| with the products on the integer pipes
__device__ __forceinline__ double sf_abs_cross(dpt u, dpt v, bool* bad) {
    return fabs(sf_mul(u.x, v.y, bad) - sf_mul(u.y, v.x, bad));
}
// 2 x: the exponent raised by one
__device__ __forceinline__ double sf_twice(double x, bool* bad) {
    const uint64_t b = sf_bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
    *bad = *bad || (e - 1u >= 2045u && !sf_zero(x));
    return sf_zero(x) ? x : sf_value(b + 0x10000000000000ull);
}

// Weights in faces of up to KT (> 3) vertices: the values and the order of
// wachspress.  The float64 unit bounds these weights (160 instructions of 20
// cycles per warp and quad, seven of them per division); here it keeps the
// additions, while products and quotients run on the integer pipes and the
// on-edge test |A| < tol |U| is decided in float32 by a margin of 1 % (A and
// U truncated to float, at most 2^-23 or 1.2e-38 smaller; |Ux| + |Uy| >= |U|).
// Points the margin does not clear, and values sf_mul / sf_div flag, take the
// general form.  1M points in quads: 327 -> 125 us.
template <int KT>
__global__ void __launch_bounds__(128) k_barycentric_small(const double2* __restrict__ pts,
                                                           const int64_t* __restrict__ fidx, int64_t n,
                                                           const double2* __restrict__ v,
                                                           const int64_t* __restrict__ faces, int K, double tol,
                                                           float tolf, double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* w = out + i * K;
    const int64_t f = fidx[i];
    if (f == -1) {
        for (int k = 0; k < K; k++) w[k] = 0.0;
        return;
    }
    const double2 pp = pts[i];
    const dpt p = mkp(pp.x, pp.y);
    int64_t idx[KT];
    int len = K;
#pragma unroll
    for (int k = 0; k < KT; k++) idx[k] = k < K ? faces[f * K + k] : CT_FILL_VALUE;
    int64_t last = idx[2];
#pragma unroll
    for (int k = KT - 1; k >= 3; k--)
        if (k < K && idx[k] == CT_FILL_VALUE) len = k;
#pragma unroll
    for (int k = 3; k < KT; k++)
        if (k == len - 1) last = idx[k];
    if (last == idx[0]) {  // a closed ring: an edge of no length, never clear
        bary_general(pp, f, (const double*)v, faces, K, tol, w);
        return;
    }
    double2 poly[KT];
#pragma unroll
    for (int k = 0; k < KT; k++) poly[k] = k < len ? v[idx[k]] : make_double2(0.0, 0.0);
    const double2 l2 = v[last];
    dpt a = mkp(l2.x, l2.y), b = mkp(poly[0].x, poly[0].y);
    bool bad = false;
    dpt U = vsub(b, a);
    double Ai = sf_abs_cross(U, vsub(p, a), &bad);
    bool clear = cl_float(Ai) > 1.01f * tolf * (fabsf(cl_float(U.x)) + fabsf(cl_float(U.y)) + 2.4e-38f);
    double ww[KT], sum = 0.0;
#pragma unroll
    for (int k = 0; k < KT; k++) {
        ww[k] = 0.0;
        if (k < len) {
            const double2 c2 = (k + 1 < KT && k + 1 < len) ? poly[k + 1 < KT ? k + 1 : 0] : poly[0];
            const dpt c = mkp(c2.x, c2.y);
            const double Ci = sf_abs_cross(U, vsub(c, a), &bad);
            U = vsub(c, b);
            const double Aj = sf_abs_cross(U, vsub(p, b), &bad);
            clear = clear && cl_float(Aj) > 1.01f * tolf * (fabsf(cl_float(U.x)) + fabsf(cl_float(U.y)) + 2.4e-38f);
            ww[k] = sf_div(sf_twice(Ci, &bad), sf_mul(Ai, Aj, &bad), &bad);
            sum += ww[k];
            a = b;
            b = c;
            Ai = Aj;
        }
    }
#pragma unroll
    for (int k = 0; k < KT; k++) ww[k] = sf_div(ww[k], sum, &bad);
    if (bad || !clear) {
        bary_general(pp, f, (const double*)v, faces, K, tol, w);
        return;
    }
#pragma unroll
    for (int k = 0; k < KT; k++)
        if (k < K) w[k] = ww[k];
}

// The same for triangles (tri_weights).
__global__ void __launch_bounds__(128) k_barycentric_tri(const double2* __restrict__ pts,
                                                         const int64_t* __restrict__ fidx, int64_t n,
                                                         const double2* __restrict__ v,
                                                         const int64_t* __restrict__ faces, double tol,
                                                         double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* w = out + i * 3;
    const int64_t f = fidx[i];
    if (f == -1) {
        w[0] = w[1] = w[2] = 0.0;
        return;
    }
    const int64_t* face = faces + f * 3;
    const double2 pp = pts[i], a2 = v[face[0]], b2 = v[face[1]], c2 = v[face[2]];
    const dpt a = mkp(a2.x, a2.y);
    const dpt ab = vsub(mkp(b2.x, b2.y), a), ac = vsub(mkp(c2.x, c2.y), a), ap = vsub(mkp(pp.x, pp.y), a);
    bool bad = false;
    const double Aa = sf_abs_cross(ab, ap, &bad), Ac = sf_abs_cross(ac, ap, &bad), A = sf_abs_cross(ab, ac, &bad);
    const double inv = sf_div(1.0, A, &bad);
    const double ww = sf_mul(inv, Aa, &bad), vv = sf_mul(inv, Ac, &bad);
    if (bad) {
        bary_general(pp, f, (const double*)v, faces, 3, tol, w);
        return;
    }
    w[0] = 1.0 - vv - ww;
    w[1] = vv;
    w[2] = ww;
}

// ---------------------------------------------------------------------------
// node-bound diagnostics (collect_node_bounds query.py:568-622,
// validate_node_bounds 625-663)
// ---------------------------------------------------------------------------
__global__ void k_parents(const int64_t* __restrict__ child, int64_t n_nodes, int64_t* __restrict__ parent) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_nodes) return;
    if (v == 0) parent[0] = -1;
    int64_t c = child[v];
    if (c > v && c + 1 < n_nodes) {
        parent[c] = v;
        parent[c + 1] = v;
    }
}

// A node's bounds are its parent's with one coordinate overwritten (left
// child: max of the parent's dim = Lmax; right child: min = Rmin).  Walking up
// from the node, the first ancestor edge that sets a coordinate wins.
__global__ void k_node_bounds(const int64_t* __restrict__ child, const double* __restrict__ Lmax,
                              const double* __restrict__ Rmin, const uint8_t* __restrict__ dim,
                              const int64_t* __restrict__ parent, int64_t n_nodes, double4 bbox,
                              double4* __restrict__ out) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_nodes) return;
    double b[4] = {bbox.x, bbox.y, bbox.z, bbox.w};
    bool set[4] = {false, false, false, false};
    int64_t u = v;
    int64_t guard = n_nodes;
    while (u > 0 && guard-- > 0) {
        int64_t p = parent[u];
        if (p < 0) break;
        int d = dim[p] ? 1 : 0;
        int side = (u == child[p]) ? 1 : 0;  // left child: side 1 (max), right: side 0 (min)
        int k = d * 2 + side;
        if (!set[k]) {
            b[k] = side ? Lmax[p] : Rmin[p];
            set[k] = true;
        }
        u = p;
    }
    out[v] = make_double4(b[0], b[1], b[2], b[3]);
}

__global__ void k_validate_bounds(const int64_t* __restrict__ child, const int64_t* __restrict__ ptr,
                                  const int64_t* __restrict__ size, const int64_t* __restrict__ bbi,
                                  const double* __restrict__ bb, const double4* __restrict__ nbnd, int64_t n_nodes,
                                  uint8_t* __restrict__ valid) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_nodes) return;
    double4 q = nbnd[v];
    dbox bx;
    bx.xmin = q.x;
    bx.xmax = q.y;
    bx.ymin = q.z;
    bx.ymax = q.w;
    int64_t c = child[v];
    bool ok = true;
    if (c == -1) {
        for (int64_t i = ptr[v]; i < ptr[v] + size[v]; i++) ok = ok && box_contained(load_box(bb + 4 * bbi[i]), bx);
    } else {
        double4 l = nbnd[c], r = nbnd[c + 1];
        dbox lb, rb;
        lb.xmin = l.x;
        lb.xmax = l.y;
        lb.ymin = l.z;
        lb.ymax = l.w;
        rb.xmin = r.x;
        rb.xmax = r.y;
        rb.ymin = r.z;
        rb.ymax = r.w;
        ok = box_contained(lb, bx) && box_contained(rb, bx);
    }
    valid[v] = (uint8_t)ok;
}

// 8-bit work class of a box (kind 0: area with a cell-size margin) or a
// segment (kind 1: length plus a cell size): 4 * log2(work) + 128, clamped.
__global__ void k_work_keys(const double4* __restrict__ q, int64_t n, int kind, float cell,
                            unsigned* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double4 v = q[i];
        float w;
        if (kind == 0) {
            float dx = (float)(v.y - v.x), dy = (float)(v.w - v.z);
            w = (fabsf(dx) + cell) * (fabsf(dy) + cell);
        } else {
            float dx = (float)(v.z - v.x), dy = (float)(v.w - v.y);
            w = sqrtf(dx * dx + dy * dy) + cell;
        }
        int k = (w > 0.0f) ? (int)floorf(4.0f * log2f(w)) + 128 : 0;  // NaN -> 0
        key[i] = (unsigned)min(max(k, 0), 255);
    }
}

// 16-bit Morton key of a box's (kind 0) or segment's (kind 1) middle on a
// 256 x 256 grid over the tree's bbox (outside and NaN: the nearest cell, 0).
__global__ void k_spatial_keys(const double4* __restrict__ q, int64_t n, int kind, double x0, double y0, float sx,
                               float sy, unsigned* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 v = q[i];
        const float a = (float)(v.x - x0), c = (float)(v.z - (kind == 0 ? y0 : x0));
        const float b = (float)(v.y - (kind == 0 ? x0 : y0)), d = (float)(v.w - y0);
        const float mx = kind == 0 ? a + b : a + c, my = kind == 0 ? c + d : b + d;
        unsigned k = 0;
        const unsigned gx = (unsigned)fminf(fmaxf(0.5f * mx * sx, 0.0f), 255.0f);
        const unsigned gy = (unsigned)fminf(fmaxf(0.5f * my * sy, 0.0f), 255.0f);
        for (int b2 = 0; b2 < 8; b2++) k |= (((gx >> b2) & 1u) << (2 * b2)) | (((gy >> b2) & 1u) << (2 * b2 + 1));
        key[i] = k;
    }
}

// At most BOX_SAMPLE boxes spread over the batch, a thread each: the mean of
// the cells they may overlap, in cells of side c, and the share whose middle
// lies within 16 cells of the next box's.
constexpr int BOX_SAMPLE = 1024;
__global__ void __launch_bounds__(BOX_SAMPLE) k_box_sample(const double4* __restrict__ boxes, int64_t n, float W,
                                                           float H, float c, double* __restrict__ out) {
    __shared__ float part[2][32];
    const int m = (int)min(n, (int64_t)BOX_SAMPLE), k = threadIdx.x;
    float v[2] = {0.0f, 0.0f};
    if (k < m) {
        const int64_t i = (int64_t)((double)n / m * k);
        const double4 b = boxes[i], d = boxes[min(i + 1, n - 1)];
        // NaN counts as no extent (and as far away)
        const float w = (float)(b.y - b.x), h = (float)(b.w - b.z);
        v[0] = (fminf(fmaxf(w, 0.0f), W) / c + 1.0f) * (fminf(fmaxf(h, 0.0f), H) / c + 1.0f);
        const float dx = (float)(d.x - b.x) + 0.5f * ((float)(d.y - d.x) - w);
        const float dy = (float)(d.z - b.z) + 0.5f * ((float)(d.w - d.z) - h);
        v[1] = fabsf(dx) <= 16.0f * c && fabsf(dy) <= 16.0f * c ? 1.0f : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if ((k & 31) == 0) part[q][k >> 5] = v[q];
    }
    __syncthreads();
    if (k < 32) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            v[q] = part[q][k];
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            if (k == 0) out[q] = (double)v[q] / m;
        }
    }
}

__global__ void k_gather_rows(const double4* __restrict__ q, const int* __restrict__ order, int64_t n,
                              double4* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = q[order[i]];
}

// block sizes of the traversal kernels (the tree's launch shape, else the defaults)
static int box_threads(const ct_tree* t) {
    int b = t->tune_query_threads;
    return (b == 64 || b == 128 || b == 256) ? b : 256;
}
static int seg_threads(const ct_tree* t) {
    int b = t->tune_query_threads;
    return (b == 64 || b == 128) ? b : 128;
}

TreeQ make_q(const ct_tree* t) {
    TreeQ T;
    T.nf = (const float4*)t->nodes_f32;
    T.nd = (const double2*)t->nodes_f64;
    T.poly = (const double2*)t->poly_f64;
    T.plen = t->n_max_vert == 3 || t->n_max_vert == 2 ? nullptr : t->poly_len;
    T.bbi = t->bb_indices;
    T.bb = t->bb_coords;
    T.err = t->error_word;
    T.n_nodes = t->n_nodes;
    T.bbox.xmin = t->bbox[0];
    T.bbox.xmax = t->bbox[1];
    T.bbox.ymin = t->bbox[2];
    T.bbox.ymax = t->bbox[3];
    T.K = t->n_max_vert;
    T.finite = t->bounds_finite != 0;
    T.box_warps = box_threads(t) / 64;  // 1, 2, 4
    T.seg_warps = seg_threads(t) / 32;  // 2, 4
    const bool box_index = t->node_box && t->leaf_start && t->bb_leaf && T.finite;
    T.bbl = box_index ? (const double4*)t->bb_leaf : nullptr;
    T.nbx = box_index ? (const NodeBox*)t->node_box : nullptr;
    T.lstart = box_index ? t->leaf_start : nullptr;
    T.ox = t->origin[0];
    T.oy = t->origin[1];
    T.bbl32 = (box_index && t->bb_leaf32) ? (const float4*)t->bb_leaf32 : nullptr;
    T.fX = (float)std::max(std::fabs(t->bbox[0] - T.ox), std::fabs(t->bbox[1] - T.ox)) * (1.0f + 0x1p-20f);
    T.fY = (float)std::max(std::fabs(t->bbox[2] - T.oy), std::fabs(t->bbox[3] - T.oy)) * (1.0f + 0x1p-20f);
    T.babs = std::max(std::max(std::fabs(t->bbox[0]), std::fabs(t->bbox[1])),
                      std::max(std::fabs(t->bbox[2]), std::fabs(t->bbox[3])));
    T.mext = 0x1p-37 * std::max(t->bbox[1] - t->bbox[0], t->bbox[3] - t->bbox[2]) + 0x1p-47;
    if (!(T.fX <= 3.0e38f && T.fY <= 3.0e38f && T.babs <= 1.0e300 && T.mext <= 1.0e300)) T.bbl32 = nullptr;
    T.parent = t->node_parent;
    T.polyf = (const float4*)t->poly_f32;
    T.plen32 = t->poly_len32;
    T.S4 = poly32_stride(t->n_max_vert);
    T.dabs = t->abs_eps;
    return T;
}

// ---------------------------------------------------------------------------
// Box index (no upstream counterpart), built once per tree:
//  * bb_leaf: bb_coords in leaf order (the leaf loop reads them in sequence
//    instead of through bb_indices);
//  * leaf_start: for every leaf position the first position of its leaf;
//  * node_box: per node the bounding box of the cells below it (leaves from
//    their cells, then up the parent chain with integer-key atomics; a leaf
//    stops climbing where its box is already covered, since whichever leaf
//    widened that node carries the wider box further up) and its leaf range.
// ---------------------------------------------------------------------------
__global__ void k_bi_leaf_boxes(const int64_t* __restrict__ bbi, const double4* __restrict__ bb, int64_t n,
                                double4* __restrict__ bbl) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        bbl[p] = bb[bbi[p]];
}

// bb_leaf in the float32 frame, rounded outward (the subtraction of the
// origin rounded outward too): contains the cell's box exactly.
__global__ void k_bi_leaf32(const double4* __restrict__ bbl, int64_t n, double ox, double oy,
                            float4* __restrict__ out) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const double4 b = bbl[p];
        out[p] = make_float4(__double2float_rd(__dsub_rd(b.x, ox)), __double2float_ru(__dsub_ru(b.y, ox)),
                             __double2float_rd(__dsub_rd(b.z, oy)), __double2float_ru(__dsub_ru(b.w, oy)));
    }
}

__global__ void k_bi_parents(const int64_t* __restrict__ child, int64_t nn, int* __restrict__ parent,
                             unsigned long long* __restrict__ keys) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nn) return;
    int64_t c = child[v];
    if (c >= 0 && c + 1 < nn) {
        parent[c] = (int)v;
        parent[c + 1] = (int)v;
    }
    keys[4 * v + 0] = ~0ull;
    keys[4 * v + 1] = 0ull;
    keys[4 * v + 2] = ~0ull;
    keys[4 * v + 3] = 0ull;
}

__global__ void k_bi_leaves(const int64_t* __restrict__ child, const int64_t* __restrict__ ptr,
                            const int64_t* __restrict__ size, int64_t nn, const double4* __restrict__ bbl, int64_t n,
                            const int* __restrict__ parent, unsigned long long* __restrict__ keys,
                            int* __restrict__ lstart, unsigned int* __restrict__ err) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nn || child[v] >= 0) return;
    int64_t p0 = ptr[v], sz = size[v];
    if (p0 < 0 || sz < 0 || p0 + sz > n) {
        set_error(err, CT_DEVERR_CAPACITY);
        return;
    }
    if (sz == 0) return;
    unsigned long long x0 = ~0ull, x1 = 0ull, y0 = ~0ull, y1 = 0ull;
    for (int64_t p = p0; p < p0 + sz; p++) {
        lstart[p] = (int)p0;
        double4 b = bbl[p];
        x0 = min(x0, fkey(b.x));
        x1 = max(x1, fkey(b.y));
        y0 = min(y0, fkey(b.z));
        y1 = max(y1, fkey(b.w));
    }
    int u = (int)v;
    for (int64_t guard = nn; u >= 0 && guard > 0; guard--) {
        unsigned long long* k = keys + 4 * (int64_t)u;
        unsigned long long o0 = atomicMin(k + 0, x0), o1 = atomicMax(k + 1, x1);
        unsigned long long o2 = atomicMin(k + 2, y0), o3 = atomicMax(k + 3, y1);
        if (o0 <= x0 && o1 >= x1 && o2 <= y0 && o3 >= y1) break;
        u = parent[u];
    }
}

__global__ void k_bi_nodes(const int64_t* __restrict__ ptr, const int64_t* __restrict__ size, int64_t nn,
                           const unsigned long long* __restrict__ keys, double ox, double oy,
                           NodeBox* __restrict__ out) {
    int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nn) return;
    NodeBox b;
    const unsigned long long* k = keys + 4 * v;
    if (k[0] == ~0ull) {  // no cells: never "inside" a query box
        b.xmin = b.ymin = __int_as_float(0x7fc00000);
        b.xmax = b.ymax = __int_as_float(0x7fc00000);
    } else {
        b.xmin = __double2float_rd(fkey_inv(k[0]) - ox);
        b.xmax = __double2float_ru(fkey_inv(k[1]) - ox);
        b.ymin = __double2float_rd(fkey_inv(k[2]) - oy);
        b.ymax = __double2float_ru(fkey_inv(k[3]) - oy);
    }
    b.ptr = (int)ptr[v];
    b.size = (int)size[v];
    b.pad0 = b.pad1 = 0;
    out[v] = b;
}

static inline unsigned grid_of(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace ctm

using namespace ctm;

// Tasks per warp: one while they do not fill the resident warps (152 SMs x
// 32), up to 8 beyond, so that a round's 32 lanes find nodes at every level.
static int walk_tasks(int64_t n) {
    int per_warp = 1;
    while (per_warp < WALK_Q && n / (2 * per_warp) >= 152 * 32) per_warp *= 2;
    return per_warp;
}

template <int MODE>
static void launch_box_walk(const TreeQ& T, const double4* boxes, int64_t n, const int* order, int64_t* cnt_or_off,
                            int64_t* ii, int64_t* jj, int* spec, int spcap, const int64_t* spec_cnt,
                            cudaStream_t st, BoxRecs recs = {}) {
    const int per_warp = walk_tasks(n);
    const int w = T.box_warps;
    const size_t smem = w * sizeof(WalkShared<WalkBox, int64_t>);
    k_box_walk<MODE><<<grid_of((n + per_warp - 1) / per_warp, w), 32 * w, smem, st>>>(
        T, boxes, n, order, per_warp, cnt_or_off, ii, jj, spec, spcap, spec_cnt, recs);
}

template <bool ITEMS, bool WRITE>
static void launch_edge_walk(int mode, const TreeQ& T, const double4* segs, int64_t n, const int* order,
                             const int* item_seg, const int* item_node, int cut, int64_t* cnt_or_off, int* out_seg,
                             int* out_val, int spcap, const int64_t* spec_cnt, cudaStream_t st) {
    const int per_warp = walk_tasks(n);
    const int w = T.seg_warps;
    const unsigned g = grid_of((n + per_warp - 1) / per_warp, w);
    const size_t smem = w * sizeof(WalkShared<WalkSeg, int>);
    if (mode == 0)
        k_edge_walk<0, ITEMS, WRITE><<<g, 32 * w, smem, st>>>(T, segs, n, order, item_seg, item_node, cut,
                                                                    per_warp, cnt_or_off, out_seg, out_val, spcap,
                                                                    spec_cnt);
    else
        k_edge_walk<1, ITEMS, WRITE><<<g, 32 * w, smem, st>>>(T, segs, n, order, item_seg, item_node, cut,
                                                                    per_warp, cnt_or_off, out_seg, out_val, spcap,
                                                                    spec_cnt);
}

extern "C" {

size_t ct_scan_workspace_size(int64_t n) {
    int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    return (size_t)(nb + 1) * sizeof(int64_t);
}

int ct_exclusive_scan(const int64_t* in, int64_t n, int64_t* out, void* ws, size_t ws_bytes, int64_t* total_host,
                      void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 0) return ct_fail(CT_ERR_ARG, "negative length");
    if (ws_bytes < ct_scan_workspace_size(n) || !ws) return ct_fail(CT_ERR_WORKSPACE, "scan workspace too small");
    int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    int64_t* sums = (int64_t*)ws;
    if (nb > 0) {
        k_scan_reduce<<<(unsigned)nb, SCAN_T, 0, st>>>(in, n, sums);
        k_scan_sums<<<1, SCAN_T, 0, st>>>(sums, nb);
        k_scan_down<<<(unsigned)nb, SCAN_T, 0, st>>>(in, n, sums, out);
    } else {
        CT_CUDA(cudaMemsetAsync(sums, 0, sizeof(int64_t), st));
    }
    CT_CHECK_LAUNCH("scan");
    if (total_host) {
        CT_CUDA(cudaMemcpyAsync(total_host, sums + nb, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        CT_CUDA(cudaStreamSynchronize(st));
    }
    return CT_OK;
}

size_t ct_box_index_scratch_size(const ct_tree* t) {
    if (!t || t->n_nodes <= 0) return 0;
    return (size_t)t->n_nodes * (4 * sizeof(unsigned long long) + sizeof(int)) + 256;
}

int ct_pack_box_index(ct_tree* t, void* scratch, size_t scratch_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (!t) return ct_fail(CT_ERR_ARG, "tree is null");
    if (!t->bb_leaf || !t->node_box || !t->leaf_start) return ct_fail(CT_ERR_ARG, "box index arrays not set");
    if (t->n_nodes <= 0 || t->n_nodes >= INT32_MAX || t->n_elements >= INT32_MAX)
        return ct_fail(CT_ERR_ARG, "tree size out of range");
    if (!scratch || scratch_bytes < ct_box_index_scratch_size(t))
        return ct_fail(CT_ERR_WORKSPACE, "box index scratch too small");
    int64_t nn = t->n_nodes, n = t->n_elements;
    unsigned long long* keys = (unsigned long long*)scratch;
    int* parent = (int*)(keys + 4 * nn);
    CT_CUDA(cudaMemsetAsync(parent, 0xff, (size_t)nn * sizeof(int), st));
    if (n > 0) {
        k_bi_leaf_boxes<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 8), 256, 0, st>>>(
            t->bb_indices, (const double4*)t->bb_coords, n, (double4*)t->bb_leaf);
        if (t->bb_leaf32)
            k_bi_leaf32<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 8), 256, 0, st>>>(
                (const double4*)t->bb_leaf, n, t->origin[0], t->origin[1], (float4*)t->bb_leaf32);
    }
    k_bi_parents<<<grid_of(nn, 256), 256, 0, st>>>(t->node_child, nn, parent, keys);
    k_bi_leaves<<<grid_of(nn, 128), 128, 0, st>>>(t->node_child, t->node_ptr, t->node_size, nn,
                                                  (const double4*)t->bb_leaf, n, parent, keys, t->leaf_start,
                                                  t->error_word);
    k_bi_nodes<<<grid_of(nn, 256), 256, 0, st>>>(t->node_ptr, t->node_size, nn, keys, t->origin[0], t->origin[1],
                                                 (NodeBox*)t->node_box);
    CT_CHECK_LAUNCH("pack_box_index");
    return CT_OK;
}

// Polygons of up to 8 vertices take the shared-memory clip, longer ones the
// general one (shared memory of a block: 31, 33 and 41 KB for clippers of up
// to 3, 4 and 8 vertices).
static void launch_clip_area(const double4* boxes, const double* va, const int64_t* fa, int Ka, const double* vb,
                             const int64_t* fb, int Kb, const int64_t* ia, const int64_t* ib, int64_t n,
                             const int* order, double* out, unsigned int* err, cudaStream_t st) {
    const unsigned grid = grid_of(n, CL_THREADS);
    const double2 *a = (const double2*)va, *b = (const double2*)vb;
    if (Ka > CL_SLOTS || Kb > 8 || Ka < 3 || Kb < 3 || (((uintptr_t)va | (uintptr_t)vb) & 15))
        k_clip_area<<<grid_of(n, 128), 128, 0, st>>>(boxes, va, fa, Ka, vb, fb, Kb, ia, ib, n, order, out, err);
    else {
        auto go = [&](auto kt) {
            constexpr int KT = decltype(kt)::value;
            if (boxes)
                k_clip_area_small<KT, true><<<grid, CL_THREADS, 0, st>>>(boxes, a, fa, Ka, b, fb, Kb, ia, ib, n,
                                                                         order, out, err);
            else
                k_clip_area_small<KT, false><<<grid, CL_THREADS, 0, st>>>(boxes, a, fa, Ka, b, fb, Kb, ia, ib, n,
                                                                          order, out, err);
        };
        if (Kb <= 3) go(std::integral_constant<int, 3>());
        else if (Kb <= 4) go(std::integral_constant<int, 4>());
        else go(std::integral_constant<int, 8>());
    }
}

static int check_tree(const ct_tree* t) {
    if (!t) return ct_fail(CT_ERR_ARG, "tree is null");
    if (t->n_nodes <= 0) return ct_fail(CT_ERR_ARG, "tree has no nodes");
    if (t->max_depth + 2 > STK && !t->node_parent)
        return ct_fail(CT_ERR_ARG, "tree deeper than 126 levels for multi-result queries (no node_parent)");
    return CT_OK;
}

// trees deeper than the traversal stack are walked through the node parents
static bool deep_tree(const ct_tree* t) { return t->max_depth + 2 > STK; }

int ct_count_boxes(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order, int64_t* counts,
                   void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    const int bt = box_threads(t);
    if (deep_tree(t))
        k_boxes<false, true><<<grid_of(n, bt), bt, 0, (cudaStream_t)stream>>>(make_q(t), (const double4*)boxes, n,
                                                                             order, counts, nullptr, nullptr);
    else
        launch_box_walk<BOX_COUNT>(make_q(t), (const double4*)boxes, n, order, counts, nullptr, nullptr, nullptr, 0,
                               nullptr, (cudaStream_t)stream);
    CT_CHECK_LAUNCH("count_boxes");
    return CT_OK;
}

int ct_write_boxes(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order, const int64_t* offsets,
                   int64_t* ii, int64_t* jj, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    const int bt = box_threads(t);
    if (deep_tree(t))
        k_boxes<true, true><<<grid_of(n, bt), bt, 0, (cudaStream_t)stream>>>(make_q(t), (const double4*)boxes, n,
                                                                            order, (int64_t*)offsets, ii, jj);
    else
        launch_box_walk<BOX_WRITE>(make_q(t), (const double4*)boxes, n, order, (int64_t*)offsets, ii, jj, nullptr, 0,
                              nullptr, (cudaStream_t)stream);
    CT_CHECK_LAUNCH("write_boxes");
    return CT_OK;
}

static int box_job_min(int32_t m) { return m > 0 ? (m < 2 ? 2 : m) : BOX_JOB_MIN; }

size_t ct_write_boxes_workspace_size(int64_t total_pairs, int32_t min_job_cells) {
    const int64_t cap = (total_pairs > 0 ? total_pairs : 0) / box_job_min(min_job_cells) + 1;
    return 256 + (size_t)cap * sizeof(BoxJob);
}

// records: the two counts, then the records
static BoxRecs box_recs(void* records, int64_t capacity, uint8_t* inside) {
    unsigned long long* counts = (unsigned long long*)records;
    return BoxRecs{(int4*)((char*)records + 256), counts, counts + 1, capacity, REC_PART, inside};
}

static void launch_box_records(const TreeQ& T, const double4* boxes, const BoxRecs& R, const int64_t* off, int64_t* ii,
                               int64_t* jj, cudaStream_t st) {
    k_box_records<<<(unsigned)std::min<int64_t>((R.cap + 255) / 256, 152 * 64), 256, 0, st>>>(T, boxes, R, off, ii, jj);
}

// The boxes walked (those of spec_cnt above spec_cap, if given), their whole
// subtrees left to k_box_records in the job workspace.
static int walk_boxes_ws(const TreeQ& T, const double4* boxes, int64_t n, const int* order, const int64_t* off,
                         int spec_cap, const int64_t* spec_cnt, int64_t total_pairs, int min_job_cells, int64_t* ii,
                         int64_t* jj, void* ws, cudaStream_t st) {
    BoxRecs R = {};
    if (T.nbx && n < INT32_MAX) {  // (without the box index no subtree is known to lie inside)
        const int jm = box_job_min(min_job_cells);
        R = box_recs(ws, (total_pairs > 0 ? total_pairs : 0) / jm + 1, nullptr);
        R.count = nullptr;
        R.part = std::max(jm, REC_PART);
        CT_CUDA(cudaMemsetAsync(R.pushed, 0, sizeof(unsigned long long), st));
    }
    launch_box_walk<BOX_WRITE>(T, boxes, n, order, (int64_t*)off, ii, jj, nullptr, spec_cap, spec_cnt, st, R);
    if (R.rec) launch_box_records(T, boxes, R, off, ii, jj, st);
    return CT_OK;
}

int ct_write_boxes_ws(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order,
                      const int64_t* offsets, int64_t total_pairs, int32_t min_job_cells, int64_t* ii, int64_t* jj,
                      void* ws, size_t ws_bytes, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (total_pairs < 0) return ct_fail(CT_ERR_ARG, "negative pair count");
    if (!ws || ws_bytes < ct_write_boxes_workspace_size(total_pairs, min_job_cells))
        return ct_fail(CT_ERR_WORKSPACE, "write_boxes workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    if (!deep_tree(t)) {
        int s2 = walk_boxes_ws(T, (const double4*)boxes, n, order, offsets, 0, nullptr, total_pairs, min_job_cells, ii, jj,
                               ws, st);
        if (s2) return s2;
        CT_CHECK_LAUNCH("write_boxes");
        return CT_OK;
    }
    if (!T.nbx) return ct_write_boxes(t, boxes, n, order, offsets, ii, jj, stream);  // no box index: no subtrees
    const int jm = box_job_min(min_job_cells);
    unsigned long long* njobs = (unsigned long long*)ws;
    BoxJob* jobs = (BoxJob*)((char*)ws + 256);
    const int64_t cap = (total_pairs > 0 ? total_pairs : 0) / jm + 1;
    CT_CUDA(cudaMemsetAsync(njobs, 0, sizeof(unsigned long long), st));
    const int bt = box_threads(t);
    k_boxes<true, true><<<grid_of(n, bt), bt, 0, st>>>(T, (const double4*)boxes, n, order, (int64_t*)offsets, ii, jj,
                                                      jobs, njobs, cap, jm);
    k_box_jobs<<<152 * 8, 256, 0, st>>>(jobs, njobs, cap, T.lstart, T.bbi, ii, jj, T.err);
    CT_CHECK_LAUNCH("write_boxes");
    return CT_OK;
}

int ct_count_boxes_spec(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order, int64_t* counts,
                        int32_t* spec, int32_t spec_cap, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    if (t->n_elements >= INT32_MAX) return ct_fail(CT_ERR_ARG, "tree size out of range");
    const int bt = box_threads(t);
    cudaStream_t st = (cudaStream_t)stream;
    const TreeQ T = make_q(t);
    const double4* B = (const double4*)boxes;
    if (deep_tree(t))
        k_boxes<false, true><<<grid_of(n, bt), bt, 0, st>>>(T, B, n, order, counts, nullptr, nullptr, nullptr, nullptr,
                                                           0, BOX_JOB_MIN, spec, spec_cap, nullptr);
    else
        launch_box_walk<BOX_COUNT>(T, B, n, order, counts, nullptr, nullptr, spec, spec_cap, nullptr, st);
    CT_CHECK_LAUNCH("count_boxes_spec");
    return CT_OK;
}

size_t ct_box_records_size(int64_t capacity) { return 256 + sizeof(int4) * (size_t)(capacity > 0 ? capacity : 1); }

int ct_count_boxes_records(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order, int64_t* counts,
                           void* records, int64_t capacity, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (!records || capacity < 1) return ct_fail(CT_ERR_ARG, "no room for records");
    if (n >= INT32_MAX || t->n_elements >= INT32_MAX) return ct_fail(CT_ERR_ARG, "batch or tree size out of range");
    cudaStream_t st = (cudaStream_t)stream;
    if (deep_tree(t)) {  // no records: the writing call walks again
        CT_CUDA(cudaMemsetAsync(records, 0xff, sizeof(unsigned long long), st));
        return ct_count_boxes(t, boxes, n, order, counts, stream);
    }
    CT_CUDA(cudaMemsetAsync(records, 0, 2 * sizeof(unsigned long long), st));
    if (n == 0) return CT_OK;
    launch_box_walk<BOX_RECORD>(make_q(t), (const double4*)boxes, n, order, counts, nullptr, nullptr, nullptr, 0, nullptr,
                                st, box_recs(records, capacity, nullptr));
    CT_CHECK_LAUNCH("count_boxes_records");
    return CT_OK;
}

int ct_write_boxes_records(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order,
                           const int64_t* offsets, const void* records, int64_t capacity, int64_t total_pairs,
                           int64_t* ii, int64_t* jj, uint8_t* inside, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (!records || capacity < 1) return ct_fail(CT_ERR_ARG, "no records");
    cudaStream_t st = (cudaStream_t)stream;
    if (inside && total_pairs > 0) CT_CUDA(cudaMemsetAsync(inside, 0, (size_t)total_pairs, st));
    if (deep_tree(t)) return ct_write_boxes(t, boxes, n, order, offsets, ii, jj, stream);
    const TreeQ T = make_q(t);
    const double4* B = (const double4*)boxes;
    const BoxRecs R = box_recs((void*)records, capacity, inside);
    launch_box_walk<BOX_WRITE>(T, B, n, order, (int64_t*)offsets, ii, jj, nullptr, 0, nullptr, st, R);
    launch_box_records(T, B, R, offsets, ii, jj, st);
    CT_CHECK_LAUNCH("write_boxes_records");
    return CT_OK;
}

int ct_box_sample(const ct_tree* t, const double* boxes, int64_t n, double* result_host2, void* ws, size_t ws_bytes,
                  void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n < 0 || !result_host2) return ct_fail(CT_ERR_ARG, "bad arguments");
    result_host2[0] = result_host2[1] = 0.0;
    if (n == 0 || t->n_elements <= 0) return CT_OK;
    if (!ws || ws_bytes < 2 * sizeof(double)) return ct_fail(CT_ERR_WORKSPACE, "workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    const double W = t->bbox[1] - t->bbox[0], H = t->bbox[3] - t->bbox[2], m = (double)t->n_elements;
    const double c = W > 0.0 && H > 0.0 ? std::sqrt(W / m * H) : std::max(W, H) / m;  // (cells in a line)
    k_box_sample<<<1, BOX_SAMPLE, 0, st>>>((const double4*)boxes, n, (float)W, (float)H,
                                           c > 1e-37 ? (float)std::min(c, 1e37) : 1e-37f, (double*)ws);
    CT_CHECK_LAUNCH("box sample");
    CT_CUDA(cudaMemcpyAsync(result_host2, ws, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CT_CUDA(cudaStreamSynchronize(st));
    return CT_OK;
}

int ct_write_small_boxes(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order,
                         const int64_t* offsets, int64_t total_pairs, int64_t* ii, int64_t* jj, void* ws,
                         size_t ws_bytes, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (deep_tree(t)) return ct_write_boxes_ws(t, boxes, n, order, offsets, total_pairs, 0, ii, jj, ws, ws_bytes, stream);
    if (!ws || ws_bytes < ct_write_boxes_workspace_size(total_pairs, 0))
        return ct_fail(CT_ERR_WORKSPACE, "write_boxes workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    const TreeQ T = make_q(t);
    unsigned long long* njobs = (unsigned long long*)ws;
    BoxJob* jobs = T.nbx ? (BoxJob*)((char*)ws + 256) : nullptr;
    const int64_t cap = (total_pairs > 0 ? total_pairs : 0) / BOX_JOB_MIN + 1;
    CT_CUDA(cudaMemsetAsync(njobs, 0, sizeof(unsigned long long), st));
    const int bt = box_threads(t);
    k_boxes<true, false><<<grid_of(n, bt), bt, 0, st>>>(T, (const double4*)boxes, n, order, (int64_t*)offsets, ii, jj,
                                                       jobs, njobs, cap, BOX_JOB_MIN);
    if (jobs) k_box_jobs<<<152 * 8, 256, 0, st>>>(jobs, njobs, cap, T.lstart, T.bbi, ii, jj, T.err);
    CT_CHECK_LAUNCH("write_small_boxes");
    return CT_OK;
}

int ct_count_small_boxes_spec(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order, int64_t* counts,
                              int32_t* spec, int32_t spec_cap, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (!spec && spec_cap == 0) {  // counts alone
        if (n == 0 || deep_tree(t)) return ct_count_boxes(t, boxes, n, order, counts, stream);
        const int bt = box_threads(t);
        k_boxes<false, false><<<grid_of(n, bt), bt, 0, (cudaStream_t)stream>>>(make_q(t), (const double4*)boxes, n, order,
                                                                              counts, nullptr, nullptr);
        CT_CHECK_LAUNCH("count_small_boxes");
        return CT_OK;
    }
    if (n == 0 || deep_tree(t)) return ct_count_boxes_spec(t, boxes, n, order, counts, spec, spec_cap, stream);
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    if (t->n_elements >= INT32_MAX) return ct_fail(CT_ERR_ARG, "tree size out of range");
    const int bt = box_threads(t);
    k_boxes<false, false><<<grid_of(n, bt), bt, 0, (cudaStream_t)stream>>>(
        make_q(t), (const double4*)boxes, n, order, counts, nullptr, nullptr, nullptr, nullptr, 0, BOX_JOB_MIN, spec,
        spec_cap, nullptr);
    CT_CHECK_LAUNCH("count_small_boxes_spec");
    return CT_OK;
}

int ct_write_boxes_spec(const ct_tree* t, const double* boxes, int64_t n, const int32_t* order,
                        const int64_t* counts, const int64_t* offsets, const int32_t* spec, int32_t spec_cap,
                        int64_t total_pairs, int32_t min_job_cells, int64_t* ii, int64_t* jj, void* ws,
                        size_t ws_bytes, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    if (total_pairs < 0) return ct_fail(CT_ERR_ARG, "negative pair count");
    if (!ws || ws_bytes < ct_write_boxes_workspace_size(total_pairs, min_job_cells))
        return ct_fail(CT_ERR_WORKSPACE, "write_boxes workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    const TreeQ T = make_q(t);
    k_boxes_spec_emit<<<(unsigned)std::min<int64_t>(grid_of(4 * n, 256), 152 * 64), 256, 0, st>>>(
        counts, offsets, n, spec, spec_cap, ii, jj);
    int64_t* off = (int64_t*)offsets;
    const double4* B = (const double4*)boxes;
    if (!deep_tree(t)) {
        int s2 = walk_boxes_ws(T, B, n, order, off, spec_cap, counts, total_pairs, min_job_cells, ii, jj, ws, st);
        if (s2) return s2;
        CT_CHECK_LAUNCH("write_boxes_spec");
        return CT_OK;
    }
    const int jm = box_job_min(min_job_cells);
    unsigned long long* njobs = (unsigned long long*)ws;
    BoxJob* jobs = T.nbx ? (BoxJob*)((char*)ws + 256) : nullptr;
    const int64_t cap = (total_pairs > 0 ? total_pairs : 0) / jm + 1;
    CT_CUDA(cudaMemsetAsync(njobs, 0, sizeof(unsigned long long), st));
    const int bt = box_threads(t);
    k_boxes<true, true><<<grid_of(n, bt), bt, 0, st>>>(T, B, n, order, off, ii, jj, jobs, njobs, cap, jm, nullptr,
                                                      spec_cap, counts);
    if (jobs) k_box_jobs<<<152 * 8, 256, 0, st>>>(jobs, njobs, cap, T.lstart, T.bbi, ii, jj, T.err);
    CT_CHECK_LAUNCH("write_boxes_spec");
    return CT_OK;
}

size_t ct_sort_workspace_size(int64_t total) {
    const size_t t = (size_t)(total > 0 ? total : 1);
    return t * 4 * 8 + (t / (WARP_SORT_MAX + 1) + 2) * sizeof(int) + 1024 + 256;
}

int ct_sort_intersections(const double* segs, int64_t n_segs, const int64_t* offsets, const int64_t* counts,
                          const int64_t* ii, const int64_t* jj_in, const double* xy_in, int64_t total,
                          int64_t* jj_out, double* xy_out, void* ws, size_t ws_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (total == 0) return CT_OK;
    if (!ws || ws_bytes < ct_sort_workspace_size(total)) return ct_fail(CT_ERR_WORKSPACE, "sort workspace too small");
    unsigned long long* kA = (unsigned long long*)ws;
    int64_t* iA = (int64_t*)(kA + total);
    unsigned long long* kB = (unsigned long long*)(iA + total);
    int64_t* iB = (int64_t*)(kB + total);
    unsigned long long* nlist = (unsigned long long*)(iB + total);  // 8 B, then the list of long segments
    int* list = (int*)(nlist + 1);
    if (n_segs > INT32_MAX) return ct_fail(CT_ERR_ARG, "at most 2^31 - 1 segments");
    CT_CUDA(cudaMemsetAsync(nlist, 0, sizeof(unsigned long long), st));
    k_tkeys<<<grid_of(total, 256), 256, 0, st>>>((const double4*)segs, ii, (const double4*)xy_in, total, kA, iA);
    k_segsort_warp<<<(unsigned)std::min<int64_t>(grid_of(n_segs * 32, 256), 152 * 32), 256, 0, st>>>(
        offsets, counts, n_segs, kA, iA, iB, list, nlist);
    k_segsort<<<152 * 4, SORT_T, 0, st>>>(offsets, counts, list, nlist, kA, iA, kB, iB, iB);
    // iB now holds, per segment, the sorted source positions (segments of one
    // result write them directly)
    k_gather_results<<<grid_of(total, 256), 256, 0, st>>>(iB, total, jj_in, (const double4*)xy_in, jj_out,
                                                          (double4*)xy_out);
    CT_CHECK_LAUNCH("sort_intersections");
    return CT_OK;
}

int ct_polygons_intersect(const double* va, const int64_t* fa, int32_t Ka, const double* vb, const int64_t* fb,
                          int32_t Kb, const int64_t* ia, const int64_t* ib, int64_t n, uint8_t* out, void* stream) {
    if (n == 0) return CT_OK;
    k_sat<<<grid_of(n, 128), 128, 0, (cudaStream_t)stream>>>(va, fa, Ka, vb, fb, Kb, ia, ib, n, out);
    CT_CHECK_LAUNCH("polygons_intersect");
    return CT_OK;
}

int ct_area_of_intersection_ordered(const double* va, const int64_t* fa, int32_t Ka, const double* vb,
                                    const int64_t* fb, int32_t Kb, const int64_t* ia, const int64_t* ib, int64_t n,
                                    const int32_t* order, double* out, unsigned int* error_word, void* stream) {
    if (n == 0) return CT_OK;
    launch_clip_area(nullptr, va, fa, Ka, vb, fb, Kb, ia, ib, n, order, out, error_word, (cudaStream_t)stream);
    CT_CHECK_LAUNCH("area_of_intersection");
    return CT_OK;
}

int ct_area_of_intersection(const double* va, const int64_t* fa, int32_t Ka, const double* vb, const int64_t* fb,
                            int32_t Kb, const int64_t* ia, const int64_t* ib, int64_t n, double* out,
                            unsigned int* error_word, void* stream) {
    return ct_area_of_intersection_ordered(va, fa, Ka, vb, fb, Kb, ia, ib, n, nullptr, out, error_word, stream);
}

int ct_box_area_of_intersection_ordered(const double* boxes, const double* vb, const int64_t* fb, int32_t Kb,
                                        const int64_t* ibox, const int64_t* iface, int64_t n, const int32_t* order,
                                        double* out, unsigned int* error_word, void* stream) {
    if (n == 0) return CT_OK;
    launch_clip_area((const double4*)boxes, nullptr, nullptr, 4, vb, fb, Kb, ibox, iface, n, order, out, error_word,
                     (cudaStream_t)stream);
    CT_CHECK_LAUNCH("box_area_of_intersection");
    return CT_OK;
}

int ct_box_area_of_intersection(const double* boxes, const double* vb, const int64_t* fb, int32_t Kb,
                                const int64_t* ibox, const int64_t* iface, int64_t n, double* out,
                                unsigned int* error_word, void* stream) {
    return ct_box_area_of_intersection_ordered(boxes, vb, fb, Kb, ibox, iface, n, nullptr, out, error_word, stream);
}

size_t ct_pair_order_workspace_size(int64_t n) {
    size_t part = ((size_t)(n > 0 ? n : 1) * sizeof(unsigned) + 255) / 256 * 256;
    return 2 * part + ct_radix_pass_workspace_size();
}

int ct_pair_order(const int64_t* fa, int32_t Ka, const int64_t* ia, const int64_t* fb, int32_t Kb, const int64_t* ib,
                  int64_t n, int32_t* order, void* ws, size_t ws_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 0 || n > INT32_MAX) return ct_fail(CT_ERR_ARG, "pair count out of range");
    if (!ws || ws_bytes < ct_pair_order_workspace_size(n)) return ct_fail(CT_ERR_WORKSPACE, "pair order workspace");
    if (n == 0) return CT_OK;
    size_t part = ((size_t)n * sizeof(unsigned) + 255) / 256 * 256;
    unsigned* kin = (unsigned*)ws;
    unsigned* kout = (unsigned*)((char*)ws + part);
    k_pair_keys<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 8), 256, 0, st>>>(fa, Ka, ia, fb, Kb, ib, n, kin);
    CT_CHECK_LAUNCH("pair keys");
    return ct_radix_pass(kin, nullptr, n, 0, kout, order, (char*)ws + 2 * part, ws_bytes - 2 * part, stream);
}

int ct_box_pair_order(const int64_t* fb, int32_t Kb, int64_t n_faces, const int64_t* ib, const uint8_t* inside,
                      int64_t n, int32_t* order, void* ws, size_t ws_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 0 || n > INT32_MAX || n_faces < 0) return ct_fail(CT_ERR_ARG, "pair or face count out of range");
    if (!ws || ws_bytes < ct_box_pair_order_workspace_size(n, n_faces))
        return ct_fail(CT_ERR_WORKSPACE, "pair order workspace");
    if (n == 0) return CT_OK;
    size_t part = ((size_t)n * sizeof(unsigned) + 255) / 256 * 256, lens = ((size_t)n_faces + 255) / 256 * 256;
    uint8_t* length = (uint8_t*)ws;
    unsigned* kin = (unsigned*)((char*)ws + lens);
    unsigned* kout = (unsigned*)((char*)kin + part);
    char* rest = (char*)kout + part;
    k_face_lengths<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(grid_of(n_faces, 256), 152 * 32)), 256, 0, st>>>(
        fb, Kb, n_faces, length);
    k_box_pair_keys<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 8), 256, 0, st>>>(length, ib, inside, n, kin);
    CT_CHECK_LAUNCH("pair keys");
    return ct_radix_pass(kin, nullptr, n, 0, kout, order, rest, ws_bytes - (size_t)(rest - (char*)ws), stream);
}

size_t ct_box_pair_order_workspace_size(int64_t n, int64_t n_faces) {
    return ct_pair_order_workspace_size(n) + ((size_t)(n_faces > 0 ? n_faces : 1) + 255) / 256 * 256;
}

int ct_compact_pairs(const double* area, const uint8_t* flag, int64_t n, const int64_t* ii, const int64_t* jj,
                     int64_t* ii_out, int64_t* jj_out, double* area_out, void* ws, size_t ws_bytes,
                     int64_t* total_host, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n == 0) {
        if (total_host) *total_host = 0;
        return CT_OK;
    }
    if (!ws || ws_bytes < ct_compact_workspace_size(n))
        return ct_fail(CT_ERR_WORKSPACE, "compaction workspace too small");
    const int64_t tiles = (n + KEEP_TILE - 1) / KEEP_TILE;
    int64_t* sums = (int64_t*)ws;
    k_keep_count<<<(unsigned)tiles, KEEP_T, 0, st>>>(area, flag, n, sums);
    const bool scan = tiles > KEEP_DIRECT;
    if (scan) k_scan_sums<<<1, SCAN_T, 0, st>>>(sums, tiles);
    k_compact<<<(unsigned)tiles, KEEP_T, 0, st>>>(area, flag, n, sums, scan, ii, jj, ii_out, jj_out, area_out,
                                                 sums + tiles);
    CT_CHECK_LAUNCH("compact");
    if (total_host) {
        CT_CUDA(cudaMemcpyAsync(total_host, sums + tiles, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        CT_CUDA(cudaStreamSynchronize(st));
    }
    return CT_OK;
}

size_t ct_compact_workspace_size(int64_t n) {
    return (size_t)((n > 0 ? n : 1) / KEEP_TILE + 2) * sizeof(int64_t);
}

int ct_barycentric_weights(const ct_tree* t, const double* points, const int64_t* face_indices, int64_t n,
                           double tolerance, double* weights, void* stream) {
    if (!t) return ct_fail(CT_ERR_ARG, "tree is null");
    if (n == 0) return CT_OK;
    int K = t->n_max_vert;
    int KW = K > 3 ? K : 3;
    const unsigned grid = grid_of(n, 128);
    cudaStream_t st = (cudaStream_t)stream;
    const double2 *P = (const double2*)points, *V = (const double2*)t->vertices;
    // faces of up to 8 vertices held in registers; longer ones in local memory
    const float tolf = (float)fmax(fabs(tolerance), 1e-37);
    if (K < 3 || K > 8 || ((uintptr_t)V & 15))
        k_barycentric<<<grid, 128, 0, st>>>(P, face_indices, n, t->vertices, t->elements, K, KW, tolerance, weights);
    else if (K == 3)
        k_barycentric_tri<<<grid, 128, 0, st>>>(P, face_indices, n, V, t->elements, tolerance, weights);
    else if (K == 4)
        k_barycentric_small<4><<<grid, 128, 0, st>>>(P, face_indices, n, V, t->elements, K, tolerance, tolf, weights);
    else
        k_barycentric_small<8><<<grid, 128, 0, st>>>(P, face_indices, n, V, t->elements, K, tolerance, tolf, weights);
    CT_CHECK_LAUNCH("barycentric");
    return CT_OK;
}

int ct_node_bounds(const int64_t* child, const double* Lmax, const double* Rmin, const uint8_t* dim, int64_t n_nodes,
                   const double* bbox_host4, int64_t* parent_ws, double* out, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n_nodes <= 0) return CT_OK;
    CT_CUDA(cudaMemsetAsync(parent_ws, 0xff, sizeof(int64_t) * n_nodes, st));
    k_parents<<<grid_of(n_nodes, 256), 256, 0, st>>>(child, n_nodes, parent_ws);
    double4 b = make_double4(bbox_host4[0], bbox_host4[1], bbox_host4[2], bbox_host4[3]);
    k_node_bounds<<<grid_of(n_nodes, 256), 256, 0, st>>>(child, Lmax, Rmin, dim, parent_ws, n_nodes, b,
                                                          (double4*)out);
    CT_CHECK_LAUNCH("node_bounds");
    return CT_OK;
}

int ct_validate_node_bounds(const int64_t* child, const int64_t* ptr, const int64_t* size, int64_t n_nodes,
                            const int64_t* bb_indices, const double* bb_coords, const double* node_bounds,
                            uint8_t* valid, void* stream) {
    if (n_nodes <= 0) return CT_OK;
    k_validate_bounds<<<grid_of(n_nodes, 256), 256, 0, (cudaStream_t)stream>>>(
        child, ptr, size, bb_indices, bb_coords, (const double4*)node_bounds, n_nodes, valid);
    CT_CHECK_LAUNCH("validate_node_bounds");
    return CT_OK;
}

size_t ct_work_order_workspace_size(int64_t n) {
    size_t nn = (size_t)(n > 0 ? n : 1);
    return 2 * ((4 * nn + 255) / 256 * 256) + ct_radix_pass_workspace_size();
}

int ct_work_order(const double* queries, int64_t n, int32_t kind, double cell_size, int32_t* order, void* ws,
                  size_t ws_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 0 || (kind != 0 && kind != 1)) return ct_fail(CT_ERR_ARG, "bad work-order arguments");
    if (!ws || ws_bytes < ct_work_order_workspace_size(n)) return ct_fail(CT_ERR_WORKSPACE, "workspace too small");
    if (n == 0) return CT_OK;
    size_t part = (4 * (size_t)n + 255) / 256 * 256;
    unsigned* kin = (unsigned*)ws;
    unsigned* kout = (unsigned*)((char*)ws + part);
    unsigned blocks = (unsigned)std::min<int64_t>((n + 255) / 256, 152 * 16);
    k_work_keys<<<blocks, 256, 0, st>>>((const double4*)queries, n, kind, (float)cell_size, kin);
    CT_CHECK_LAUNCH("work keys");
    return ct_radix_pass(kin, nullptr, n, 0, kout, order, (char*)ws + 2 * part, ws_bytes - 2 * part, stream);
}

int ct_count_edge_candidates(const ct_tree* t, int32_t mode, const double* segs, int64_t n, const int32_t* order,
                              int64_t* counts, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (mode == 0 && t->n_max_vert != 2) return ct_fail(CT_ERR_ARG, "edge-edge mode needs an edge tree");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const int et = seg_threads(t);
    const double4* S = (const double4*)segs;
    const unsigned g = grid_of(n, et);
    if (deep_tree(t)) {
        if (mode == 0) k_edge_cands_deep<false, 0><<<g, et, 0, st>>>(T, S, n, order, counts, 0, 0);
        else k_edge_cands_deep<false, 1><<<g, et, 0, st>>>(T, S, n, order, counts, 0, 0);
    } else {
        launch_edge_walk<false, false>(mode, T, S, n, order, nullptr, nullptr, 0, counts, nullptr, nullptr, 0,
                                       nullptr, st);
    }
    CT_CHECK_LAUNCH("count_edge_candidates");
    return CT_OK;
}

int ct_write_edge_candidates(const ct_tree* t, int32_t mode, const double* segs, int64_t n, const int32_t* order,
                              const int64_t* offsets, int32_t* cand_seg, int32_t* cand_pos, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (n > INT32_MAX) return ct_fail(CT_ERR_ARG, "at most 2^31 - 1 segments");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const int et = seg_threads(t);
    const double4* S = (const double4*)segs;
    const unsigned g = grid_of(n, et);
    int64_t* off = (int64_t*)offsets;
    if (deep_tree(t)) {
        if (mode == 0) k_edge_cands_deep<true, 0><<<g, et, 0, st>>>(T, S, n, order, off, cand_seg, cand_pos);
        else k_edge_cands_deep<true, 1><<<g, et, 0, st>>>(T, S, n, order, off, cand_seg, cand_pos);
    } else {
        launch_edge_walk<false, true>(mode, T, S, n, order, nullptr, nullptr, 0, off, cand_seg, cand_pos, 0, nullptr,
                                      st);
    }
    CT_CHECK_LAUNCH("write_edge_candidates");
    return CT_OK;
}

static int check_split(const ct_tree* t, int32_t mode, int32_t cut) {
    int s = check_tree(t);
    if (s) return s;
    if (mode != 0 && mode != 1) return ct_fail(CT_ERR_ARG, "mode must be 0 or 1");
    if (mode == 0 && t->n_max_vert != 2) return ct_fail(CT_ERR_ARG, "edge-edge mode needs an edge tree");
    if (cut < 0 || cut > 64) return ct_fail(CT_ERR_ARG, "cut depth must be in [0, 64]");
    if (deep_tree(t)) return ct_fail(CT_ERR_ARG, "tree too deep for the split traversal");
    return CT_OK;
}

int ct_count_edge_items(const ct_tree* t, int32_t mode, const double* segs, int64_t n, const int32_t* order,
                        int32_t cut, int64_t* counts, void* stream) {
    int s = check_split(t, mode, cut);
    if (s) return s;
    if (n == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const double4* S = (const double4*)segs;
    launch_edge_walk<true, false>(mode, T, S, n, order, nullptr, nullptr, cut, counts, nullptr, nullptr, 0, nullptr,
                                  st);
    CT_CHECK_LAUNCH("count_edge_items");
    return CT_OK;
}

int ct_write_edge_items(const ct_tree* t, int32_t mode, const double* segs, int64_t n, const int32_t* order,
                        int32_t cut, const int64_t* offsets, int32_t* item_seg, int32_t* item_node, void* stream) {
    int s = check_split(t, mode, cut);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (n > INT32_MAX) return ct_fail(CT_ERR_ARG, "at most 2^31 - 1 segments");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const double4* S = (const double4*)segs;
    int64_t* off = (int64_t*)offsets;
    launch_edge_walk<true, true>(mode, T, S, n, order, nullptr, nullptr, cut, off, item_seg, item_node, 0, nullptr,
                                 st);
    CT_CHECK_LAUNCH("write_edge_items");
    return CT_OK;
}

int ct_count_item_candidates(const ct_tree* t, int32_t mode, const double* segs, const int32_t* item_seg,
                             const int32_t* item_node, int64_t n_items, int64_t* counts, void* stream) {
    int s = check_split(t, mode, 0);
    if (s) return s;
    if (n_items == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const double4* S = (const double4*)segs;
    launch_edge_walk<false, false>(mode, T, S, n_items, nullptr, item_seg, item_node, 0, counts, nullptr, nullptr, 0,
                                   nullptr, st);
    CT_CHECK_LAUNCH("count_item_candidates");
    return CT_OK;
}

int ct_write_item_candidates(const ct_tree* t, int32_t mode, const double* segs, const int32_t* item_seg,
                             const int32_t* item_node, int64_t n_items, const int64_t* offsets, int32_t* cand_seg,
                             int32_t* cand_pos, void* stream) {
    int s = check_split(t, mode, 0);
    if (s) return s;
    if (n_items == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const double4* S = (const double4*)segs;
    int64_t* off = (int64_t*)offsets;
    launch_edge_walk<false, true>(mode, T, S, n_items, nullptr, item_seg, item_node, 0, off, cand_seg, cand_pos, 0,
                                  nullptr, st);
    CT_CHECK_LAUNCH("write_item_candidates");
    return CT_OK;
}

int ct_count_item_candidates_spec(const ct_tree* t, int32_t mode, const double* segs, const int32_t* item_seg,
                                  const int32_t* item_node, int64_t n_items, int64_t* counts, int32_t* spec,
                                  int32_t spec_cap, void* stream) {
    int s = check_split(t, mode, 0);
    if (s) return s;
    if (n_items == 0) return CT_OK;
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    launch_edge_walk<false, false>(mode, make_q(t), (const double4*)segs, n_items, nullptr, item_seg, item_node, 0,
                                   counts, nullptr, spec, spec_cap, nullptr, (cudaStream_t)stream);
    CT_CHECK_LAUNCH("count_item_candidates_spec");
    return CT_OK;
}

int ct_write_item_candidates_spec(const ct_tree* t, int32_t mode, const double* segs, const int32_t* item_seg,
                                  const int32_t* item_node, int64_t n_items, const int64_t* counts,
                                  const int64_t* offsets, const int32_t* spec, int32_t spec_cap, int32_t* cand_seg,
                                  int32_t* cand_pos, void* stream) {
    int s = check_split(t, mode, 0);
    if (s) return s;
    if (n_items == 0) return CT_OK;
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    cudaStream_t st = (cudaStream_t)stream;
    k_edge_spec_emit<<<(unsigned)std::min<int64_t>(grid_of(16 * n_items, 256), 152 * 64), 256, 0, st>>>(
        counts, offsets, n_items, item_seg, spec, spec_cap, cand_seg, cand_pos);
    launch_edge_walk<false, true>(mode, make_q(t), (const double4*)segs, n_items, nullptr, item_seg, item_node, 0,
                                  (int64_t*)offsets, cand_seg, cand_pos, spec_cap, counts, st);
    CT_CHECK_LAUNCH("write_item_candidates_spec");
    return CT_OK;
}

int ct_segment_candidate_ranges(const int64_t* item_off, const int64_t* item_cnt, int64_t n,
                                const int64_t* item_cand_off, const int64_t* item_cand_cnt, int64_t n_items,
                                int64_t* cand_off, int64_t* cand_cnt, void* stream) {
    if (n < 0 || n_items < 0) return ct_fail(CT_ERR_ARG, "negative count");
    if (n == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    k_seg_from_items<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 32), 256, 0, st>>>(
        item_off, item_cnt, n, item_cand_off, item_cand_cnt, n_items, cand_off, cand_cnt);
    CT_CHECK_LAUNCH("segment_candidate_ranges");
    return CT_OK;
}

int ct_count_edge_candidates_spec(const ct_tree* t, int32_t mode, const double* segs, int64_t n,
                                  const int32_t* order, int64_t* counts, int32_t* spec, int32_t spec_cap,
                                  void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (mode != 0 && mode != 1) return ct_fail(CT_ERR_ARG, "mode must be 0 or 1");
    if (mode == 0 && t->n_max_vert != 2) return ct_fail(CT_ERR_ARG, "edge-edge mode needs an edge tree");
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    const int et = seg_threads(t);
    const double4* S = (const double4*)segs;
    const unsigned g = grid_of(n, et);
    if (deep_tree(t)) {
        if (mode == 0) k_edge_cands_deep<false, 0><<<g, et, 0, st>>>(T, S, n, order, counts, 0, spec, spec_cap);
        else k_edge_cands_deep<false, 1><<<g, et, 0, st>>>(T, S, n, order, counts, 0, spec, spec_cap);
    } else {
        launch_edge_walk<false, false>(mode, T, S, n, order, nullptr, nullptr, 0, counts, nullptr, spec, spec_cap,
                                       nullptr, st);
    }
    CT_CHECK_LAUNCH("count_edge_candidates_spec");
    return CT_OK;
}

int ct_write_edge_candidates_spec(const ct_tree* t, int32_t mode, const double* segs, int64_t n,
                                  const int32_t* order, const int64_t* counts, const int64_t* offsets,
                                  const int32_t* spec, int32_t spec_cap, int32_t* cand_seg, int32_t* cand_pos,
                                  void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n == 0) return CT_OK;
    if (n > INT32_MAX) return ct_fail(CT_ERR_ARG, "at most 2^31 - 1 segments");
    if (mode != 0 && mode != 1) return ct_fail(CT_ERR_ARG, "mode must be 0 or 1");
    if (!spec || spec_cap < 1 || spec_cap > 4096) return ct_fail(CT_ERR_ARG, "spec_cap must be in [1, 4096]");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    k_edge_spec_emit<<<(unsigned)std::min<int64_t>(grid_of(16 * n, 256), 152 * 64), 256, 0, st>>>(
        counts, offsets, n, nullptr, spec, spec_cap, cand_seg, cand_pos);
    const int et = seg_threads(t);
    const double4* S = (const double4*)segs;
    const unsigned g = grid_of(n, et);
    int64_t* off = (int64_t*)offsets;
    if (deep_tree(t)) {
        if (mode == 0)
            k_edge_cands_deep<true, 0><<<g, et, 0, st>>>(T, S, n, order, off, cand_seg, cand_pos, spec_cap, counts);
        else
            k_edge_cands_deep<true, 1><<<g, et, 0, st>>>(T, S, n, order, off, cand_seg, cand_pos, spec_cap, counts);
    } else {
        launch_edge_walk<false, true>(mode, T, S, n, order, nullptr, nullptr, 0, off, cand_seg, cand_pos, spec_cap,
                                      counts, st);
    }
    CT_CHECK_LAUNCH("write_edge_candidates_spec");
    return CT_OK;
}

int ct_cs_certificates(const ct_tree* t, const double* segs, const int32_t* cand_seg, const int32_t* cand_pos,
                       int64_t n_cand, int8_t* out, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n_cand == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    k_cs_certificates<<<(unsigned)std::min<int64_t>(grid_of(n_cand, 128), 152 * 64), 128, 0, st>>>(
        make_q(t), (const double4*)segs, cand_seg, cand_pos, n_cand, out);
    CT_CHECK_LAUNCH("cs_certificates");
    return CT_OK;
}

int ct_test_edge_candidates(const ct_tree* t, int32_t mode, const double* segs, const int32_t* cand_seg,
                            const int32_t* cand_pos, int64_t n_cand, int64_t* keep, double* xy, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n_cand == 0) return CT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    unsigned g = (unsigned)std::min<int64_t>(grid_of(n_cand, 128), 152 * 64);
    if (mode == 0)
        k_edge_test<0, int64_t><<<g, 128, 0, st>>>(T, (const double4*)segs, cand_seg, cand_pos, n_cand, keep,
                                                   (double4*)xy);
    else
        k_edge_test<1, int64_t><<<g, 128, 0, st>>>(T, (const double4*)segs, cand_seg, cand_pos, n_cand, keep,
                                                   (double4*)xy);
    CT_CHECK_LAUNCH("test_edge_candidates");
    return CT_OK;
}

int ct_compact_edge_hits(const ct_tree* t, const int64_t* keep, const int64_t* pos, int64_t n_cand,
                         const int32_t* cand_seg, const int32_t* cand_pos, const double* xy_cand,
                         const int64_t* cand_off, const int64_t* cand_cnt, int64_t n, int64_t* ii, int64_t* jj,
                         double* xy, int64_t* offsets, int64_t* counts, void* stream) {
    if (!t) return ct_fail(CT_ERR_ARG, "tree is null");
    cudaStream_t st = (cudaStream_t)stream;
    if (n_cand > 0)
        k_edge_compact<<<(unsigned)std::min<int64_t>(grid_of(n_cand, 256), 152 * 32), 256, 0, st>>>(
            keep, pos, n_cand, cand_seg, cand_pos, t->bb_indices, (const double4*)xy_cand, ii, jj, (double4*)xy);
    if (n > 0)
        k_edge_seg_counts<<<(unsigned)std::min<int64_t>(grid_of(n, 256), 152 * 32), 256, 0, st>>>(
            cand_off, cand_cnt, keep, pos, n_cand, n, offsets, counts);
    CT_CHECK_LAUNCH("compact_edge_hits");
    return CT_OK;
}

size_t ct_spatial_order_workspace_size(int64_t n) {
    size_t nn = (size_t)(n > 0 ? n : 1);
    return 3 * ((4 * nn + 255) / 256 * 256) + ct_radix_pass_workspace_size();
}

int ct_spatial_order(const double* queries, int64_t n, int32_t kind, const double* bbox_host4, int32_t* order,
                     void* ws, size_t ws_bytes, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 0 || n > INT32_MAX || (kind != 0 && kind != 1) || !bbox_host4)
        return ct_fail(CT_ERR_ARG, "bad spatial-order arguments");
    if (!ws || ws_bytes < ct_spatial_order_workspace_size(n)) return ct_fail(CT_ERR_WORKSPACE, "workspace too small");
    if (n == 0) return CT_OK;
    const size_t part = (4 * (size_t)n + 255) / 256 * 256;
    unsigned* kin = (unsigned*)ws;
    unsigned* kout = (unsigned*)((char*)ws + part);
    int* iout = (int*)((char*)ws + 2 * part);
    void* rws = (char*)ws + 3 * part;
    const double ex = bbox_host4[1] - bbox_host4[0], ey = bbox_host4[3] - bbox_host4[2];
    const float sx = ex > 0.0 ? (float)(256.0 / ex) : 0.0f, sy = ey > 0.0 ? (float)(256.0 / ey) : 0.0f;
    const unsigned blocks = (unsigned)std::min<int64_t>((n + 255) / 256, 152 * 16);
    k_spatial_keys<<<blocks, 256, 0, st>>>((const double4*)queries, n, kind, bbox_host4[0], bbox_host4[2], sx, sy,
                                           kin);
    CT_CHECK_LAUNCH("spatial keys");
    int s = ct_radix_pass(kin, nullptr, n, 0, kout, iout, rws, ws_bytes - 3 * part, stream);
    if (s) return s;
    return ct_radix_pass(kout, iout, n, 8, kin, order, rws, ws_bytes - 3 * part, stream);
}

int ct_gather_rows(const double* queries, const int32_t* order, int64_t n, double* out, void* stream) {
    if (n <= 0) return CT_OK;
    k_gather_rows<<<(unsigned)std::min<int64_t>((n + 255) / 256, 152 * 16), 256, 0, (cudaStream_t)stream>>>(
        (const double4*)queries, order, n, (double4*)out);
    CT_CHECK_LAUNCH("gather rows");
    return CT_OK;
}

int ct_test_edge_candidates_u8(const ct_tree* t, int32_t mode, const double* segs, const int32_t* cand_seg,
                               const int32_t* cand_pos, int64_t n_cand, uint8_t* keep, double* xy, void* stream) {
    int s = check_tree(t);
    if (s) return s;
    if (n_cand == 0) return CT_OK;
    if (mode != 0 && mode != 1) return ct_fail(CT_ERR_ARG, "mode must be 0 or 1");
    cudaStream_t st = (cudaStream_t)stream;
    TreeQ T = make_q(t);
    unsigned g = (unsigned)std::min<int64_t>(grid_of(n_cand, 128), 152 * 64);
    if (mode == 0)
        k_edge_test<0, uint8_t><<<g, 128, 0, st>>>(T, (const double4*)segs, cand_seg, cand_pos, n_cand, keep,
                                                   (double4*)xy);
    else
        k_edge_test<1, uint8_t><<<g, 128, 0, st>>>(T, (const double4*)segs, cand_seg, cand_pos, n_cand, keep,
                                                   (double4*)xy);
    CT_CHECK_LAUNCH("test_edge_candidates");
    return CT_OK;
}

size_t ct_edge_hit_counts_workspace_size(int64_t n) { return ct_scan_workspace_size(n) + 256; }

int ct_edge_hit_counts(const uint8_t* keep, const int64_t* cand_off, const int64_t* cand_cnt, const int32_t* order,
                       int64_t n, int64_t* counts, int64_t* offsets, void* ws, size_t ws_bytes, int64_t* total_host,
                       int64_t* longest_host, void* stream) {
    if (n < 0) return ct_fail(CT_ERR_ARG, "negative length");
    if (!ws || ws_bytes < ct_edge_hit_counts_workspace_size(n)) return ct_fail(CT_ERR_WORKSPACE, "workspace too small");
    if (!total_host || !longest_host) return ct_fail(CT_ERR_ARG, "no host results");
    cudaStream_t st = (cudaStream_t)stream;
    // block sums, the total behind them, and the longest behind that: one copy
    const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    int64_t* sums = (int64_t*)ws;
    CT_CUDA(cudaMemsetAsync(sums + nb, 0, 2 * sizeof(int64_t), st));
    if (n > 0) {
        k_hit_counts<<<(unsigned)std::min<int64_t>(grid_of(n, 32), 152 * 16), 256, 0, st>>>(
            keep, cand_off, cand_cnt, order, n, counts, (unsigned long long*)(sums + nb + 1));
        k_scan_reduce<<<(unsigned)nb, SCAN_T, 0, st>>>(counts, n, sums);
        k_scan_sums<<<1, SCAN_T, 0, st>>>(sums, nb);
        k_scan_down<<<(unsigned)nb, SCAN_T, 0, st>>>(counts, n, sums, offsets);
    }
    CT_CHECK_LAUNCH("edge_hit_counts");
    int64_t got[2] = {0, 0};
    CT_CUDA(cudaMemcpyAsync(got, sums + nb, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CT_CUDA(cudaStreamSynchronize(st));
    *total_host = got[0];
    *longest_host = got[1];
    return CT_OK;
}

size_t ct_finish_edge_hits_workspace_size(int64_t total, int64_t longest) {
    const size_t t = (size_t)(total > 0 ? total : 1);
    const size_t lists = ((t / (WARP_SORT_MAX + 1) + 2) * sizeof(int) + 256 + 255) / 256 * 256;
    return lists + (longest > FIN_SMEM ? t * 2 * (sizeof(unsigned long long) + sizeof(unsigned)) + 256 : 0);
}

int ct_finish_edge_hits(const ct_tree* t, const double* segs, const int32_t* order, const uint8_t* keep,
                        const int32_t* cand_pos, const double* xy_cand, const int64_t* cand_off,
                        const int64_t* cand_cnt, int64_t n, const int64_t* counts, const int64_t* offsets,
                        int64_t total, int64_t longest, int64_t* ii, int64_t* jj, double* xy, void* ws,
                        size_t ws_bytes, void* stream) {
    if (!t) return ct_fail(CT_ERR_ARG, "tree is null");
    if (n < 0 || n > INT32_MAX) return ct_fail(CT_ERR_ARG, "at most 2^31 - 1 segments");
    if (total == 0 || n == 0) return CT_OK;
    if (!ws || ws_bytes < ct_finish_edge_hits_workspace_size(total, longest))
        return ct_fail(CT_ERR_WORKSPACE, "finish workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* nlist = (unsigned long long*)ws;
    int* list = (int*)(nlist + 1);
    const size_t lists = (((size_t)total / (WARP_SORT_MAX + 1) + 2) * sizeof(int) + 256 + 255) / 256 * 256;
    unsigned long long* gk = (unsigned long long*)((char*)ws + lists);
    unsigned* gx = (unsigned*)(gk + 2 * total);
    const HitSort H{(const double4*)segs, order, keep, cand_pos, t->bb_indices, (const double4*)xy_cand, cand_off,
                    cand_cnt, counts, offsets, ii, jj, (double4*)xy};
    CT_CUDA(cudaMemsetAsync(nlist, 0, sizeof(unsigned long long), st));
    k_finish_warp<<<(unsigned)std::min<int64_t>(grid_of(n, 8), 152 * 32), 256, 0, st>>>(H, n, list, nlist);
    if (longest > WARP_SORT_MAX) k_finish_block<<<152 * 8, FIN_T, 0, st>>>(H, list, nlist, total, gk, gx);
    CT_CHECK_LAUNCH("finish_edge_hits");
    return CT_OK;
}

}  // extern "C"
