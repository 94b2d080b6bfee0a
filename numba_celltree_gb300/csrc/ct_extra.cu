// ct_extra.cu -- the two exported helpers that no query calls
// (liang_barsky_line_box_clip algorithms/liang_barsky.py:10-64,
// points_in_triangles geometry_utils.py:273-289), batched, and the step right
// after the intersection queries in regridding: a CSR weight matrix from the
// query-major (row, column, area) pairs of intersect_faces / intersect_boxes
// and its area-weighted mean (the dense weight-matrix aggregation of
// examples/spatial_indexing_2d_grids.py:245-313, done sparse).
#include <cmath>
#include <cstdint>

#include "ct_common.cuh"
#include "ct_internal.h"
#include "ct_sf64.cuh"

namespace cte {

// point_inside_box geometry_utils.py:528-529 (strict)
__device__ __forceinline__ bool inside_box(dpt a, double xmin, double xmax, double ymin, double ymax) {
    return xmin < a.x && a.x < xmax && ymin < a.y && a.y < ymax;
}

// liang_barsky_line_box_clip liang_barsky.py:10-64
__device__ bool liang_barsky(dpt a, dpt b, double xmin, double xmax, double ymin, double ymax, dpt* c, dpt* d) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    *c = mkp(nan, nan);
    *d = mkp(nan, nan);
    double dx = b.x - a.x, dy = b.y - a.y;
    if (dx == 0.0 && dy == 0.0) return false;
    if (inside_box(a, xmin, xmax, ymin, ymax) && inside_box(b, xmin, xmax, ymin, ymax)) {
        *c = a;
        *d = b;
        return true;
    }
    double t0 = 0.0, t1 = 1.0;
    const double P[4] = {-dx, dx, -dy, dy};
    const double Q[4] = {a.x - xmin, xmax - a.x, a.y - ymin, ymax - a.y};
    for (int k = 0; k < 4; k++) {
        double p = P[k], q = Q[k];
        if (p == 0) {
            if (q < 0) return false;
        } else {
            double t = q / p;
            if (p < 0) {
                if (t > t1) return false;
                if (t > t0) t0 = t;
            } else if (p > 0) {
                if (t < t0) return false;
                if (t < t1) t1 = t;
            }
        }
    }
    if (t0 == t1) return false;
    *c = mkp(a.x + t0 * dx, a.y + t0 * dy);
    *d = mkp(a.x + t1 * dx, a.y + t1 * dy);
    return true;
}

// point_in_triangle geometry_utils.py:241-270
__device__ bool point_in_triangle(dpt p, dpt a, dpt b, dpt c, double tol) {
    dpt ap = vsub(p, a), bp = vsub(p, b), cp = vsub(p, c);
    dpt ab = vsub(b, a), bc = vsub(c, b), ca = vsub(a, c);
    double A = crossp(ab, ap), B = crossp(bc, bp), C = crossp(ca, cp);
    bool sA = A > 0, sB = B > 0, sC = C > 0;
    if ((sA == sB) && (sB == sC)) return true;
    return (within_perp(A, ab, tol) && in_bounds(p, a, b)) || (within_perp(B, bc, tol) && in_bounds(p, b, c)) ||
           (within_perp(C, ca, tol) && in_bounds(p, c, a));
}

__global__ void k_liang_barsky(const double2* __restrict__ a, const double2* __restrict__ b,
                               const double4* __restrict__ box, int64_t n, uint8_t* __restrict__ ok,
                               double2* __restrict__ c, double2* __restrict__ d) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double4 bx = box[i];
        dpt cc, dd;
        bool r = liang_barsky(mkp(a[i].x, a[i].y), mkp(b[i].x, b[i].y), bx.x, bx.y, bx.z, bx.w, &cc, &dd);
        ok[i] = (uint8_t)r;
        c[i] = make_double2(cc.x, cc.y);
        d[i] = make_double2(dd.x, dd.y);
    }
}

__global__ void k_points_in_triangles(const double2* __restrict__ pts, const int64_t* __restrict__ fidx, int64_t n,
                                      const int64_t* __restrict__ faces, int K, const double* __restrict__ v,
                                      int64_t n_faces, double tol, uint8_t* __restrict__ out,
                                      unsigned int* __restrict__ bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t f = fidx[i];
        if (f < 0 || f >= n_faces) {  // upstream indexes without a check
            atomicOr(bad, 1u);
            out[i] = 0;
            continue;
        }
        const int64_t* t = faces + f * K;
        dpt A = mkp(v[2 * t[0]], v[2 * t[0] + 1]), B = mkp(v[2 * t[1]], v[2 * t[1] + 1]);
        dpt C = mkp(v[2 * t[2]], v[2 * t[2] + 1]);
        out[i] = (uint8_t)point_in_triangle(mkp(pts[i].x, pts[i].y), A, B, C, tol);
    }
}

// Row indices must lie in [0, n_rows) and be non-decreasing (the pairs come
// query-major); one streaming pass checks both.
__global__ void k_rows_check(const int64_t* __restrict__ rows, int64_t n_pairs, int64_t n_rows,
                             unsigned int* __restrict__ bad) {
    unsigned int e = 0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_pairs;
         t += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = rows[t];
        if (r < 0 || r >= n_rows) e |= 1u;
        if (t > 0 && r < rows[t - 1]) e |= 2u;
    }
    if (e) atomicOr(bad, e);
}

// row_ptr[r] = first pair of a row >= r: a binary search per row.  The rows
// are sorted already, so nothing has to be counted: against an atomic count
// per pair and a scan the 91M pairs of 250k boxes take 0.16 instead of
// 1.2 ms, almost all of it the check above (bound by reading the rows once).
// Unsorted rows (reported by the check) still give values in [0, n_pairs].
__global__ void k_row_search(const int64_t* __restrict__ rows, int64_t n_pairs, int64_t n_rows,
                             int64_t* __restrict__ row_ptr) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > n_rows) return;
    int64_t lo = 0, hi = n_pairs;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (rows[mid] < r) lo = mid + 1;
        else hi = mid;
    }
    row_ptr[r] = r == n_rows ? n_pairs : lo;
}

// Sum of weights and of weight * x over each row's entries in entry order
// (lane-strided partial sums, then a fixed-order tree), mean =
// sum(w x) / sum(w), NaN for rows without weight.  The float64 unit (20 cycles
// per warp addition or product, 144 per division) bounds it: a warp per row
// spends 13 float64 instructions on a row of three entries.  So a warp takes
// `rpw` rows, those of up to 8 entries a lane each, all at once, the longer
// ones one after another on all lanes with four entries per lane loaded ahead.
// A short row's lane adds in the order of the tree over 32 lanes (whose other
// lanes hold zeros), and the long rows' two sums go down one tree, the upper
// half of the lanes taking over the second: the sums are the same bits.
// Products of long rows and all quotients run on the integer pipes.
// 1M rows of 3.4 entries: 282 -> 113 us against short rows on 8 lanes each and
// two trees; 250k rows of 280 entries 1.10 -> 1.07 ms.
constexpr int CSR_SHORT = 8;

// v[k] + v[k + o] for k < o, o = 4, 2, 1; entries above m are zeros (m, the
// longest of the warp's short rows, is the same in all lanes).  A sum that
// starts from 0.0 never is -0.0, so neither is this one.
__device__ __forceinline__ double csr_tree(double (&v)[CSR_SHORT], int m) {
    if (m > 4) {
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] += v[k + 4];
    }
    if (m > 2) {
        v[0] += v[2];
        v[1] += v[3];
    }
    const double sum = m > 1 ? v[0] + v[1] : v[0];
    return sf_zero(sum) ? 0.0 : sum;
}

__device__ __forceinline__ double csr_quotient(double a, double b) {
    bool bad = false;
    double q = sf_div(a, b, &bad);
    if (bad) q = a / b;
    return q;
}

__global__ void __launch_bounds__(256) k_csr_mean(const int64_t* __restrict__ row_ptr,
                                                  const int64_t* __restrict__ cols, const double* __restrict__ w,
                                                  int64_t n_rows, int64_t n_cols, const double* __restrict__ x,
                                                  double* __restrict__ mean, double* __restrict__ wsum_out,
                                                  unsigned int* __restrict__ bad, int rpw) {
    const unsigned FULL = 0xffffffffu;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    bool out_of_range = false;
    for (int64_t r0 = warp * rpw; r0 < n_rows; r0 += nw * rpw) {
        const bool have = lane < rpw && r0 + lane < n_rows;
        int64_t s = 0, e = 0;
        if (have) {
            s = row_ptr[r0 + lane];
            e = row_ptr[r0 + lane + 1];
        }
        {
            const int n = e - s <= CSR_SHORT ? (int)(e - s) : 0;
            const int m = __reduce_max_sync(FULL, n);
            double wk[CSR_SHORT], xk[CSR_SHORT];
#pragma unroll
            for (int k = 0; k < CSR_SHORT; k++) {
                wk[k] = xk[k] = 0.0;
                if (k < n) {
                    const int64_t c = cols[s + k];
                    if (c < 0 || c >= n_cols) {
                        out_of_range = true;
                    } else {
                        wk[k] = w[s + k];
                        xk[k] = x[c];
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < CSR_SHORT; k++)
                if (k < m) xk[k] = k < n ? wk[k] * xk[k] : 0.0;
            const double sw = csr_tree(wk, m), swx = csr_tree(xk, m);
            if (have && e - s <= CSR_SHORT) {
                mean[r0 + lane] = (sw > 0.0) ? csr_quotient(swx, sw) : nan;
                if (wsum_out) wsum_out[r0 + lane] = sw;
            }
        }
        for (unsigned left = __ballot_sync(FULL, e - s > CSR_SHORT); left; left &= left - 1) {
            const int row = __ffs(left) - 1;
            const int64_t rs = __shfl_sync(FULL, s, row), re = __shfl_sync(FULL, e, row);
            double sw = 0.0, swx = 0.0;
            for (int64_t k = rs + lane; k < re; k += 128) {
                int64_t c[4];
                double wk[4], xk[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int64_t ku = k + 32 * u;
                    c[u] = ku < re ? cols[ku] : 0;
                    wk[u] = ku < re ? w[ku] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) xk[u] = (c[u] >= 0 && c[u] < n_cols) ? x[c[u]] : 0.0;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (k + 32 * u >= re) break;
                    if (c[u] < 0 || c[u] >= n_cols) {
                        out_of_range = true;
                        continue;
                    }
                    bool odd = false;
                    double p = sf_mul(wk[u], xk[u], &odd);
                    if (odd) p = wk[u] * xk[u];
                    sw += wk[u];
                    swx += p;
                }
            }
            // lanes 0 .. 15 go on with the weights, 16 .. 31 with the products
            const double give = lane < 16 ? swx : sw, keep = lane < 16 ? sw : swx;
            double v = keep + __shfl_xor_sync(FULL, give, 16);
            for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o, 16);
            swx = __shfl_sync(FULL, v, 16);
            if (lane == 0) {
                mean[r0 + row] = (v > 0.0) ? csr_quotient(swx, v) : nan;
                if (wsum_out) wsum_out[r0 + row] = v;
            }
        }
    }
    if (out_of_range) atomicOr(bad, 1u);
}

static unsigned grid_for(int64_t n, int t) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + t - 1) / t, 152 * 16)); }

}  // namespace cte

using namespace cte;

extern "C" {

int ct_liang_barsky_line_box_clip(const double* a, const double* b, const double* boxes, int64_t n, uint8_t* ok,
                                  double* c, double* d, void* stream) {
    if (n < 0) return ct_fail(CT_ERR_ARG, "negative length");
    if (n == 0) return CT_OK;
    k_liang_barsky<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>((const double2*)a, (const double2*)b,
                                                                      (const double4*)boxes, n, ok, (double2*)c,
                                                                      (double2*)d);
    CT_CHECK_LAUNCH("liang_barsky");
    return CT_OK;
}

int ct_points_in_triangles(const double* points, const int64_t* face_indices, int64_t n, const int64_t* faces,
                           int32_t n_max_vert, int64_t n_faces, const double* vertices, double tolerance,
                           uint8_t* out, unsigned int* error_word, void* stream) {
    if (n < 0 || n_max_vert < 3) return ct_fail(CT_ERR_ARG, "bad sizes");
    if (n == 0) return CT_OK;
    k_points_in_triangles<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        (const double2*)points, face_indices, n, faces, n_max_vert, vertices, n_faces, tolerance, out, error_word);
    CT_CHECK_LAUNCH("points_in_triangles");
    return CT_OK;
}

size_t ct_csr_workspace_size(int64_t n_rows) {
    (void)n_rows;
    return 256;  // not used: an interface of callers
}

int ct_csr_row_ptr(const int64_t* rows, int64_t n_pairs, int64_t n_rows, int64_t* row_ptr, void* ws,
                   size_t ws_bytes, unsigned int* error_word, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n_pairs < 0 || n_rows < 0) return ct_fail(CT_ERR_ARG, "negative length");
    if (!ws || ws_bytes < ct_csr_workspace_size(n_rows)) return ct_fail(CT_ERR_WORKSPACE, "csr workspace too small");
    if (n_pairs > 0) {
        k_rows_check<<<grid_for(n_pairs, 256), 256, 0, st>>>(rows, n_pairs, n_rows, error_word);
        CT_CHECK_LAUNCH("csr check");
    }
    k_row_search<<<(unsigned)(n_rows / 256 + 1), 256, 0, st>>>(rows, n_pairs, n_rows, row_ptr);
    CT_CHECK_LAUNCH("csr rows");
    return CT_OK;
}

int ct_csr_weighted_mean(const int64_t* row_ptr, const int64_t* cols, const double* weights, int64_t n_rows,
                         int64_t n_cols, const double* x, double* mean, double* weight_sum, unsigned int* error_word,
                         void* stream) {
    if (n_rows < 0 || n_cols < 0) return ct_fail(CT_ERR_ARG, "negative length");
    if (n_rows == 0) return CT_OK;
    // rows per warp: as many as keep four tasks per resident warp (152 SMs x
    // 64 warps), so that long rows still balance
    int rpw = 32;
    while (rpw > 4 && n_rows / rpw < 152 * 64 * 4) rpw /= 2;
    const int64_t warps = (n_rows + rpw - 1) / rpw;
    unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, 152 * 32));
    k_csr_mean<<<blocks, 256, 0, (cudaStream_t)stream>>>(row_ptr, cols, weights, n_rows, n_cols, x, mean, weight_sum,
                                                         error_word, rpw);
    CT_CHECK_LAUNCH("csr weighted mean");
    return CT_OK;
}

}  // extern "C"
