// H restricted to one set of rows, materialised as a sparse matrix.
//
// The reference's Lanczos loops (qmb/rldiag.py:19-52, qmb/haar.py:107-183)
// call apply_within on the same rows once per iteration, so every iteration
// walks the whole term table again.  Here the rows are compared with each
// other, or their terms walked, twice in total (count the entries of every
// row, then fill them) and each iteration is a sparse matrix-vector product
// over the stored entries, which reads nnz x 20 bytes from HBM instead of
// walking T terms per row.
//
// Layout (CSR): row j holds, at [row_ptr[j], row_ptr[j + 1]), first the
// diagonal entry (column j, the sum of the diagonal terms, possibly zero),
// then one entry per (term, row i) pair that maps row i onto row j, with the
// sign-folded coefficient as value; pairs that reach the same (j, i) through
// different terms are separate entries.  Rows must be distinct.
#include <cuda_runtime.h>

#include "pairs.cuh"

namespace qmbx {
namespace {

// Grouped / tiled walks (warp or thread per walked row j, daggered terms):
// every hit is an entry (row j, column = the looked-up row).
template <int W, bool FILL>
struct MatrixRows : VisitorBase {
    HashView lookup;
    const double2* coef;     // adjoint part: stored coefficient, sign folded
    const int32_t* unique;   // walk index -> row
    int32_t* count;          // COUNT: off-diagonal entries per row
    int64_t* cursor;         // FILL: next free entry of each row
    int32_t* col;
    double2* val;
    struct Acc {
        int32_t row;
        int n;
    };
    static constexpr bool kBatched = true;
    __device__ __forceinline__ void init(Acc& a, int64_t u, const Key<W>&, int*) const {
        a.row = __ldg(unique + u);
        a.n = 0;
    }
    __device__ __forceinline__ bool probe(Acc&, const Key<W>&, const Key<W>& img, int parity, int64_t slot,
                                          int2& h) const {
        const int64_t pos = hash_find<W>(lookup, img);
        if (pos < 0) return false;
        h = make_int2((int)slot | (parity << 31), (int)pos);
        return true;
    }
    __device__ __forceinline__ void apply_hit(Acc& a, int2 h) const {
        if (!FILL) {
            ++a.n;
            return;
        }
        const double2 cf = __ldg(coef + (h.x & 0x7fffffff));
        const int64_t e = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(cursor + a.row), 1ull);
        col[e] = h.y;
        val[e] = h.x < 0 ? make_double2(-cf.x, -cf.y) : cf;
    }
    __device__ __forceinline__ void visit(Acc& a, const Key<W>& c, const Key<W>& img, int parity, int64_t slot) const {
        int2 h;
        if (probe(a, c, img, parity, slot, h)) apply_hit(a, h);
    }
    __device__ __forceinline__ void visit_diag(Acc&, const Key<W>&, int, int64_t) const {}
    __device__ __forceinline__ void reduce(Acc& a) const {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) a.n += __shfl_xor_sync(0xffffffffu, a.n, d);
    }
    __device__ __forceinline__ void finish(Acc& a, int64_t, const Key<W>&) const {
        if (!FILL) count[a.row] = a.n;
    }
};

// Pivot-major walk: hits carry their walked row; entries claimed with atomics.
template <int W, bool FILL>
struct MatrixPivot : VisitorBase {
    static constexpr bool kStateless = true;
    HashView lookup;
    const double2* coef;
    const int32_t* unique;
    int32_t* count;
    int64_t* cursor;
    int32_t* col;
    double2* val;
    struct Acc {};
    __device__ __forceinline__ bool probe_row(const Key<W>&, const Key<W>& img, int parity, int64_t slot, int64_t u,
                                              int4& h) const {
        const int64_t pos = hash_find<W>(lookup, img);
        if (pos < 0) return false;
        h = make_int4((int)slot | (parity << 31), (int)pos, (int)u, 0);
        return true;
    }
    __device__ __forceinline__ void apply_row_hit(int4 h) const {
        const int32_t row = __ldg(unique + h.z);
        if (!FILL) {
            atomicAdd(count + row, 1);
            return;
        }
        const double2 cf = __ldg(coef + (h.x & 0x7fffffff));
        const int64_t e = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(cursor + row), 1ull);
        col[e] = h.y;
        val[e] = h.x < 0 ? make_double2(-cf.x, -cf.y) : cf;
    }
};

// Pair scan: a hit is an entry in the row its term leads to.
template <bool FILL>
struct MatrixPairs {
    const double2* coef;     // forward part
    int32_t* count;
    int64_t* cursor;
    int32_t* col;
    double2* val;
    __device__ __forceinline__ bool recording() const { return false; }
    __device__ __forceinline__ void record(const int4*, int, int) const {}
    __device__ __forceinline__ void apply(int4 h) const {
        if (!FILL) {
            atomicAdd(count + h.z, 1);
            return;
        }
        const double2 cf = __ldg(coef + (h.x & 0x7fffffff));
        const int64_t e = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(cursor + h.z), 1ull);
        col[e] = h.y;
        val[e] = h.x < 0 ? make_double2(-cf.x, -cf.y) : cf;
    }
};

// The diagonal entry of every walked row (first entry of the row).
template <int W>
struct MatrixDiagonal : VisitorBase {
    const double2* dcoef;
    const int32_t* unique;
    const int64_t* row_ptr;
    int32_t* col;
    double2* val;
    struct Acc {
        double re, im;
    };
    __device__ __forceinline__ void init(Acc& a, int64_t, const Key<W>&, int*) const { a.re = a.im = 0.0; }
    __device__ __forceinline__ void visit(Acc&, const Key<W>&, const Key<W>&, int, int64_t) const {}
    __device__ __forceinline__ void visit_diag(Acc& a, const Key<W>&, int parity, int64_t slot) const {
        const double2 cf = __ldg(dcoef + slot);
        a.re += parity ? -cf.x : cf.x;
        a.im += parity ? -cf.y : cf.y;
    }
    __device__ __forceinline__ void reduce(Acc& a) const {
        a.re = warp_sum(a.re);
        a.im = warp_sum(a.im);
    }
    template <int L>
    __device__ __forceinline__ void reduce_lanes(Acc& a) const {
        a.re = lanes_sum<L>(a.re);
        a.im = lanes_sum<L>(a.im);
    }
    __device__ __forceinline__ void finish(Acc& a, int64_t u, const Key<W>&) const {
        const int32_t row = __ldg(unique + u);
        const int64_t e = row_ptr[row];
        col[e] = row;
        val[e] = make_double2(a.re, a.im);
    }
};

// count[i] += 1 (the diagonal entry); the 64-bit total of the counts goes to *total
__global__ void plus_one_kernel(int32_t* __restrict__ count, int64_t n, unsigned long long* __restrict__ total) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long v = 0;
    if (i < n) {
        count[i] += 1;
        v = (unsigned long long)(uint32_t)count[i];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(total, v);
}

// row_ptr[i] = offsets[i] (exclusive scan of the per-row counts), row_ptr[n] = total
__global__ void row_ptr_kernel(const int32_t* __restrict__ offsets, const int* __restrict__ total, int64_t n,
                               int64_t* __restrict__ row_ptr) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) row_ptr[i] = (int64_t)(uint32_t)offsets[i];
    if (i == n) row_ptr[n] = (int64_t)(uint32_t)*total;
}

// cursor[i] = row_ptr[i] + 1: the diagonal entry keeps the first place
__global__ void cursor_kernel(const int64_t* __restrict__ row_ptr, int64_t n, int64_t* __restrict__ cursor) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) cursor[i] = row_ptr[i] + 1;
}

// Row j of A times x, one warp: lanes over the row's entries in order, four
// entries a lane and step with all their loads in flight, a fixed butterfly
// sum: the same bits on every call.  The FP64 pipe (two lanes a clock and SM)
// and the gathers bound it: real entries take two FP64 instructions instead of
// the six of a complex product and sum.  8.7M real entries over 16,384 rows
// 168 -> 99 us.
__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}

__device__ __forceinline__ double2 row_times(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                                             const double2* __restrict__ val, const double2* __restrict__ x, int64_t j,
                                             int lane) {
    constexpr int U = 4;
    const int64_t b = __ldg(row_ptr + j), e = __ldg(row_ptr + j + 1);
    double re = 0.0, im = 0.0;
    for (int64_t k = b + lane; k - lane < e; k += 32 * U) {  // (the warp stays together)
        int32_t c[U];
        double2 v[U], p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = k + 32 * u < e ? __ldg(col + k + 32 * u) : -1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (c[u] >= 0) {
                v[u] = __ldg(val + k + 32 * u);
                p[u] = __ldg(x + c[u]);
            }
        }
        // real entries need no imaginary products (they add zeros, unless x is not finite)
        bool whole = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (c[u] >= 0) {
                re = fma(v[u].x, p[u].x, re);
                im = fma(v[u].x, p[u].y, im);
                whole = whole || nonzero(v[u].y) || !finite_bits(p[u].x) || !finite_bits(p[u].y);
            }
        }
        if (__any_sync(0xffffffffu, whole)) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (c[u] >= 0) {
                    re = fma(-v[u].y, p[u].y, re);
                    im = fma(v[u].y, p[u].x, im);
                }
            }
        }
    }
    return make_double2(warp_sum(re), warp_sum(im));
}

// Row j of A times x, one thread, entries in order: for rows whose mean is below kFewEntries.
constexpr int64_t kFewEntries = 4;

__device__ __forceinline__ double2 short_row_times(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                                                   const double2* __restrict__ val, const double2* __restrict__ x,
                                                   int64_t j) {
    const int64_t b = __ldg(row_ptr + j), e = __ldg(row_ptr + j + 1);
    double re = 0.0, im = 0.0;
    for (int64_t k = b; k < e; ++k) {
        const double2 v = __ldg(val + k);
        const double2 p = __ldg(x + __ldg(col + k));
        re += v.x * p.x - v.y * p.y;
        im += v.x * p.y + v.y * p.x;
    }
    return make_double2(re, im);
}

// y = A x, a warp per row.
__global__ void __launch_bounds__(kThreads) spmv_kernel(int64_t n, const int64_t* __restrict__ row_ptr,
                                                        const int32_t* __restrict__ col,
                                                        const double2* __restrict__ val,
                                                        const double2* __restrict__ x, double2* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kWarpsPerBlock;
    for (int64_t j = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); j < n; j += warps) {
        const double2 r = row_times(row_ptr, col, val, x, j, lane);
        if (lane == 0) y[j] = r;
    }
}

// ---------------------------------------------------------------------------
// One Lanczos iteration in three launches, the recurrence's scalars staying on
// the device: w = A v and the partial sums of alpha = Re<w, v>; w -= alpha v +
// beta_prev v_prev and the partial sums of its norm; v_next = w / beta.  Every
// block of a launch sums the previous launch's partial sums for itself, in a
// fixed order.  (As a dozen library calls an iteration, with a host read of
// beta, 16,384 rows took 250 us beside the product, 79 of them the norm.)
// ---------------------------------------------------------------------------

constexpr int kLanczosBlocks = 512;  // blocks of the vector passes at most
constexpr int kLanczosParts = 4096;  // partial sums of a launch at most

// Sum of n values over the block in a fixed order; every thread gets it.
__device__ __forceinline__ double sum_parts(const double* __restrict__ parts, int n, double* s_warp) {
    double x = 0.0;
    for (int k = threadIdx.x; k < n; k += kThreads) x += parts[k];
    x = warp_sum(x);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
    __syncthreads();
    x = 0.0;
#pragma unroll
    for (int w = 0; w < kWarpsPerBlock; ++w) x += s_warp[w];
    __syncthreads();
    return x;
}

__device__ __forceinline__ void store_part(double x, double* parts, double* s_warp) {
    x = warp_sum(x);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarpsPerBlock; ++w) t += s_warp[w];
        parts[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kThreads) lanczos_product_kernel(int64_t n, const int64_t* __restrict__ row_ptr,
                                                                   const int32_t* __restrict__ col,
                                                                   const double2* __restrict__ val,
                                                                   const double2* __restrict__ v,
                                                                   double2* __restrict__ w, double* __restrict__ parts) {
    __shared__ double s_warp[kWarpsPerBlock];
    double dot = 0.0;
    if (__ldg(row_ptr + n) < kFewEntries * n) {
        for (int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x; j < n; j += (int64_t)gridDim.x * kThreads) {
            const double2 r = short_row_times(row_ptr, col, val, v, j);
            w[j] = r;
            const double2 p = __ldg(v + j);
            dot += r.x * p.x + r.y * p.y;
        }
        store_part(dot, parts, s_warp);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kWarpsPerBlock;
    for (int64_t j = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); j < n; j += warps) {
        const double2 r = row_times(row_ptr, col, val, v, j, lane);
        if (lane == 0) {
            w[j] = r;
            const double2 p = __ldg(v + j);
            dot += r.x * p.x + r.y * p.y;
        }
    }
    store_part(dot, parts, s_warp);
}

__global__ void __launch_bounds__(kThreads) lanczos_update_kernel(int64_t n, const double* __restrict__ parts, int n_parts,
                                                                  const double2* __restrict__ v_prev,
                                                                  const double* __restrict__ beta_prev,
                                                                  const double2* __restrict__ v, double2* __restrict__ w,
                                                                  double* __restrict__ alpha,
                                                                  double* __restrict__ norms) {
    __shared__ double s_warp[kWarpsPerBlock];
    const double a = sum_parts(parts, n_parts, s_warp);
    const double b = v_prev != nullptr ? *beta_prev : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *alpha = a;
    double norm = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
        double2 x = w[i];
        const double2 p = __ldg(v + i);
        x.x -= a * p.x;
        x.y -= a * p.y;
        if (v_prev != nullptr) {
            const double2 q = __ldg(v_prev + i);
            x.x -= b * q.x;
            x.y -= b * q.y;
        }
        w[i] = x;
        norm += x.x * x.x + x.y * x.y;
    }
    store_part(norm, norms, s_warp);
}

__global__ void __launch_bounds__(kThreads) lanczos_scale_kernel(int64_t n, const double* __restrict__ norms, int n_parts,
                                                                 const double2* __restrict__ w,
                                                                 double2* __restrict__ v_next, double* __restrict__ beta) {
    __shared__ double s_warp[kWarpsPerBlock];
    const double b = sqrt(sum_parts(norms, n_parts, s_warp));
    if (blockIdx.x == 0 && threadIdx.x == 0) *beta = b;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
        const double2 x = __ldg(w + i);
        v_next[i] = make_double2(x.x / b, x.y / b);
    }
}

// y = A x for rows with few entries (the mean below kFewEntries): one thread
// per row, entries summed in order.
__global__ void __launch_bounds__(kThreads) spmv_rows_kernel(int64_t n, const int64_t* __restrict__ row_ptr,
                                                             const int32_t* __restrict__ col,
                                                             const double2* __restrict__ val,
                                                             const double2* __restrict__ x, double2* __restrict__ y) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) y[j] = short_row_times(row_ptr, col, val, x, j);
}

// Y = A X for m vectors (X, Y row-major [n][m]): one warp per row, lane l
// owns vectors l, l + 32, ...; the row's entries are read once per 32
// vectors (the same address across lanes) and summed in order.
__global__ void __launch_bounds__(kThreads) spmm_kernel(int64_t n, int m, const int64_t* __restrict__ row_ptr,
                                                        const int32_t* __restrict__ col,
                                                        const double2* __restrict__ val,
                                                        const double2* __restrict__ x, double2* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kWarpsPerBlock;
    for (int64_t j = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); j < n; j += warps) {
        const int64_t b = __ldg(row_ptr + j), e = __ldg(row_ptr + j + 1);
        for (int c = lane; c < m; c += 32) {
            double re = 0.0, im = 0.0;
            for (int64_t k = b; k < e; ++k) {
                const double2 v = __ldg(val + k);
                const double2 p = __ldg(x + (int64_t)__ldg(col + k) * m + c);
                re += v.x * p.x - v.y * p.y;
                im += v.x * p.y + v.y * p.x;
            }
            y[j * m + c] = make_double2(re, im);
        }
    }
}

// ---------------------------------------------------------------------------
// E = Re<psi|H psi> / <psi|psi> and its gradient 2 g (H psi - E psi) / <psi|psi>
// in FP64, for psi in FP64 or FP32: one pass and a sum instead of nine library
// calls (65,536 rows: 60 us of kernels), one pass instead of six.
// ---------------------------------------------------------------------------

template <bool F32>
__device__ __forceinline__ double2 amplitude_at(const void* psi, int64_t i) {
    if (F32) {
        const float2 p = __ldg(static_cast<const float2*>(psi) + i);
        return make_double2((double)p.x, (double)p.y);
    }
    return __ldg(static_cast<const double2*>(psi) + i);
}

template <bool F32>
__global__ void __launch_bounds__(kThreads) energy_parts_kernel(int64_t n, const void* __restrict__ psi,
                                                                const double2* __restrict__ hpsi,
                                                                double* __restrict__ parts) {
    __shared__ double s_warp[kWarpsPerBlock];
    double num = 0.0, norm = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
        const double2 p = amplitude_at<F32>(psi, i), h = __ldg(hpsi + i);
        num += p.x * h.x + p.y * h.y;
        norm += p.x * p.x + p.y * p.y;
    }
    store_part(num, parts, s_warp);
    __syncthreads();
    store_part(norm, parts + kLanczosBlocks, s_warp);
}

// out[0] = E, out[1] = <psi|psi>
__global__ void __launch_bounds__(kThreads) energy_sum_kernel(const double* __restrict__ parts, int n_parts,
                                                              double* __restrict__ out) {
    __shared__ double s_warp[kWarpsPerBlock];
    const double num = sum_parts(parts, n_parts, s_warp);
    const double norm = sum_parts(parts + kLanczosBlocks, n_parts, s_warp);
    if (threadIdx.x == 0) {
        out[0] = num / norm;
        out[1] = norm;
    }
}

template <bool F32>
__global__ void energy_grad_kernel(int64_t n, const void* __restrict__ psi, const double2* __restrict__ hpsi,
                                   const double* __restrict__ sums, const double* __restrict__ grad,
                                   void* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double e = sums[0], norm = sums[1], g = grad[0] * 2.0;
    const double2 p = amplitude_at<F32>(psi, i), h = __ldg(hpsi + i);
    const double re = g * (h.x - e * p.x) / norm, im = g * (h.y - e * p.y) / norm;
    if (F32) {
        static_cast<float2*>(out)[i] = make_float2((float)re, (float)im);
    } else {
        static_cast<double2*>(out)[i] = make_double2(re, im);
    }
}

struct MatrixLayout {
    HashRows rows;
    int32_t* count;
    int32_t* scan;
    int* total;
    unsigned long long* total64;
    int64_t* cursor;
};

template <int W>
MatrixLayout take_matrix(Arena& ws, int64_t n) {
    MatrixLayout L;
    L.rows = take_hashrows<W>(ws, n);
    const uint64_t cap = (uint64_t)(n > 0 ? n : 1);
    L.count = ws.take<int32_t>(cap);
    L.scan = ws.take<int32_t>((uint64_t)scan_scratch(n));
    L.total = ws.take<int>(1);
    L.total64 = ws.take<unsigned long long>(1);
    L.cursor = ws.take<int64_t>(cap);
    return L;
}

// The pair scan's scratch behind the first ws.used bytes; false when the sizes
// give it none or it does not fit.
template <int W>
bool take_matrix_pairs(const qmbx_table_header* h, const Arena& ws, int64_t n, PairWork& pairs) {
    if (!pairs_scratch(h, n, n)) return false;
    Arena rest = ws;
    pairs = take_pair_work<W>(rest, n, n, true, h->n_sites);
    return rest.fits();
}

// Walk the changing terms of every row (daggered terms, gather direction), or
// scan the pairs of rows (pairs != NULL).
template <int W, bool FILL>
int matrix_walk(const void* table_host, const void* table_dev, const MatrixLayout& L, int64_t n, const int64_t* row_ptr,
                int32_t* col, double2* val, PairWork* pairs, cudaStream_t s) {
    PartView adj = part_view(table_host, table_dev, QMBX_PART_ADJ);
    PartView diag = part_view(table_host, table_dev, QMBX_PART_DIAG);
    PartView none = adj;
    none.n = 0;
    const HashView look = L.rows.hash();
    UniqueRows<W> src{L.rows.keys, L.rows.unique};
    const int* walk_rows = L.rows.count;
    if (adj.n > 0 && pairs != nullptr) {
        // the device chooses the scan or the walk below; the other finds no rows
        int st = choose_pairs<W>(*pairs, L.rows, L.rows, L.rows, adj, s);
        if (st != QMBX_OK || (st = build_pairs<W>(L.rows, L.rows, header_of(table_host)->n_sites, *pairs, s)) != QMBX_OK) return st;
        walk_rows = pairs->gate + 1;
        const PartView fwd = part_view(table_host, table_dev, QMBX_PART_FWD);
        MatrixPairs<FILL> v{fwd.coef, L.count, L.cursor, col, val};
        if ((st = launch_pair_scan<W>(v, *pairs, table_host, table_dev, pairs->gate, s, kGroupEnumerate)) != QMBX_OK) return st;
    }
    if (adj.n > 0) {
        const int group = pairs != nullptr ? kGroupOther : kGroupEnumerate;
        const Walk kind = choose_walk(adj, n, true);
        if (kind == Walk::kPivot) {
            MatrixPivot<W, FILL> v{{}, look, adj.coef, L.rows.unique, L.count, L.cursor, col, val};
            QMBX_KERNEL(group, s, pivot_kernel<W><<<pivot_grid(), kThreads, 0, s>>>(v, src, walk_rows, n, adj));
        } else {
            MatrixRows<W, FILL> v{{}, look, adj.coef, L.rows.unique, L.count, L.cursor, col, val};
            if (kind == Walk::kGrouped) {
                QMBX_KERNEL(group, s, grouped_kernel<W><<<grouped_grid(n), kThreads, 0, s>>>(v, src, walk_rows, n, adj, none));
            } else {
                QMBX_KERNEL(group, s, enumerate_kernel<W><<<grid_for(n, kThreads), kThreads, 0, s>>>(v, src, walk_rows, n, adj, none));
            }
        }
        QMBX_LAUNCH_CHECK("matrix walk");
    }
    if (FILL) {
        MatrixDiagonal<W> dv{{}, diag.coef, L.rows.unique, row_ptr, col, val};
        int st = launch_diagonal<W>(dv, src, L.rows.count, n, diag, s, kGroupDiagonal);
        if (st != QMBX_OK) return st;
    }
    return QMBX_OK;
}

template <int W>
int matrix_count(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n, int64_t* row_ptr,
                 int64_t* nnz, Arena& ws, cudaStream_t s) {
    MatrixLayout L = take_matrix<W>(ws, n);
    if (ws.base == nullptr) return QMBX_OK;
    if (!ws.fits()) return fail(QMBX_ERR_WORKSPACE, "matrix needs %llu bytes of workspace", (unsigned long long)ws.used);
    const int nq = header_of(table_host)->n_qubytes;
    int st;
    if ((st = build_hashrows<W>(configs, nq, L.rows, s)) != QMBX_OK) return st;
    QMBX_CUDA_TRY(cudaMemsetAsync(L.count, 0, (size_t)n * sizeof(int32_t), s));
    PairWork pairs{};
    const bool scan = pairs_wanted(header_of(table_host), n, n) && take_matrix_pairs<W>(header_of(table_host), ws, n, pairs);
    if ((st = matrix_walk<W, false>(table_host, table_dev, L, n, nullptr, nullptr, nullptr, scan ? &pairs : nullptr, s)) != QMBX_OK) return st;
    QMBX_CUDA_TRY(cudaMemsetAsync(L.total64, 0, sizeof(unsigned long long), s));
    QMBX_KERNEL(kGroupOther, s, plus_one_kernel<<<grid_for(n, kThreads), kThreads, 0, s>>>(L.count, n, L.total64));
    if ((st = exclusive_scan(L.count, L.count, n, L.total, L.scan, s)) != QMBX_OK) return st;
    QMBX_KERNEL(kGroupOther, s, row_ptr_kernel<<<grid_for(n + 1, kThreads), kThreads, 0, s>>>(L.count, L.total, n, row_ptr));
    QMBX_LAUNCH_CHECK("matrix row pointers");
    int unique = 0;
    unsigned long long total = 0;
    QMBX_CUDA_TRY(cudaMemcpyAsync(&unique, L.rows.count, sizeof(int), cudaMemcpyDeviceToHost, s));
    QMBX_CUDA_TRY(cudaMemcpyAsync(&total, L.total64, sizeof(total), cudaMemcpyDeviceToHost, s));
    QMBX_CUDA_TRY(cudaStreamSynchronize(s));
    if (unique != n) return fail(QMBX_ERR_ARGUMENT, "matrix rows must be distinct (%d distinct of %lld)", unique, (long long)n);
    // the per-row offsets are scanned in 32 bits
    if (total >= (1ull << 31)) return fail(QMBX_ERR_ARGUMENT, "matrix has %llu entries, 2^31 or more", total);
    *nnz = (int64_t)total;
    return QMBX_OK;
}

template <int W>
int matrix_fill(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n, const int64_t* row_ptr,
                int32_t* col, double2* val, Arena& ws, cudaStream_t s) {
    MatrixLayout L = take_matrix<W>(ws, n);
    if (ws.base == nullptr) return QMBX_OK;
    if (!ws.fits()) return fail(QMBX_ERR_WORKSPACE, "matrix needs %llu bytes of workspace", (unsigned long long)ws.used);
    const int nq = header_of(table_host)->n_qubytes;
    int st;
    if ((st = build_hashrows<W>(configs, nq, L.rows, s)) != QMBX_OK) return st;
    QMBX_KERNEL(kGroupOther, s, cursor_kernel<<<grid_for(n, kThreads), kThreads, 0, s>>>(row_ptr, n, L.cursor));
    QMBX_LAUNCH_CHECK("matrix cursors");
    PairWork pairs{};
    const bool scan = pairs_wanted(header_of(table_host), n, n) && take_matrix_pairs<W>(header_of(table_host), ws, n, pairs);
    return matrix_walk<W, true>(table_host, table_dev, L, n, row_ptr, col, val, scan ? &pairs : nullptr, s);
}

int matrix_args(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n, void* workspace) {
    int st = check_table(table_host, table_dev);
    if (st != QMBX_OK) return st;
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (n > 0 && configs == nullptr) return fail(QMBX_ERR_ARGUMENT, "configs must not be NULL");
    if (workspace != nullptr && reinterpret_cast<uintptr_t>(workspace) % QMBX_ALIGN != 0) {
        return fail(QMBX_ERR_ARGUMENT, "workspace must be %d-byte aligned", QMBX_ALIGN);
    }
    return QMBX_OK;
}

}  // namespace
}  // namespace qmbx

using namespace qmbx;

extern "C" int qmbx_matrix_workspace(const void* table_host, int64_t n, uint64_t* bytes) {
    clear_error();
    const qmbx_table_header* h = header_of(table_host);
    if (h == nullptr || h->magic != QMBX_MAGIC) return fail(QMBX_ERR_ARGUMENT, "not a compiled qmbx table");
    if (bytes == nullptr) return fail(QMBX_ERR_ARGUMENT, "bytes must not be NULL");
    Arena probe(nullptr, 0);
    const bool pairs = pairs_scratch(h, n, n);
#define QMBX_MATRIX_BYTES(W)                                                        \
    case W:                                                                         \
        take_matrix<W>(probe, n);                                                   \
        if (pairs) take_pair_work<W>(probe, n, n, true, h->n_sites);                \
        break;
    switch (h->n_words) {
        QMBX_MATRIX_BYTES(1)
        QMBX_MATRIX_BYTES(2)
        QMBX_MATRIX_BYTES(3)
        QMBX_MATRIX_BYTES(4)
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
#undef QMBX_MATRIX_BYTES
    *bytes = probe.used;
    return QMBX_OK;
}

extern "C" int qmbx_matrix_count(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n,
                                 int64_t* row_ptr, int64_t* nnz, void* workspace, uint64_t workspace_bytes,
                                 qmbx_stream_t stream) {
    clear_error();
    int st = matrix_args(table_host, table_dev, configs, n, workspace);
    if (st != QMBX_OK) return st;
    if (row_ptr == nullptr || nnz == nullptr) return fail(QMBX_ERR_ARGUMENT, "row_ptr and nnz must not be NULL");
    *nnz = 0;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) {
        QMBX_CUDA_TRY(cudaMemsetAsync(row_ptr, 0, sizeof(int64_t), s));
        return QMBX_OK;
    }
    if (workspace == nullptr) return fail(QMBX_ERR_WORKSPACE, "matrix needs a workspace");
    Arena ws(workspace, workspace_bytes);
    switch (header_of(table_host)->n_words) {
        case 1: return matrix_count<1>(table_host, table_dev, configs, n, row_ptr, nnz, ws, s);
        case 2: return matrix_count<2>(table_host, table_dev, configs, n, row_ptr, nnz, ws, s);
        case 3: return matrix_count<3>(table_host, table_dev, configs, n, row_ptr, nnz, ws, s);
        case 4: return matrix_count<4>(table_host, table_dev, configs, n, row_ptr, nnz, ws, s);
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
}

extern "C" int qmbx_matrix_fill(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n,
                                const int64_t* row_ptr, int32_t* col, double* val, void* workspace,
                                uint64_t workspace_bytes, qmbx_stream_t stream) {
    clear_error();
    int st = matrix_args(table_host, table_dev, configs, n, workspace);
    if (st != QMBX_OK) return st;
    if (n == 0) return QMBX_OK;
    if (row_ptr == nullptr || col == nullptr || val == nullptr) return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    if (workspace == nullptr) return fail(QMBX_ERR_WORKSPACE, "matrix needs a workspace");
    Arena ws(workspace, workspace_bytes);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    double2* v = reinterpret_cast<double2*>(val);
    switch (header_of(table_host)->n_words) {
        case 1: return matrix_fill<1>(table_host, table_dev, configs, n, row_ptr, col, v, ws, s);
        case 2: return matrix_fill<2>(table_host, table_dev, configs, n, row_ptr, col, v, ws, s);
        case 3: return matrix_fill<3>(table_host, table_dev, configs, n, row_ptr, col, v, ws, s);
        case 4: return matrix_fill<4>(table_host, table_dev, configs, n, row_ptr, col, v, ws, s);
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
}

extern "C" int qmbx_matrix_apply(int64_t n, const int64_t* row_ptr, const int32_t* col, const double* val,
                                 const double* x, double* y, qmbx_stream_t stream) {
    clear_error();
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (n == 0) return QMBX_OK;
    if (row_ptr == nullptr || col == nullptr || val == nullptr || x == nullptr || y == nullptr) {
        return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    QMBX_KERNEL(kGroupSpmv, s, spmv_kernel<<<grouped_grid(n), kThreads, 0, s>>>(n, row_ptr, col, reinterpret_cast<const double2*>(val), reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y)));
    QMBX_LAUNCH_CHECK("spmv_kernel");
    return QMBX_OK;
}

extern "C" int qmbx_matrix_apply_many(int64_t n, int64_t nnz, int32_t m, const int64_t* row_ptr, const int32_t* col,
                                      const double* val, const double* x, double* y, qmbx_stream_t stream) {
    clear_error();
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (nnz < 0 || m < 1) return fail(QMBX_ERR_ARGUMENT, "entry count or vector count out of range");
    if (n == 0) return QMBX_OK;
    if (row_ptr == nullptr || col == nullptr || (nnz > 0 && val == nullptr) || x == nullptr || y == nullptr) {
        return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const double2* v = reinterpret_cast<const double2*>(val);
    const double2* xx = reinterpret_cast<const double2*>(x);
    double2* yy = reinterpret_cast<double2*>(y);
    if (m > 1) {
        QMBX_KERNEL(kGroupSpmv, s, spmm_kernel<<<grouped_grid(n), kThreads, 0, s>>>(n, m, row_ptr, col, v, xx, yy));
    } else if (nnz < kFewEntries * n) {
        QMBX_KERNEL(kGroupSpmv, s, spmv_rows_kernel<<<grid_for(n, kThreads), kThreads, 0, s>>>(n, row_ptr, col, v, xx, yy));
    } else {
        QMBX_KERNEL(kGroupSpmv, s, spmv_kernel<<<grouped_grid(n), kThreads, 0, s>>>(n, row_ptr, col, v, xx, yy));
    }
    QMBX_LAUNCH_CHECK("matrix product");
    return QMBX_OK;
}

extern "C" int qmbx_lanczos_step(int64_t n, const int64_t* row_ptr, const int32_t* col, const double* val,
                                 const double* v_prev, const double* beta_prev, const double* v, double* v_next,
                                 double* alpha, double* beta, void* scratch, uint64_t scratch_bytes,
                                 qmbx_stream_t stream) {
    clear_error();
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (n == 0) return QMBX_OK;
    if (row_ptr == nullptr || col == nullptr || val == nullptr || v == nullptr || v_next == nullptr || alpha == nullptr ||
        beta == nullptr || (v_prev == nullptr) != (beta_prev == nullptr)) {
        return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    }
    if (scratch == nullptr || reinterpret_cast<uintptr_t>(scratch) % QMBX_ALIGN != 0) {
        return fail(QMBX_ERR_ARGUMENT, "scratch must be a %d-byte aligned device buffer", QMBX_ALIGN);
    }
    Arena ws(scratch, scratch_bytes);
    double2* w = ws.take<double2>((uint64_t)n);
    double* parts = ws.take<double>(kLanczosParts);
    double* norms = ws.take<double>(kLanczosBlocks);
    if (!ws.fits()) return fail(QMBX_ERR_WORKSPACE, "a Lanczos step needs %llu bytes of scratch", (unsigned long long)ws.used);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const double2* vv = reinterpret_cast<const double2*>(v);
    const int products = grouped_grid(n) < kLanczosParts ? grouped_grid(n) : kLanczosParts;
    const int blocks = grid_for(n, kThreads) < (unsigned)kLanczosBlocks ? (int)grid_for(n, kThreads) : kLanczosBlocks;
    QMBX_KERNEL(kGroupSpmv, s, lanczos_product_kernel<<<products, kThreads, 0, s>>>(n, row_ptr, col, reinterpret_cast<const double2*>(val), vv, w, parts));
    QMBX_KERNEL(kGroupOther, s, lanczos_update_kernel<<<blocks, kThreads, 0, s>>>(n, parts, products, reinterpret_cast<const double2*>(v_prev), beta_prev, vv, w, alpha, norms));
    QMBX_KERNEL(kGroupOther, s, lanczos_scale_kernel<<<blocks, kThreads, 0, s>>>(n, norms, blocks, w, reinterpret_cast<double2*>(v_next), beta));
    QMBX_LAUNCH_CHECK("Lanczos step");
    return QMBX_OK;
}

extern "C" int qmbx_energy(int64_t n, int32_t single, const void* psi, const double* hpsi, double* sums, double* scratch,
                           qmbx_stream_t stream) {
    clear_error();
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if ((n > 0 && (psi == nullptr || hpsi == nullptr)) || sums == nullptr || scratch == nullptr) {
        return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const double2* h = reinterpret_cast<const double2*>(hpsi);
    const int blocks = grid_for(n, kThreads) < (unsigned)kLanczosBlocks ? (int)grid_for(n, kThreads) : kLanczosBlocks;
    if (single) {
        QMBX_KERNEL(kGroupOther, s, energy_parts_kernel<true><<<blocks, kThreads, 0, s>>>(n, psi, h, scratch));
    } else {
        QMBX_KERNEL(kGroupOther, s, energy_parts_kernel<false><<<blocks, kThreads, 0, s>>>(n, psi, h, scratch));
    }
    QMBX_KERNEL(kGroupOther, s, energy_sum_kernel<<<1, kThreads, 0, s>>>(scratch, blocks, sums));
    QMBX_LAUNCH_CHECK("energy");
    return QMBX_OK;
}

extern "C" int qmbx_energy_grad(int64_t n, int32_t single, const void* psi, const double* hpsi, const double* sums,
                                const double* grad, void* out, qmbx_stream_t stream) {
    clear_error();
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (n == 0) return QMBX_OK;
    if (psi == nullptr || hpsi == nullptr || sums == nullptr || grad == nullptr || out == nullptr) {
        return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const double2* h = reinterpret_cast<const double2*>(hpsi);
    if (single) {
        QMBX_KERNEL(kGroupOther, s, energy_grad_kernel<true><<<grid_for(n, kThreads), kThreads, 0, s>>>(n, psi, h, sums, grad, out));
    } else {
        QMBX_KERNEL(kGroupOther, s, energy_grad_kernel<false><<<grid_for(n, kThreads), kThreads, 0, s>>>(n, psi, h, sums, grad, out));
    }
    QMBX_LAUNCH_CHECK("energy gradient");
    return QMBX_OK;
}
