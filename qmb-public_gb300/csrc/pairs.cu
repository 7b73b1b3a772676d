// Preparing row sets for the pair scan (pairs.cuh): distinct rows ordered by
// particle number, and their bit planes.
#include <cuda_runtime.h>

#include <cstdlib>

#include "pairs.cuh"

namespace qmbx {
namespace {

template <int W>
__device__ __forceinline__ int particles(const Key<W>& k) {
    int n = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) n += __popcll(k.w[q]);
    return n;
}

// hist[p] = distinct rows with p particles.  Most sets hold one number only,
// so a warp adds one count per number it sees.
template <int W>
__global__ void pair_count_kernel(const uint64_t* __restrict__ keys, const int32_t* __restrict__ unique,
                                  const int* __restrict__ count, int* __restrict__ hist) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = u < *count;
    const int p = live ? particles<W>(load_key<W>(keys, __ldg(unique + u))) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, p);
    if (live && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(hist + p, __popc(peers));
}

// Place every distinct row: behind the rows of smaller numbers, in any order
// among its own.
template <int W>
__global__ void __launch_bounds__(kThreads) pair_place_kernel(const uint64_t* __restrict__ keys,
                                                              const int32_t* __restrict__ unique,
                                                              const int* __restrict__ count, int* __restrict__ hist,
                                                              uint64_t* __restrict__ out_keys,
                                                              int32_t* __restrict__ out_row) {
    constexpr int kNumbers = 64 * W + 1;
    __shared__ int s_base[kNumbers + 31];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int before = 0;
        for (int c = 0; c < kNumbers; c += 32) {
            const int h = c + lane < kNumbers ? hist[c + lane] : 0;
            int x = h;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            s_base[c + lane] = before + x - h;
            before += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = u < *count;
    int32_t row = 0;
    Key<W> k{};
    int p = -1;
    if (live) {
        row = __ldg(unique + u);
        k = load_key<W>(keys, row);
        p = particles<W>(k);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, p);
    const int leader = __ffs(peers) - 1;
    int at = 0;
    if (live && lane == leader) at = atomicAdd(hist + kNumbers + p, __popc(peers));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (live) {
        const int64_t pos = (int64_t)s_base[p] + at + __popc(peers & ((1u << lane) - 1u));
        store_key<W>(out_keys, pos, k);
        out_row[pos] = row;
    }
}

// A warp forms one word of every plane: the ballot over its 32 rows.
template <int W>
__global__ void __launch_bounds__(kThreads) pair_planes_kernel(const uint64_t* __restrict__ keys,
                                                               const int* __restrict__ count, int sites,
                                                               uint32_t* __restrict__ planes) {
    constexpr int kWords = 32 * pair_words<W>();
    const int lane = threadIdx.x & 31;
    const int64_t word = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const int64_t n = *count;
    const int64_t words = (n + pair_tile<W>() - 1) / pair_tile<W>() * kWords;  // the last tile is filled with zeros
    if (word >= words) return;
    const int64_t pos = 32 * word + lane;
    Key<W> k{};
    if (pos < n) k = load_key<W>(keys, pos);
    uint32_t* out = planes + word / kWords * sites * kWords + word % kWords;
#pragma unroll
    for (int q = 0; q < 2 * W; ++q) {
        uint32_t mine = 0;
#pragma unroll
        for (int b = 0; b < 32; ++b) {
            const int bit = (32 * (q & 1) + b) ^ 56;  // site 32 q + b of the row
            const uint32_t m = __ballot_sync(0xffffffffu, (k.w[q >> 1] >> bit) & 1ull);
            if (lane == b) mine = m;
        }
        if (32 * q + lane < sites) out[(32 * q + lane) * kWords] = mine;
    }
}

// The list of every row's occupied sites (PairSet::list), a thread per row.
template <int W>
__global__ void __launch_bounds__(kThreads) pair_list_kernel(const uint64_t* __restrict__ keys,
                                                             const int* __restrict__ count, int sites,
                                                             uint16_t* __restrict__ lists) {
    const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= *count) return;
    const Key<W> k = load_key<W>(keys, pos);
    uint16_t* list = lists + pos * sites;
    int n = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) {
        for (uint64_t m = k.w[q]; m != 0;) {
            const int bit = 63 - __clzll((long long)m);
            m ^= 1ull << bit;
            list[n++] = (uint16_t)((64 * q + (bit ^ 56)) * 32);  // key bit to site (see format.h)
        }
    }
    if (n & 1) list[n] = (uint16_t)(sites * 32);
}

template <int W>
__global__ void pair_gate_kernel(const uint64_t* __restrict__ keys, const int* __restrict__ count,
                                 const int* __restrict__ walked, int* __restrict__ gate) {
    const int64_t n = *count;
    const bool scan = n > 0 && particles<W>(load_key<W>(keys, n - 1)) > 3;  // rows are ordered by number
    gate[0] = scan ? *walked : 0;
    gate[1] = scan ? 0 : *walked;
}

}  // namespace

template <int W>
int choose_pairs(const PairWork& p, const HashRows& walked, cudaStream_t s) {
    const PairSet& a = pairs_swapped(p) ? p.j : p.i;
    QMBX_KERNEL(kGroupOther, s, pair_gate_kernel<W><<<1, 1, 0, s>>>(a.keys, a.count, walked.count, p.gate));
    QMBX_LAUNCH_CHECK("pair_gate_kernel");
    return QMBX_OK;
}

template <int W>
PairSet take_pair_set(Arena& ws, int64_t n, int sites) {
    PairSet out{};
    const uint64_t cap = (uint64_t)(n > 0 ? n : 1);
    const uint64_t tiles = (cap + pair_tile<W>() - 1) / pair_tile<W>();
    out.n = n;
    out.keys = ws.take<uint64_t>(cap * W);
    out.row = ws.take<int32_t>(cap);
    out.planes = ws.take<uint32_t>(tiles * (uint64_t)sites * 32 * pair_words<W>());
    out.list = ws.take<uint16_t>((cap + kPairRun - 1) / kPairRun * kPairRun * (uint64_t)sites);
    out.hist = ws.take<int>(2 * (64 * W + 1));
    return out;
}

template <int W>
int build_pair_set(const HashRows& rows, int sites, bool planes, bool lists, PairSet& out, cudaStream_t s) {
    out.count = rows.count;
    QMBX_CUDA_TRY(cudaMemsetAsync(out.hist, 0, 2 * (64 * W + 1) * sizeof(int), s));
    const int64_t words = (rows.n + pair_tile<W>() - 1) / pair_tile<W>() * 32 * pair_words<W>();
    QMBX_KERNEL(kGroupKeys, s, pair_count_kernel<W><<<grid_for(rows.n, kThreads), kThreads, 0, s>>>(rows.keys, rows.unique, rows.count, out.hist));
    QMBX_KERNEL(kGroupKeys, s, pair_place_kernel<W><<<grid_for(rows.n, kThreads), kThreads, 0, s>>>(rows.keys, rows.unique, rows.count, out.hist, out.keys, out.row));
    if (lists) QMBX_KERNEL(kGroupKeys, s, pair_list_kernel<W><<<grid_for(rows.n, kThreads), kThreads, 0, s>>>(out.keys, rows.count, sites, out.list));
    if (planes) QMBX_KERNEL(kGroupKeys, s, pair_planes_kernel<W><<<grid_for(words, kWarpsPerBlock), kThreads, 0, s>>>(out.keys, rows.count, sites, out.planes));
    QMBX_LAUNCH_CHECK("build_pair_set");
    return QMBX_OK;
}

#define QMBX_INSTANTIATE_PAIRS(W)                                     \
    template PairSet take_pair_set<W>(Arena&, int64_t, int);          \
    template int choose_pairs<W>(const PairWork&, const HashRows&, cudaStream_t); \
    template int build_pair_set<W>(const HashRows&, int, bool, bool, PairSet&, cudaStream_t);

QMBX_INSTANTIATE_PAIRS(1)
QMBX_INSTANTIATE_PAIRS(2)
QMBX_INSTANTIATE_PAIRS(3)
QMBX_INSTANTIATE_PAIRS(4)

bool pairs_possible(const qmbx_table_header* h) { return h->n_class_buckets > 0; }

namespace {

// The sizes at which the scan beats the term walks, measured on FP64 calls
// (whole calls, scan against the faster walk).  A walk's work is its rows
// times the terms they reach, the scan's its pairs of rows: 200,000 x 20,000
// rows of 55,371 terms on 28 sites 0.62 against 0.94 ms, 65,536 rows of
// 669,579 terms on 52 sites 0.44 against 13.4 ms.  Small calls are launches
// (400 rows of 55,371 terms 138 against 109 us, 2,000 rows 113 against 165
// us).  Operators that hold few of the possible transitions connect few of
// the pairs that the scan looks up.
bool scan_pays(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    const double walked = (double)(n_i < n_j ? n_i : n_j), other = (double)(n_i < n_j ? n_j : n_i);
    const double terms = (double)h->part[QMBX_PART_FWD].n, sites = (double)h->n_sites;
    const double moves = sites * (sites - 1) / 2;
    return other * sites < 250.0 * terms && walked * terms > 1e8 && terms > 0.01 * moves * moves;
}

// Small calls always have scratch for the scan, so that it can be forced on them.
constexpr int64_t kPairsAlways = int64_t(1) << 17;

}  // namespace

bool pairs_scratch(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    return pairs_possible(h) && n_i > 0 && n_j > 0 && (scan_pays(h, n_i, n_j) || n_i + n_j <= kPairsAlways);
}

bool pairs_wanted(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    if (!pairs_possible(h) || n_i <= 0 || n_j <= 0 || deterministic_mode()) return false;
    const char* e = getenv("QMBX_WALK");
    const char f = e != nullptr ? e[0] : 0;
    if (f == 's') return true;
    return f != 't' && f != 'g' && f != 'p' && scan_pays(h, n_i, n_j);
}

int pair_chunk(int64_t n_list, int64_t n_planes, int tile) {
    const int64_t tiles = (n_planes + tile - 1) / tile;
    constexpr int64_t step = kWarpsPerBlock * kPairRun;
    int64_t rows = n_list * tiles / (16 * 152) / step * step;
    // few rows: a run or less a warp, so that the items spread over the SMs
    if (rows < step) rows = step;
    if (rows > 8192) rows = 8192;
    return (int)rows;
}

}  // namespace qmbx
