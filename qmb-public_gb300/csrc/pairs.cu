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
                                  const int* __restrict__ count, const int* __restrict__ gate,
                                  int* __restrict__ hist) {
    if (*gate == 0) return;
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
                                                              const int* __restrict__ count,
                                                              const int* __restrict__ gate, int* __restrict__ hist,
                                                              uint64_t* __restrict__ out_keys,
                                                              int32_t* __restrict__ out_row) {
    constexpr int kNumbers = 64 * W + 1;
    __shared__ int s_base[kNumbers + 31];
    if (*gate == 0) return;
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

// The planes of the rows (a warp forms one word of every plane: the ballot
// over its 32 rows), the list of every row's occupied sites (PairSet::list, a
// thread per row), or both.
template <int W>
__global__ void __launch_bounds__(kThreads) pair_form_kernel(const uint64_t* __restrict__ keys,
                                                             const int* __restrict__ count,
                                                             const int* __restrict__ gate, int sites,
                                                             uint32_t* __restrict__ planes,
                                                             uint16_t* __restrict__ lists) {
    if (*gate == 0) return;
    constexpr int kWords = 32 * pair_words<W>();
    const int lane = threadIdx.x & 31;
    const int64_t word = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const int64_t n = *count;
    const int64_t words = (n + pair_tile<W>() - 1) / pair_tile<W>() * kWords;  // the last tile is filled with zeros
    if (word >= words) return;
    const int64_t pos = 32 * word + lane;
    Key<W> k{};
    if (pos < n) k = load_key<W>(keys, pos);
    if (planes != nullptr) {
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
    if (lists != nullptr && pos < n) {
        uint16_t* list = lists + pos * sites;
        int at = 0;
#pragma unroll
        for (int q = 0; q < W; ++q) {
            for (uint64_t m = k.w[q]; m != 0;) {
                const int bit = 63 - __clzll((long long)m);
                m ^= 1ull << bit;
                list[at++] = (uint16_t)((64 * q + (bit ^ 56)) * 32);  // key bit to site (see format.h)
            }
        }
        if (at & 1) list[at] = (uint16_t)(sites * 32);
    }
}

// choose_pairs' sample: a warp takes a row a of the list side, 256 rows b of the other one from a place of its own,
// and the sizes of a's pivot groups.  The last block to finish sums up.
constexpr int kGateBlocks = 152;
constexpr int kGateRows = 256;

template <int W>
__global__ void __launch_bounds__(kThreads) pair_gate_kernel(UniqueRows<W> a, const int* __restrict__ a_count,
                                                             UniqueRows<W> b, const int* __restrict__ b_count,
                                                             const int2* __restrict__ groups, int same, int forced,
                                                             double fixed_ps,
                                                             const int* __restrict__ walked,
                                                             unsigned long long* sums, int* __restrict__ gate) {
    __shared__ uint8_t s_pos[kWarpsPerBlock][64 * W];
    __shared__ unsigned int s_sum[3];  // close pairs, reached terms, particles
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int64_t na = *a_count, nb = *b_count;
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
    __syncthreads();
    if (na > 0 && nb > 0) {
        const uint64_t w = (uint64_t)blockIdx.x * kWarpsPerBlock + warp;
        const int64_t ia = (int64_t)(w * (uint64_t)na / (uint64_t)(kGateBlocks * kWarpsPerBlock));
        const Key<W> c = a.get(ia);
        const uint64_t start = ((w * 0x9E3779B97F4A7C15ull) >> 24) % (uint64_t)nb;
        int close = 0, reach = 0, occ = 0;
#pragma unroll
        for (int u = 0; u < kGateRows / 32; ++u) {
            int64_t ib = (int64_t)start + 32 * u + lane;
            if (ib >= nb) ib %= nb;
            const Key<W> k = b.get(ib);
            int gone = 0, come = 0;
#pragma unroll
            for (int q = 0; q < W; ++q) {
                gone += __popcll(c.w[q] & ~k.w[q]);
                come += __popcll(k.w[q] & ~c.w[q]);
            }
            close += gone == come && gone <= 2 && !(same && ia == ib) ? 1 : 0;
        }
        uint8_t* pos = s_pos[warp];
#pragma unroll
        for (int h = 0; h < 2 * W; ++h) {
            const uint32_t bits = (uint32_t)(c.w[h >> 1] >> (32 * (h & 1)));
            if (bits >> lane & 1u) pos[occ + __popc(bits & lt)] = (uint8_t)(32 * h + lane);
            occ += __popc(bits);
        }
        __syncwarp();
        auto size = [&](int64_t g) {
            const int2 se = __ldg(groups + g);
            return se.y - se.x;
        };
        if (lane == 0) reach += size(0);
        for (int i = lane; i < occ; i += 32) reach += size(qmbx_single_group(pos[i]));
        for (int i = 0; i < occ; ++i) {
            for (int k = i + 1 + lane; k < occ; k += 32) reach += size(qmbx_pair_group(W, pos[i], pos[k]));
        }
        close = (int)__reduce_add_sync(0xffffffffu, (unsigned)close);
        const unsigned high = __reduce_add_sync(0xffffffffu, (unsigned)reach >> 16);
        const unsigned low = __reduce_add_sync(0xffffffffu, (unsigned)reach & 0xffffu);
        if (lane == 0) {
            atomicAdd(&s_sum[0], (unsigned)close);
            atomicAdd(&s_sum[2], (unsigned)occ);
            atomicAdd(sums + 1, ((unsigned long long)high << 16) + low);
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    atomicAdd(sums + 0, (unsigned long long)s_sum[0]);
    atomicAdd(sums + 2, (unsigned long long)s_sum[2]);
    __threadfence();
    if (atomicAdd(sums + 3, 1ull) != gridDim.x - 1) return;
    __threadfence();
    constexpr double kWarps = (double)kGateBlocks * kWarpsPerBlock;
    const double close = (double)*(volatile unsigned long long*)(sums + 0) / (kWarps * kGateRows);
    const double reach = (double)*(volatile unsigned long long*)(sums + 1) / kWarps;
    const double particles = (double)*(volatile unsigned long long*)(sums + 2) / kWarps;
    const double pairs = (double)na * (double)nb * (same ? 0.5 : 1.0);
    const double scan_ps = fixed_ps + pairs * (0.0075 * particles + close * (same ? 80.0 : 40.0));
    const double walk_ps = 5.0 * (double)*walked * reach;
    // forced: still not for rows of three particles and fewer
    const bool scan = na > 0 && nb > 0 && (forced ? particles > 3.0 : scan_ps < walk_ps);
    gate[0] = scan ? *walked : 0;
    gate[1] = scan ? 0 : *walked;
}

}  // namespace

template <int W>
int choose_pairs(const PairWork& p, const HashRows& rows_i, const HashRows& rows_j, const HashRows& walked,
                 const PartView& terms, cudaStream_t s) {
    const HashRows& a = pairs_swapped(p) ? rows_j : rows_i;
    const HashRows& b = pairs_swapped(p) ? rows_i : rows_j;
    QMBX_CUDA_TRY(cudaMemsetAsync(p.next, 0, p.clear_bytes, s));
    const double fixed_ps = choose_walk(terms, walked.n, true) == Walk::kPivot ? 0.0 : 35e6;
    QMBX_KERNEL(kGroupOther, s, pair_gate_kernel<W><<<kGateBlocks, kThreads, 0, s>>>(UniqueRows<W>{a.keys, a.unique}, a.count, UniqueRows<W>{b.keys, b.unique}, b.count, terms.groups, p.same ? 1 : 0, pairs_forced() ? 1 : 0, fixed_ps, walked.count, p.next + 2, p.gate));
    QMBX_LAUNCH_CHECK("pair_gate_kernel");
    return QMBX_OK;
}

template <int W>
PairSet take_pair_set(Arena& ws, int64_t n, int sites, int* hist) {
    PairSet out{};
    const uint64_t cap = (uint64_t)(n > 0 ? n : 1);
    const uint64_t tiles = (cap + pair_tile<W>() - 1) / pair_tile<W>();
    out.n = n;
    out.keys = ws.take<uint64_t>(cap * W);
    out.row = ws.take<int32_t>(cap);
    out.planes = ws.take<uint32_t>(tiles * (uint64_t)sites * 32 * pair_words<W>());
    out.list = ws.take<uint16_t>((cap + kPairRun - 1) / kPairRun * kPairRun * (uint64_t)sites);
    out.hist = hist;
    return out;
}

template <int W>
int build_pair_set(const HashRows& rows, int sites, bool planes, bool lists, const int* gate, PairSet& out, cudaStream_t s) {
    out.count = rows.count;
    const int64_t words = (rows.n + pair_tile<W>() - 1) / pair_tile<W>() * 32 * pair_words<W>();
    QMBX_KERNEL(kGroupKeys, s, pair_count_kernel<W><<<grid_for(rows.n, kThreads), kThreads, 0, s>>>(rows.keys, rows.unique, rows.count, gate, out.hist));
    QMBX_KERNEL(kGroupKeys, s, pair_place_kernel<W><<<grid_for(rows.n, kThreads), kThreads, 0, s>>>(rows.keys, rows.unique, rows.count, gate, out.hist, out.keys, out.row));
    QMBX_KERNEL(kGroupKeys, s, pair_form_kernel<W><<<grid_for(words, kWarpsPerBlock), kThreads, 0, s>>>(out.keys, rows.count, gate, sites, planes ? out.planes : nullptr, lists ? out.list : nullptr));
    QMBX_LAUNCH_CHECK("build_pair_set");
    return QMBX_OK;
}

#define QMBX_INSTANTIATE_PAIRS(W)                                     \
    template PairSet take_pair_set<W>(Arena&, int64_t, int, int*);    \
    template int choose_pairs<W>(const PairWork&, const HashRows&, const HashRows&, const HashRows&, const PartView&, cudaStream_t); \
    template int build_pair_set<W>(const HashRows&, int, bool, bool, const int*, PairSet&, cudaStream_t);

QMBX_INSTANTIATE_PAIRS(1)
QMBX_INSTANTIATE_PAIRS(2)
QMBX_INSTANTIATE_PAIRS(3)
QMBX_INSTANTIATE_PAIRS(4)

bool pairs_possible(const qmbx_table_header* h) { return h->n_class_buckets > 0; }

namespace {

// The sizes at which the scan can beat the term walks; choose_pairs then looks
// at the rows.  (us, FP64 calls within one set, scan against the faster walk)
//   terms x walked rows: small calls are launches, and a call that may scan
//     and walks has 25 us of them for nothing.  3,792 rows under 55,371 terms
//     (2.1e8) 111 against 208 with 5 + 5 electrons, 128 against 143 with 3 + 3
//     and 151 (walked) against 122 with 2 + 2; 1,805 rows (1e8) 110 against
//     148, 113 against 104 and, clustered, 196 against 117.
//   other side x sites: in choose_pairs' costs a pair of rows may cost 0.0075
//     N / (5 N^2 / S^2) of a reached term at N of S sites, so the walk is the
//     cheaper for any rows filled up to 3/8 past 250 terms a row and site.
//   terms per possible transition: below one in a hundred next to none of the
//     pairs within two moves are connected (lattices).
bool scan_pays(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    const double walked = (double)(n_i < n_j ? n_i : n_j), other = (double)(n_i < n_j ? n_j : n_i);
    const double terms = (double)h->part[QMBX_PART_FWD].n, sites = (double)h->n_sites;
    const double moves = sites * (sites - 1) / 2;
    return other * sites < 250.0 * terms && walked * terms > 2e8 && terms > 0.01 * moves * moves;
}

// Calls on more rows have no scratch for a scan that QMBX_WALK forces on them.
constexpr int64_t kPairsForced = int64_t(1) << 17;

}  // namespace

bool pairs_forced() {
    const char* e = getenv("QMBX_WALK");
    return e != nullptr && e[0] == 's';
}

// Scratch is for the sizes that may be scanned, and for small calls while QMBX_WALK forces the scan on them: every
// call compares what it was given with what its scan needs, and walks without.
bool pairs_scratch(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    if (!pairs_possible(h) || n_i <= 0 || n_j <= 0) return false;
    return scan_pays(h, n_i, n_j) || (pairs_forced() && n_i + n_j <= kPairsForced);
}

bool pairs_wanted(const qmbx_table_header* h, int64_t n_i, int64_t n_j) {
    if (!pairs_possible(h) || n_i <= 0 || n_j <= 0 || deterministic_mode()) return false;
    return pairs_forced() || (!walk_forced() && scan_pays(h, n_i, n_j));
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
