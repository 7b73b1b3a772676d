// Key handling: packing rows into big-endian key words, prefix sums, and
// de-duplicated row sets.
//
// The reference sorts rows with thrust and a byte-wise comparator
// (qmb/_hamiltonian_cuda.cu:245-251, :624-629, :956-961); here row sets are
// hash sets over 64-bit key words.
#include <cuda_runtime.h>

#include <cstdlib>

#include "device.cuh"

namespace qmbx {

// ---------------------------------------------------------------------------
// pack / unpack
// ---------------------------------------------------------------------------

template <int W>
__global__ void pack_kernel(const uint8_t* __restrict__ rows, int64_t n, int nq, uint64_t* __restrict__ keys) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t* r = rows + i * nq;
#pragma unroll
    for (int q = 0; q < W; ++q) {
        uint64_t w = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int b = 8 * q + j;
            uint64_t byte = b < nq ? (uint64_t)r[b] : 0;
            w |= byte << (8 * (7 - j));
        }
        keys[i * W + q] = w;
    }
}

template <int W>
int pack_rows(const uint8_t* rows, int64_t n, int nq, uint64_t* keys, cudaStream_t s) {
    if (n == 0) return QMBX_OK;
    QMBX_KERNEL(kGroupKeys, s, pack_kernel<W><<<grid_for(n, kThreads), kThreads, 0, s>>>(rows, n, nq, keys));
    QMBX_LAUNCH_CHECK("pack_kernel");
    return QMBX_OK;
}

// ---------------------------------------------------------------------------
// exclusive scan (reduce, scan of block sums, scan with offsets)
// ---------------------------------------------------------------------------

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanChunk = kScanThreads * kScanItems;

__global__ void set_zero_kernel(int32_t* p) { *p = 0; }

__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t* s_warp, int32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int32_t w = lane < nwarps ? s_warp[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            int32_t y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        if (lane < nwarps) s_warp[lane] = w;
    }
    __syncthreads();
    int32_t before = warp > 0 ? s_warp[warp - 1] : 0;
    if (total) *total = s_warp[nwarps - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void scan_reduce_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ sums) {
    __shared__ int32_t s_warp[32];
    int64_t base = (int64_t)blockIdx.x * kScanChunk;
    int32_t acc = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
        if (i < n) acc += in[i];
    }
    int32_t total;
    block_exclusive_scan(acc, s_warp, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void scan_sums_kernel(int32_t* __restrict__ sums, int64_t nb, int* __restrict__ total_out) {
    __shared__ int32_t s_warp[32];
    // each thread scans a contiguous run of per-block sums
    int64_t per = (nb + blockDim.x - 1) / blockDim.x;
    int64_t lo = (int64_t)threadIdx.x * per;
    int64_t hi = lo + per < nb ? lo + per : nb;
    int32_t local = 0;
    for (int64_t i = lo; i < hi; ++i) local += sums[i];
    int32_t total;
    int32_t before = block_exclusive_scan(local, s_warp, &total);
    for (int64_t i = lo; i < hi; ++i) {
        int32_t v = sums[i];
        sums[i] = before;
        before += v;
    }
    if (threadIdx.x == 0 && total_out) *total_out = total;
}

__global__ void scan_apply_kernel(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n,
                                  const int32_t* __restrict__ sums) {
    __shared__ int32_t s_warp[32];
    int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int32_t local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + k;
        v[k] = i < n ? in[i] : 0;
        local += v[k];
    }
    int32_t run = block_exclusive_scan(local, s_warp, nullptr) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

// Exclusive scan of up to kScanChunk values in one block (one launch instead of three).
__global__ void scan_single_kernel(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n,
                                   int* __restrict__ total_out) {
    __shared__ int32_t s_warp[32];
    const int64_t base = (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int32_t local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k;
        v[k] = i < n ? in[i] : 0;
        local += v[k];
    }
    int32_t total;
    int32_t run = block_exclusive_scan(local, s_warp, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
    if (threadIdx.x == 0 && total_out) *total_out = total;
}

int64_t scan_scratch(int64_t n) {
    int64_t nb = (n + kScanChunk - 1) / kScanChunk;
    return nb < 1 ? 1 : nb;
}

int exclusive_scan(const int32_t* in, int32_t* out, int64_t n, int* total, int32_t* scratch, cudaStream_t s,
                   int group) {
    int64_t nb = scan_scratch(n);
    if (n > 0 && n <= kScanChunk) {
        QMBX_KERNEL(group, s, scan_single_kernel<<<1, kScanThreads, 0, s>>>(in, out, n, total));
        QMBX_LAUNCH_CHECK("exclusive_scan");
        return QMBX_OK;
    }
    if (n > 0) QMBX_KERNEL(group, s, scan_reduce_kernel<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, scratch));
    else QMBX_KERNEL(group, s, set_zero_kernel<<<1, 1, 0, s>>>(scratch));
    QMBX_KERNEL(group, s, scan_sums_kernel<<<1, kScanThreads, 0, s>>>(scratch, nb, total));
    if (n > 0) QMBX_KERNEL(group, s, scan_apply_kernel<<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, scratch));
    QMBX_LAUNCH_CHECK("exclusive_scan");
    return QMBX_OK;
}

// ---------------------------------------------------------------------------
// hash-based de-duplicated row sets
// ---------------------------------------------------------------------------

// Insert every row; a key already present keeps the lowest row.  A slot is
// claimed by a CAS on its row word and then given its fingerprint; a row
// that finds its key in a claimed slot (compared in full: the fingerprint
// may not be written yet) lowers that slot's row with atomicMin.  Every row
// of a key meets the same slot, the first claimed on the key's probe
// sequence.
template <int W>
__global__ void hashrows_insert_kernel(const uint64_t* __restrict__ keys, int64_t n, uint64_t* __restrict__ slots,
                                       uint64_t mask, uint32_t* __restrict__ bloom, uint32_t bloom_mask) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const Key<W> k = load_key<W>(keys, r);
    const uint64_t hv = key_hash<W>(k);
    if (bloom != nullptr) {
        const uint64_t f = bloom_mix(hv);
        atomicOr(bloom + bloom_word(f, bloom_mask), bloom_bits(f));
    }
    uint64_t i = hash_home(hv, hash_shift(mask + 1));
    uint32_t* w = reinterpret_cast<uint32_t*>(slots);
    for (uint64_t probe = 0; probe <= mask; ++probe) {
        uint32_t* row = w + slot_row_word(i);
        uint32_t cur = *(volatile uint32_t*)row;
        if (cur == kEmptyRow) {
            cur = atomicCAS(row, kEmptyRow, (uint32_t)r);
            if (cur == kEmptyRow) {
                w[slot_tag_word(i)] = hash_tag(hv);
                return;
            }
        }
        if (key_eq<W>(load_key<W>(keys, (int64_t)cur), k)) {
            atomicMin(row, (uint32_t)r);
            return;
        }
        i = (i + 1) & mask;
    }
}

// first[r] = lowest row with row r's key; every such first row is listed in
// unique[0 .. *count) (in no particular order: a warp reserves its places
// with one atomic).
template <int W>
__global__ void hashrows_resolve_kernel(const uint64_t* __restrict__ keys, int64_t n, HashView h,
                                        int32_t* __restrict__ first, int32_t* __restrict__ unique,
                                        int* __restrict__ count) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = r < n;
    int64_t f = -1;
    if (live) {
        f = hash_find<W>(h, load_key<W>(keys, r));
        first[r] = (int32_t)f;
    }
    const bool head = live && f == r;
    const unsigned m = __ballot_sync(0xffffffffu, head);
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (head) unique[at + __popc(m & ((1u << lane) - 1u))] = (int32_t)r;
}

template <int W>
HashRows take_hashrows(Arena& ws, int64_t n) {
    HashRows out;
    uint64_t cap = (uint64_t)(n > 0 ? n : 1);
    out.n = n;
    out.keys = ws.take<uint64_t>(cap * W);
    uint64_t slots = 64;
    while (slots < 4 * cap) slots <<= 1;
    out.slots = ws.take<uint64_t>(slots);
    out.slot_mask = slots - 1;
    out.first = ws.take<int32_t>(cap);
    out.unique = ws.take<int32_t>(cap);
    out.count = ws.take<int>(1);
    out.bloom_words = bloom_words_for(n);
    out.bloom = out.bloom_words ? ws.take<uint32_t>(out.bloom_words) : nullptr;
    return out;
}

template <int W>
int build_hashset(const uint8_t* rows, int nq, HashRows& out, cudaStream_t s) {
    const int64_t n = out.n;
    QMBX_CUDA_TRY(cudaMemsetAsync(out.slots, 0xff, (out.slot_mask + 1) * sizeof(uint64_t), s));
    if (n == 0) return QMBX_OK;
    int st;
    if ((st = pack_rows<W>(rows, n, nq, out.keys, s)) != QMBX_OK) return st;
    const unsigned grid = grid_for(n, kThreads);
    // the filter (when the set has one) is complete before the first lookup (the resolve pass)
    if (out.bloom_words) QMBX_CUDA_TRY(cudaMemsetAsync(out.bloom, 0, (size_t)out.bloom_words * sizeof(uint32_t), s));
    QMBX_KERNEL(kGroupKeys, s, hashrows_insert_kernel<W><<<grid, kThreads, 0, s>>>(out.keys, n, out.slots, out.slot_mask,
                                                                  out.bloom_words ? out.bloom : nullptr,
                                                                  out.bloom_words ? out.bloom_words - 1 : 0));
    QMBX_LAUNCH_CHECK("build_hashset");
    return QMBX_OK;
}

template <int W>
int build_hashrows(const uint8_t* rows, int nq, HashRows& out, cudaStream_t s) {
    QMBX_CUDA_TRY(cudaMemsetAsync(out.count, 0, sizeof(int), s));
    int st = build_hashset<W>(rows, nq, out, s);
    if (st != QMBX_OK || out.n == 0) return st;
    QMBX_KERNEL(kGroupKeys, s, hashrows_resolve_kernel<W><<<grid_for(out.n, kThreads), kThreads, 0, s>>>(out.keys, out.n, out.hash(), out.first, out.unique, out.count));
    QMBX_LAUNCH_CHECK("build_hashrows");
    return QMBX_OK;
}

// ---------------------------------------------------------------------------
// rows that share all key words but one (Reach)
// ---------------------------------------------------------------------------

template <int W>
__device__ __forceinline__ void reach_place(Key<W> k, int left_out, uint64_t words, uint64_t& at, unsigned long long& bits) {
#pragma unroll
    for (int q = 0; q < W; ++q) k.w[q] = q == left_out ? (uint64_t)(q + 1) : k.w[q];
    const uint64_t f = bloom_mix(key_hash<W>(k));
    at = (f >> 40) & (words - 1);
    bits = (1ull << ((f >> 8) & 63)) | (1ull << ((f >> 14) & 63)) | (1ull << ((f >> 20) & 63)) | (1ull << ((f >> 26) & 63));
}

template <int W>
__global__ void reach_insert_kernel(const uint64_t* __restrict__ keys, const int32_t* __restrict__ unique,
                                    const int* __restrict__ count, Reach r) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= *count) return;
    const Key<W> k = load_key<W>(keys, __ldg(unique + u));
#pragma unroll
    for (int w = 0; w < W; ++w) {
        uint64_t at;
        unsigned long long bits;
        reach_place<W>(k, w, r.words, at, bits);
        const unsigned long long old = atomicOr(r.once + w * r.words + at, bits);
        if ((old & bits) == bits) atomicOr(r.twice + w * r.words + at, bits);
    }
}

// A walked row that is itself in the looked-up set shares all its words with
// its own copy, which no term that changes a row leads to: only places that
// two rows or more took count for it.
template <int W>
__global__ void reach_flags_kernel(const uint64_t* __restrict__ keys, const int32_t* __restrict__ unique,
                                   const int* __restrict__ count, int same, HashView look, Reach r) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= *count) return;
    const Key<W> k = load_key<W>(keys, __ldg(unique + u));
    unsigned flags = 0;
    const bool own = same || hash_find<W>(look, k) >= 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        uint64_t at;
        unsigned long long bits;
        reach_place<W>(k, w, r.words, at, bits);
        const unsigned long long have = __ldg((own ? r.twice : r.once) + w * r.words + at);
        if ((have & bits) == bits) flags |= 1u << w;
    }
    r.flags[u] = (uint8_t)flags;
}

template <int W>
Reach take_reach(Arena& ws, int64_t n_walk, int64_t n_look) {
    Reach r{};
    r.words = 1024;
    while (r.words * 2 < (uint64_t)(n_look > 0 ? n_look : 1) && r.words < (1ull << 24)) r.words <<= 1;
    r.once = ws.take<unsigned long long>(r.words * W);
    r.twice = ws.take<unsigned long long>(r.words * W);
    r.flags = ws.take<uint8_t>((uint64_t)(n_walk > 0 ? n_walk : 1));
    return r;
}

template <int W>
int build_reach(const HashRows& walk, const HashRows& look, bool same, const Reach& r, cudaStream_t s) {
    QMBX_CUDA_TRY(cudaMemsetAsync(r.once, 0, (size_t)r.words * W * sizeof(unsigned long long), s));
    QMBX_CUDA_TRY(cudaMemsetAsync(r.twice, 0, (size_t)r.words * W * sizeof(unsigned long long), s));
    QMBX_KERNEL(kGroupKeys, s, reach_insert_kernel<W><<<grid_for(look.n, kThreads), kThreads, 0, s>>>(look.keys, look.unique, look.count, r));
    QMBX_KERNEL(kGroupKeys, s, reach_flags_kernel<W><<<grid_for(walk.n, kThreads), kThreads, 0, s>>>(walk.keys, walk.unique, walk.count, same ? 1 : 0, look.hash(), r));
    QMBX_LAUNCH_CHECK("build_reach");
    return QMBX_OK;
}

#define QMBX_INSTANTIATE_KEYS(W)                                                          \
    template int pack_rows<W>(const uint8_t*, int64_t, int, uint64_t*, cudaStream_t);     \
    template HashRows take_hashrows<W>(Arena&, int64_t);                                  \
    template Reach take_reach<W>(Arena&, int64_t, int64_t);                               \
    template int build_reach<W>(const HashRows&, const HashRows&, bool, const Reach&, cudaStream_t); \
    template int build_hashset<W>(const uint8_t*, int, HashRows&, cudaStream_t);          \
    template int build_hashrows<W>(const uint8_t*, int, HashRows&, cudaStream_t);

QMBX_INSTANTIATE_KEYS(1)
QMBX_INSTANTIATE_KEYS(2)
QMBX_INSTANTIATE_KEYS(3)
QMBX_INSTANTIATE_KEYS(4)

}  // namespace qmbx

namespace qmbx {

static int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (sms[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 132;
        sms[dev] = v;
    }
    return sms[dev];
}

int pivot_grid() { return sm_count() * 4; }

int row_split(int64_t n_rows) {
    const int64_t warps = (int64_t)sm_count() * 32 * 2;  // two waves of 32 resident warps per SM
    if (n_rows <= 0 || n_rows >= warps) return 1;
    const int64_t k = (warps + n_rows - 1) / n_rows;
    return (int)(k < 16 ? k : 16);
}

bool walk_forced() {
    const char* e = getenv("QMBX_WALK");
    return e != nullptr && (e[0] == 't' || e[0] == 'g' || e[0] == 'p');
}

Walk choose_walk(const PartView& part, int64_t n_rows, bool pivot_ok) {
    const char* e = getenv("QMBX_WALK");
    const char f = e != nullptr ? e[0] : 0;
    if (part.n == 0 || f == 't') return Walk::kTiled;
    if (f == 'p') return pivot_ok ? Walk::kPivot : Walk::kGrouped;
    if (f == 'g') return Walk::kGrouped;
    if (part.n >= kGroupedMinTerms) {
        // groups holding hundreds of terms amortise staging them in shared memory
        const bool big_groups = part.n_nonempty > 0 && part.n >= (int64_t)kPivotMeanGroup * part.n_nonempty;
        if (pivot_ok && big_groups) return Walk::kPivot;
        // groups of a few terms (the diagonal part of an ab-initio table) over many rows: testing
        // every term of a shared-memory tile against each row, all lanes on the same term, costs
        // less than dealing the small groups to the lanes (C5's 1M-row diagonal: 12.9 -> ~3 ms)
        if (!part.wide && part.n <= kTiledMaxTerms && n_rows >= kFewWideRows) return Walk::kTiled;
        return Walk::kGrouped;
    }
    return n_rows < (part.wide ? kFewWideRows : kFewRows) ? Walk::kGrouped : Walk::kTiled;
}

bool deterministic_mode() {
    const char* e = getenv("QMBX_DETERMINISTIC");
    return e != nullptr && e[0] != 0 && e[0] != '0';
}

int grouped_grid(int64_t n_rows) {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (sms[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 132;
        sms[dev] = v;
    }
    int64_t want = (n_rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
    int64_t cap = (int64_t)sms[dev] * 16;
    if (want > cap) want = cap;
    return (int)(want > 0 ? want : 1);
}

}  // namespace qmbx
