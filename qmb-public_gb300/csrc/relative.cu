// find_relative and single_relative.
//
// The reference keeps a global min-heap of count_selected records guarded by
// per-node spin locks (qmb/_hamiltonian_cuda.cu:276-675) and samples
// single_relative neighbours under per-row locks (:805-996).  Here neither
// needs a lock or any device-side wait:
//
//   find_relative  pass 1 counts records per weight bucket (the top 12 bits of
//                  an FP32 estimate |coef|^2 |psi|^2 of the weight) over every
//                  16th source row (every row of small inputs); one block
//                  picks from the scaled counts a bucket that should hold
//                  about twice count_selected records above it; pass 2 keeps
//                  the records at or above the bucket below that one.  The
//                  kept records get the reference's exact FP64 weight
//                  (:494-497) and a 128-bit rank key (weight, visiting order);
//                  a radix select finds the count_selected-th key, and the
//                  rows up to it are sorted, de-duplicated and unpacked, all
//                  from counts on the device.  The host reads once: if fewer
//                  than count_selected records were kept, pass 2 and the rest
//                  run again with an exact threshold.
//   single_relative  the first term, in descending order of its
//                  Efraimidis-Spirakis key, that leads outside the input; the
//                  walks keep the best key of a row's candidates in registers.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdlib>

#include "device.cuh"

namespace qmbx {
namespace {

namespace cg = cooperative_groups;

constexpr int kBuckets = 4096;

// Figures of the calling thread's last find_relative call (qmbx_find_relative_stats).
struct FindStats {
    int64_t records;      // records emitted by the selection pass
    int64_t walks;        // threshold and emission passes run
    int64_t sort_passes;  // radix passes over records and selected rows
    int64_t sort_bytes;   // passes x 2 (read + write) x items x item bytes
    int64_t selected;     // records selected before de-duplication
    int64_t rows_out;     // distinct rows returned
};
thread_local FindStats g_find_stats{};

__device__ __forceinline__ int weight_bucket(float est) {
    // 0 for zero (or underflowed) estimates; otherwise 1 + the top 12 bits of
    // the IEEE pattern, which is monotone for non-negative floats
    return est > 0.f ? 1 + (int)(__float_as_uint(est) >> 20) : 0;
}

// The reference's weight (qmb/_hamiltonian_cuda.cu:494-497), every product
// and sum rounded once in that order.
__device__ __forceinline__ double exact_weight(double2 cf, double2 p, int parity) {
    double re = __dsub_rn(__dmul_rn(cf.x, p.x), __dmul_rn(cf.y, p.y));
    double im = __dadd_rn(__dmul_rn(cf.x, p.y), __dmul_rn(cf.y, p.x));
    if (parity) {
        re = -re;
        im = -im;
    }
    return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

// Device-side state of one find_relative call: the selection threshold of
// the emission pass, its record count, and the selected and returned rows.
// Read by the host once, at the end.
struct FindCtl {
    unsigned long long n_emit;     // records emitted (atomic counter of the emission pass)
    unsigned long long n_zero;     // emitted records of zero exact weight
    unsigned long long n_sel;      // records selected
    unsigned long long n_unique;   // distinct rows returned
    int overflow;
    int emit_from;                 // lowest bucket the emission pass keeps
    int count_from;                // the first count's bucket (> 0) if a whole count from it follows, else 0
    unsigned int first_done;       // blocks of the first count that have finished, and of the whole one
    unsigned int above_done;
    unsigned int n_long[2];        // groups queued for their rest (LongGroup): by the threshold's count, by the emission
};

// The rest of a pivot group that a row reaches far into: terms t .. end of row `row`.
struct LongGroup {
    int row, t, end;
};

// The histogram (EMIT = false) and emission (EMIT = true) passes as
// visitors of the enumeration kernels.  Every (term, row) image that is not
// an excluded row is a candidate record; diagonal terms produce the row
// itself.  The histogram lives in shared memory and is flushed once per block.
struct RelativeArgs {
    const double2* psi;      // configs_i amplitudes, input order
    int64_t n_i;
    HashView excl;           // hash set over the unique exclude keys
    PartView off, diag;
    // histogram passes
    unsigned long long* hist;
    int hist_exact;          // 1: count only records outside the exclusion set (the exact rerun);
                             // 0: count every record (a threshold estimate: no exclusion lookups)
    unsigned long long* deep;  // bounded passes: by bucket, terms that the truncated count left out (an estimate)
    LongGroup* queue;
    unsigned int queue_cap;
    // pass 2 (emit_from, the record counter and the overflow flag live in ctl)
    FindCtl* ctl;
    int64_t cap_emit;
    uint64_t* emit_rank;     // [cap][2]: (slot | part << 62 | parity << 63, row) from the walk;
                             // (~weight bits, ~order) after rank_records_kernel
    uint64_t* emit_keys;     // [cap][W]
};

template <int W, bool EMIT>
struct RelativeVisitor : VisitorBase {
    RelativeArgs a;
    static constexpr int kShared = kBuckets;
    struct Acc {
        double2 p;
        float m;
        int64_t row;
        int* hist;
        int emit_from;  // the emission pass's threshold bucket, read once per row
    };
    // the histogram pass counts every record per bucket in shared memory; the
    // emission pass counts only what it emits (its record counter)
    __device__ __forceinline__ void block_init(int* sh) const {
        if (EMIT) return;
        for (int k = threadIdx.x; k < kBuckets; k += blockDim.x) sh[k] = 0;
    }
    __device__ __forceinline__ void block_flush(int* sh) const {
        if (EMIT) return;
        for (int k = threadIdx.x; k < kBuckets; k += blockDim.x) {
            int v = sh[k];
            if (v) atomicAdd(a.hist + k, (unsigned long long)v);
        }
    }
    __device__ __forceinline__ void init(Acc& acc, int64_t row, const Key<W>&, int* sh) const {
        acc.p = __ldg(a.psi + row);
        // FP32 estimate of |psi|^2 (no FP64 in the walk)
        const float px = (float)acc.p.x, py = (float)acc.p.y;
        acc.m = __fadd_rn(__fmul_rn(px, px), __fmul_rn(py, py));
        acc.row = row;
        acc.hist = sh;
        acc.emit_from = EMIT ? a.ctl->emit_from : 0;
    }
    static constexpr bool kProbe = true;
    HashView lookup;  // the exclusion set
    // A candidate record whose image is not excluded.  The emission pass
    // stores what identifies the record (term slot and part, parity, row);
    // its exact FP64 weight is formed afterwards by rank_records_kernel, so
    // that the walk issues no FP64 instruction.
    __device__ __forceinline__ int bucket(const Acc& acc, const PartView& pv, int64_t slot) const {
        return weight_bucket(__fmul_rn(__ldg(pv.norm + slot), acc.m));
    }
    // The emission pass's record at or above the threshold whose image is not excluded.
    __device__ __forceinline__ void emit(const Acc& acc, const Key<W>& img, int part, int parity,
                                         int64_t slot) const {
        const unsigned long long at = atomicAdd(&a.ctl->n_emit, 1ull);
        if ((int64_t)at >= a.cap_emit) {
            a.ctl->overflow = 1;
            return;
        }
        a.emit_rank[2 * at + 0] = (uint64_t)slot | ((uint64_t)part << 62) | ((uint64_t)parity << 63);
        a.emit_rank[2 * at + 1] = (uint64_t)acc.row;
#pragma unroll
        for (int q = 0; q < W; ++q) a.emit_keys[at * W + q] = img.w[q];
    }
    // One candidate record (term slot of part pv, image img).  The histogram
    // pass counts it by bucket (outside the exclusion set only when exact, or
    // for diagonal records).  The emission pass compares its bucket with the
    // threshold first: nearly every record falls below it and then needs no
    // exclusion lookup.
    __device__ __forceinline__ void candidate(Acc& acc, const Key<W>& img, const PartView& pv, int part, int parity,
                                              int64_t slot) const {
        if (!EMIT) {
            // diagonal records (part 1) are always looked up: their image is the row itself,
            // which the exclusion set usually holds, and their weights are among the largest
            if ((a.hist_exact || part == 1) && hash_find<W>(lookup, img) >= 0) return;
            atomicAdd(&acc.hist[bucket(acc, pv, slot)], 1);
            return;
        }
        if (bucket(acc, pv, slot) < acc.emit_from) return;
        if (hash_find<W>(lookup, img) >= 0) return;
        emit(acc, img, part, parity, slot);
    }
    __device__ __forceinline__ void visit(Acc& acc, const Key<W>&, const Key<W>& img, int parity, int64_t slot) const {
        candidate(acc, img, a.off, 0, parity, slot);
    }
    __device__ __forceinline__ void visit_diag(Acc& acc, const Key<W>& c, int parity, int64_t slot) const {
        candidate(acc, c, a.diag, 1, parity, slot);
    }
    __device__ __forceinline__ void reduce(Acc&) const {}
    __device__ __forceinline__ void finish(Acc&, int64_t, const Key<W>&) const {}
};

// Inclusive scan of v over the T threads of a block in thread order (s_warp: 32 values).
template <int Threads = 1024, class T>
__device__ __forceinline__ T block_inclusive_scan(T v, T* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < Threads / 32 ? s_warp[lane] : T(0);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    return warp > 0 ? x + s_warp[warp - 1] : x;
}

// The highest bucket b > 0 whose buckets >= b hold at least `target` records
// by the counts of a histogram pass (scaled by `scale`), 0 when there is none.
// Every thread of the block's `Threads` gets it: thread t sums the buckets
// [4096 - P (t + 1), 4096 - P t), a scan over the threads (highest buckets
// first) finds the one thread where the running count reaches the target, and
// that thread walks its buckets.
template <int Threads>
__device__ __forceinline__ int choose_bucket(const unsigned long long* hist, double scale, double target,
                                             unsigned long long* s_warp, int* s_found) {
    constexpr int kPer = kBuckets / Threads;
    const int t = threadIdx.x;
    const int hi = kBuckets - kPer * t;  // thread t covers buckets [hi - kPer, hi)
    if (t == 0) *s_found = 0;
    // integer counts, scaled only where compared: the running count is exact and monotone, so
    // exactly one thread sees it cross the target
    unsigned long long mine = 0;
    for (int b = hi - 1; b >= hi - kPer && b >= 1; --b) mine += __ldcg(hist + b);
    const unsigned long long run = block_inclusive_scan<Threads>(mine, s_warp);
    if (scale * (double)run >= target && scale * (double)(run - mine) < target) {
        // the one thread whose buckets reach the target
        unsigned long long above = run - mine;
        for (int b = hi - 1; b >= hi - kPer && b >= 1; --b) {
            above += __ldcg(hist + b);
            if (scale * (double)above >= target) {
                *s_found = b;
                break;
            }
        }
    }
    __syncthreads();
    const int found = *s_found;
    __syncthreads();  // s_found and s_warp are written again
    return found;
}

// emit_from from the counts of a histogram pass, by one block: one bucket
// below the one that choose_bucket finds (0 when all buckets above 0 hold
// fewer).  deep (or NULL): by bucket, what the pass left out; where that could
// be more than half of the target from the bucket on, count_from asks for a
// whole count.  The counts are left cleared.
template <int Threads>
__device__ __forceinline__ void choose_emit(unsigned long long* hist, const unsigned long long* deep, double scale,
                                            double target, FindCtl* ctl, unsigned long long* s_warp, int* s_found) {
    const int b = choose_bucket<Threads>(hist, scale, target, s_warp, s_found);
    unsigned long long left_out = 0;
    for (int k = threadIdx.x; k < kBuckets; k += Threads) {
        if (deep != nullptr && k >= (b > 1 ? b : 1)) left_out += __ldcg(deep + k);
        hist[k] = 0;
    }
    left_out = block_inclusive_scan<Threads>(left_out, s_warp);
    if (threadIdx.x == Threads - 1) {
        ctl->emit_from = b > 1 ? b - 1 : 0;
        ctl->count_from = scale * (double)left_out > 0.5 * target ? (b > 1 ? b : 1) : 0;
    }
}

constexpr int kChooseThreads = 1024;

__global__ void __launch_bounds__(kChooseThreads) choose_emit_kernel(unsigned long long* hist, double scale, double target,
                                                                     FindCtl* ctl) {
    __shared__ unsigned long long s_warp[32];
    __shared__ int s_found;
    choose_emit<kChooseThreads>(hist, nullptr, scale, target, ctl, s_warp, &s_found);
}

// The same passes over parts whose groups hold many terms (PartView::wide) in
// falling order of their norms, bounded by the norms.  A warp takes a row (or
// one of `split` shares of it); the lanes take its pivot groups, and a group's
// terms are read only while the bound of the rest of the group (the norms
// themselves for tables sorted by |coef|) can still reach the threshold.
// Selections take few records of a row (121k of 5.7e7 for the top 50,000 of
// 20,000 rows under 55,371 terms), so most groups end at their first bound:
// the pass is a few instructions per group instead of a test per term, and is
// bound by the latency of its reads.  On GB300, emission passes (with the
// rests) against the walks: those rows 428 -> 81 us, the top 1,000,000 of
// 8,192 rows under 3.1M terms 4.58 -> 0.35 ms (pivot-major walk and diagonal
// pass), the top 200,000 of 4,099 rows under 669,579 terms 1.42 -> 0.08 ms.
//
// Three passes share the code:
//   kFirst  counts the first `depth` steps of 32 terms of every group, all
//           buckets: the records near the threshold are the first of their
//           groups.  What it leaves out only lowers the threshold; an estimate
//           of it goes to a.deep.
//   kAbove  counts every record of the buckets from `from` on.
//   kEmit   emits them.
// The last two leave a group after kInline steps of eight lanes and queue its
// rest, which a warp each takes up afterwards (bounded_rest): a row with most
// of the weight, as configurations of a wave function have them, reaches
// thousands of terms of every group, one after the other a chain of
// milliseconds for the one warp that has the row.
//
// Diagonal terms give the row itself: one exclusion lookup per row, and a
// group a lane (their groups hold a term or two).
enum BoundedPass { kFirst, kAbove, kEmit };
constexpr int kInline = 2;

// A record of bucket b per lane where `on`: counted, or emitted.
template <int W, int Pass>
__device__ __forceinline__ void bounded_take(const RelativeArgs& a, int* hist, bool on, int b, const Key<W>& img, int part,
                                             int parity, int64_t slot, int64_t row, int lane) {
    if (Pass != kEmit) {
        if (on) atomicAdd(hist + b, 1);
        return;
    }
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (m == 0) return;
    unsigned long long at = 0;
    if (lane == __ffs(m) - 1) at = atomicAdd(&a.ctl->n_emit, (unsigned long long)__popc(m));
    at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
    if (!on) return;
    if ((int64_t)at >= a.cap_emit) {
        a.ctl->overflow = 1;
        return;
    }
    a.emit_rank[2 * at + 0] = (uint64_t)slot | ((uint64_t)part << 62) | ((uint64_t)parity << 63);
    a.emit_rank[2 * at + 1] = (uint64_t)row;
#pragma unroll
    for (int q = 0; q < W; ++q) a.emit_keys[at * W + q] = img.w[q];
}

// A term whose bound is not below the threshold (NaN: not known to be).
__device__ __forceinline__ bool bounded_reaches(float bound, float m, int from) {
    const float e = __fmul_rn(bound, m);
    return e != e || weight_bucket(e) >= from;
}

// Term t of the changing part for the row (c, m): whether it can still reach the threshold is returned, its record
// taken.  Everything a term needs is read at once: one trip to L2 before its lookup.
template <int W, int Pass>
__device__ __forceinline__ bool bounded_term(const RelativeArgs& a, int* hist, bool in, int t, const Key<W>& c, float m,
                                             int from, int64_t row, int lane) {
    const PartView& pv = a.off;
    bool on = false;
    int par = 0, b = 0;
    Key<W> img{};
    if (in) {
        TermRec<W> rec;
        bool narrow = false;
        if constexpr (W == 1) narrow = pv.narrow != nullptr;
        if (narrow) {
            load_narrow<W>(rec, pv, t);
        } else {
            load_test<W>(rec, pv, t);
            if (Pass == kEmit) load_apply<W>(rec, pv, t);
        }
        b = weight_bucket(__fmul_rn(__ldg(pv.norm + t), m));
        if (Pass != kFirst) in = bounded_reaches(__ldg(pv.bound + t), m, from);
        on = in && b >= from && rec.applies(c);
        if (Pass == kEmit && on) {
            par = rec.image(c, img);
            on = hash_find<W>(a.excl, img) < 0;
        }
    }
    bounded_take<W, Pass>(a, hist, on, b, img, 0, par, t, row, lane);
    return in;
}

__device__ __forceinline__ float bounded_weight(const double2* psi, int64_t row) {
    const double2 p = __ldg(psi + row);
    const float px = (float)p.x, py = (float)p.y;
    return __fadd_rn(__fmul_rn(px, px), __fmul_rn(py, py));
}

template <int W, int Pass>
__device__ void bounded_rows(const RelativeArgs& a, const uint64_t* __restrict__ keys, int64_t n, int split, int depth,
                             int from, int* hist, int* deep, uint8_t* pos, unsigned int* n_long) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int64_t items = n * split, stride = (int64_t)gridDim.x * kWarpsPerBlock;
    for (int64_t u = (int64_t)blockIdx.x * kWarpsPerBlock + warp; u < items; u += stride) {
        const int64_t row = u / split;
        const int share = (int)(u - row * split);
        const Key<W> c = load_key<W>(keys, row);
        const float m = bounded_weight(a.psi, row);
        // occupied key positions, ascending
        int occ = 0;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2 * W; ++h) {
            const uint32_t bits = (uint32_t)(c.w[h >> 1] >> (32 * (h & 1)));
            if (bits >> lane & 1u) pos[occ + __popc(bits & lt)] = (uint8_t)(32 * h + lane);
            occ += __popc(bits);
        }
        __syncwarp();
        const bool row_excluded = hash_find<W>(a.excl, c) >= 0;
        for (int part = 0; part < (row_excluded ? 1 : 2); ++part) {
            const PartView& pv = part == 0 ? a.off : a.diag;
            if (pv.n == 0) continue;
            // i < 0: group 0 and the single groups; else the pairs (position i, a later one)
            for (int i = share - 1; i < occ; i += split) {
                const int count = i < 0 ? 1 + occ : occ - i - 1;
                for (int k0 = 0; k0 < count; k0 += 32) {
                    const int k = k0 + lane;
                    int2 se = make_int2(0, 0);
                    if (k < count) {
                        const int64_t g = i >= 0 ? qmbx_pair_group(W, pos[i], pos[i + 1 + k])
                                                 : (k == 0 ? 0 : qmbx_single_group(pos[k - 1]));
                        se = __ldg(pv.groups + g);
                    }
                    bool alive = se.x < se.y;
                    if (Pass != kFirst && alive) alive = bounded_reaches(__ldg(pv.bound + se.x), m, from);
                    if (part == 1) {
                        // a group a lane
                        for (int t = se.x; __any_sync(0xffffffffu, alive && t < se.y); ++t) {
                            bool on = false;
                            int par = 0, b = 0;
                            if (alive && t < se.y) {
                                TermRec<W> rec;
                                load_test<W>(rec, pv, t);
                                b = weight_bucket(__fmul_rn(__ldg(pv.norm + t), m));
                                on = rec.applies(c) && b >= from;
                                if (Pass == kEmit && on) {
                                    load_apply<W>(rec, pv, t);
                                    Key<W> img;
                                    par = rec.image(c, img);
                                }
                            }
                            bounded_take<W, Pass>(a, hist, on, b, c, 1, par, t, row, lane);
                        }
                        continue;
                    }
                    if (Pass == kFirst && alive && se.y - se.x > 32 * depth) {
                        // what is left out, half of it taken to apply, goes to the bucket of its bound
                        const float rest = __fmul_rn(__ldg(pv.bound + se.x + 32 * depth), m);
                        const int b = rest == rest ? weight_bucket(rest) : kBuckets - 1;
                        atomicAdd(deep + b, (se.y - se.x - 32 * depth + 1) / 2);
                        se.y = se.x + 32 * depth;
                    }
                    // above a threshold: four groups at a time, eight lanes each (a group gives a record or
                    // two); the first count: a group at a time
                    constexpr int L = Pass == kFirst ? 32 : 8;
                    const int sub = lane / L;
                    for (unsigned todo = __ballot_sync(0xffffffffu, alive); todo != 0;) {
                        int src = -1;
#pragma unroll
                        for (int q = 0; q < 32 / L; ++q) {
                            const int next = __ffs(todo) - 1;
                            if (sub == q) src = next;
                            todo &= todo - 1;  // (0 stays 0)
                        }
                        const int start = __shfl_sync(0xffffffffu, se.x, src < 0 ? 0 : src);
                        const int end = __shfl_sync(0xffffffffu, se.y, src < 0 ? 0 : src);
                        int t = start + lane % L;
                        bool open = src >= 0;
                        for (int step = 0; __any_sync(0xffffffffu, open); ++step) {
                            if (Pass != kFirst && step == kInline) {
                                // queue the rest; a full queue leaves it here
                                bool placed = false;
                                if (open && lane % L == 0) {
                                    const unsigned int at = atomicAdd(n_long, 1u);
                                    placed = at < a.queue_cap;
                                    if (placed) a.queue[at] = LongGroup{(int)row, t, end};
                                }
                                placed = __shfl_sync(0xffffffffu, placed, sub * L);
                                open = open && !placed;
                                if (!__any_sync(0xffffffffu, open)) break;
                            }
                            const bool in = bounded_term<W, Pass>(a, hist, open && t < end, t, c, m, from, row, lane);
                            // the bounds fall: a group ends at the first lane that stops
                            const unsigned ins = __ballot_sync(0xffffffffu, in);
                            constexpr unsigned kAll = 0xffffffffu >> (32 - L);
                            open = (ins >> (L * sub) & kAll) == kAll;
                            t += L;
                        }
                    }
                }
            }
        }
    }
}

// The queued rests, a warp each, 32 terms a step.
template <int W, int Pass>
__device__ void bounded_rest(const RelativeArgs& a, const uint64_t* __restrict__ keys, int from, int* hist,
                             const unsigned int* n_long) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int queued = __ldcg(n_long);
    const unsigned int n = queued < a.queue_cap ? queued : a.queue_cap;
    for (unsigned int k = blockIdx.x * kWarpsPerBlock + warp; k < n; k += gridDim.x * kWarpsPerBlock) {
        const LongGroup g{__ldcg(&a.queue[k].row), __ldcg(&a.queue[k].t), __ldcg(&a.queue[k].end)};
        const Key<W> c = load_key<W>(keys, g.row);
        const float m = bounded_weight(a.psi, g.row);
        bool open = true;
        for (int t = g.t + lane; open; t += 32) {
            const bool in = bounded_term<W, Pass>(a, hist, t < g.end, t, c, m, from, g.row, lane);
            open = __all_sync(0xffffffffu, in);
        }
    }
}

__device__ __forceinline__ void bounded_flush(int* shared, unsigned long long* counts) {
    __syncthreads();
    for (int k = threadIdx.x; k < kBuckets; k += kThreads) {
        const int v = shared[k];
        if (v) atomicAdd(counts + k, (unsigned long long)v);
        shared[k] = 0;
    }
    __syncthreads();
}

// The first count; the last block to finish chooses the threshold by it.
template <int W>
__global__ void __launch_bounds__(kThreads) find_first_kernel(RelativeArgs a, const uint64_t* __restrict__ keys, int64_t n,
                                                              int split, int depth, double scale, double target) {
    __shared__ int s_hist[kBuckets], s_deep[kBuckets];
    __shared__ uint8_t s_pos[kWarpsPerBlock][64 * W];
    __shared__ unsigned long long s_warp[32];
    __shared__ int s_found;
    __shared__ bool s_last;
    for (int k = threadIdx.x; k < kBuckets; k += kThreads) s_hist[k] = s_deep[k] = 0;
    __syncthreads();
    bounded_rows<W, kFirst>(a, keys, n, split, depth, 0, s_hist, s_deep, s_pos[threadIdx.x >> 5], nullptr);
    bounded_flush(s_hist, a.hist);
    bounded_flush(s_deep, a.deep);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&a.ctl->first_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    choose_emit<kThreads>(a.hist, a.deep, scale, target, a.ctl, s_warp, &s_found);
}

// The whole count from the first one's bucket on, where choose_emit asks for
// it (rows of very different weights): the rows, then the queued rests and, by
// the last block to finish, the threshold.  The counts are left cleared.
//   top 200,000 of 4,099 rows of 14 on 52, amplitudes falling exponentially:
//   1,699,998 records emitted by the first count alone, 369,709 by both
template <int W>
__global__ void __launch_bounds__(kThreads) find_above_kernel(RelativeArgs a, const uint64_t* __restrict__ keys, int64_t n,
                                                              int split) {
    __shared__ int s_hist[kBuckets];
    __shared__ uint8_t s_pos[kWarpsPerBlock][64 * W];
    const int from = a.ctl->count_from;
    if (from == 0) return;
    for (int k = threadIdx.x; k < kBuckets; k += kThreads) s_hist[k] = 0;
    __syncthreads();
    bounded_rows<W, kAbove>(a, keys, n, split, 0, from, s_hist, nullptr, s_pos[threadIdx.x >> 5], a.ctl->n_long);
    bounded_flush(s_hist, a.hist);
}

template <int W>
__global__ void __launch_bounds__(kThreads) find_above_rest_kernel(RelativeArgs a, const uint64_t* __restrict__ keys,
                                                                   double scale, double target) {
    __shared__ int s_hist[kBuckets];
    __shared__ unsigned long long s_warp[32];
    __shared__ int s_found;
    __shared__ bool s_last;
    const int from = a.ctl->count_from;
    if (from == 0) return;
    for (int k = threadIdx.x; k < kBuckets; k += kThreads) s_hist[k] = 0;
    __syncthreads();
    bounded_rest<W, kAbove>(a, keys, from, s_hist, a.ctl->n_long);
    bounded_flush(s_hist, a.hist);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&a.ctl->above_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    choose_emit<kThreads>(a.hist, nullptr, scale, target, a.ctl, s_warp, &s_found);
}

// The emission pass: the rows, and the queued rests behind them.
template <int W>
__global__ void __launch_bounds__(kThreads) find_emit_kernel(RelativeArgs a, const uint64_t* __restrict__ keys, int64_t n,
                                                             int split) {
    __shared__ uint8_t s_pos[kWarpsPerBlock][64 * W];
    bounded_rows<W, kEmit>(a, keys, n, split, 0, a.ctl->emit_from, nullptr, nullptr, s_pos[threadIdx.x >> 5], a.ctl->n_long + 1);
}

template <int W>
__global__ void __launch_bounds__(kThreads) find_rest_kernel(RelativeArgs a, const uint64_t* __restrict__ keys) {
    bounded_rest<W, kEmit>(a, keys, a.ctl->emit_from, nullptr, a.ctl->n_long + 1);
}

// Whether the bounded passes serve the part (QMBX_WALK forces the walks).
bool relative_bounded(const PartView& off) {
    const char* e = getenv("QMBX_WALK");
    return off.n >= kGroupedMinTerms && off.wide && off.falling && off.bound != nullptr &&
           !(e != nullptr && (e[0] == 't' || e[0] == 'g' || e[0] == 'p'));
}

// Steps of 32 terms the bounded histogram reads of a group: rows reach at
// least a dozen or so groups, so this is several times the records a group
// gives to a selection of k.
int histogram_depth(int64_t k, int64_t n_i) {
    const int64_t steps = 1 + 2 * k / (n_i > 0 ? n_i : 1) / 128;
    return (int)(steps < (1 << 20) ? steps : 1 << 20);
}

// Shares a row is split in for the emission: rows differ widely in the records
// they give (|psi|^2), so that rows of many are cut into shares of about 32.
int emission_split(int64_t k, int64_t n_i) {
    const int64_t shares = 2 * k / (n_i > 0 ? n_i : 1) / 32;
    const int64_t fill = row_split(n_i);
    return (int)(shares > 16 ? 16 : shares > fill ? shares : fill);
}

template <int W>
int launch_threshold(const RelativeArgs& r, const uint64_t* keys, int64_t n, int64_t k, int64_t n_i, double target, cudaStream_t s) {
    const int split = row_split(n);
    const double scale = (double)n_i / (double)n;
    QMBX_KERNEL(kGroupEnumerate, s, find_first_kernel<W><<<grouped_grid(n * split), kThreads, 0, s>>>(r, keys, n, split, histogram_depth(k, n_i), scale, target));
    QMBX_KERNEL(kGroupOther, s, find_above_kernel<W><<<grouped_grid(n * split), kThreads, 0, s>>>(r, keys, n, split));
    QMBX_KERNEL(kGroupOther, s, find_above_rest_kernel<W><<<pivot_grid(), kThreads, 0, s>>>(r, keys, scale, target));
    QMBX_LAUNCH_CHECK("find_relative threshold");
    return QMBX_OK;
}

template <int W>
int launch_emit(const RelativeArgs& r, const uint64_t* keys, int64_t n, int64_t k, cudaStream_t s) {
    const int split = emission_split(k, n);
    QMBX_KERNEL(kGroupEnumerate, s, find_emit_kernel<W><<<grouped_grid(n * split), kThreads, 0, s>>>(r, keys, n, split));
    QMBX_KERNEL(kGroupOther, s, find_rest_kernel<W><<<2 * pivot_grid(), kThreads, 0, s>>>(r, keys));
    QMBX_LAUNCH_CHECK("find_relative emission pass");
    return QMBX_OK;
}

template <int W, bool EMIT>
int launch_relative(const RelativeArgs& r, const uint64_t* keys_i, int64_t n_i, cudaStream_t s) {
    RelativeVisitor<W, EMIT> v;
    v.a = r;
    v.lookup = r.excl;
    KeyRows<W> src{keys_i};
    const Walk kind = choose_walk(r.off, n_i, true);
    if (kind == Walk::kGrouped) {
        // few rows (the sampled threshold pass, small seed sets): a row's groups shared by several warps
        const int split = row_split(n_i);
        if (split > 1) {
            QMBX_KERNEL(kGroupEnumerate, s, grouped_split_kernel<W><<<grouped_grid(n_i * split), kThreads, 0, s>>>(v, src, n_i, split, r.off, r.diag));
        } else {
            QMBX_KERNEL(kGroupEnumerate, s, grouped_kernel<W><<<grouped_grid(n_i), kThreads, 0, s>>>(v, src, nullptr, n_i, r.off, r.diag));
        }
    } else if (kind == Walk::kPivot) {
        // pivot-major walk of the changing terms, then the diagonal terms tiled
        QMBX_KERNEL(kGroupEnumerate, s, pivot_kernel<W><<<pivot_grid(), kThreads, 0, s>>>(v, src, nullptr, n_i, r.off));
        if (r.diag.n > 0) {
            PartView none = r.off;
            none.n = 0;
            if (choose_walk(r.diag, n_i, false) == Walk::kGrouped) {
                QMBX_KERNEL(kGroupDiagonal, s, grouped_kernel<W><<<grouped_grid(n_i), kThreads, 0, s>>>(v, src, nullptr, n_i, none, r.diag));
            } else {
                QMBX_KERNEL(kGroupDiagonal, s, enumerate_kernel<W><<<grid_for(n_i, kThreads), kThreads, 0, s>>>(v, src, nullptr, n_i, none, r.diag));
            }
        }
    } else {
        QMBX_KERNEL(kGroupEnumerate, s, enumerate_kernel<W><<<grid_for(n_i, kThreads), kThreads, 0, s>>>(v, src, nullptr, n_i, r.off, r.diag));
    }
    QMBX_LAUNCH_CHECK(EMIT ? "find_relative emission pass" : "find_relative histogram pass");
    return QMBX_OK;
}

// Inputs of 4,096 rows or more count records on every kSampleStride-th row
// in pass 1.
constexpr int64_t kSampleStride = 16;
constexpr int64_t kSampleMinRows = 4096;

// Every kSampleStride-th row of keys and psi.
template <int W>
__global__ void sample_rows_kernel(const uint64_t* __restrict__ keys, const double2* __restrict__ psi, int64_t n_s,
                                   uint64_t* __restrict__ keys_s, double2* __restrict__ psi_s) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_s) return;
    const int64_t r = j * kSampleStride;
#pragma unroll
    for (int q = 0; q < W; ++q) keys_s[j * W + q] = keys[r * W + q];
    psi_s[j] = psi[r];
}

// ---------------------------------------------------------------------------
// The tail of a call in two cooperative launches (one block of 1,024 threads
// per SM, the blocks in step through grid barriers) that take their counts
// from the device: the selection of the count_selected heaviest records, and
// the sort, de-duplication and unpacking of their rows.  As some 45 launches
// with two host round trips between them the tail was bound by launching them
// (the top 50,000 of 121k records: 156 us of kernels in 0.4 ms).
// ---------------------------------------------------------------------------

constexpr int kTailThreads = 1024;
constexpr int kTailWarps = kTailThreads / 32;

constexpr int kSelectBits = 11;
constexpr int kSelectBins = 1 << kSelectBits;
static_assert(3 * kSelectBins * sizeof(unsigned int) <= kBuckets * sizeof(unsigned long long), "the bins reuse the histogram");

// `cnt` key bits starting `from` bits below the most significant bit of (k0, k1).
__device__ __forceinline__ uint32_t key_bits(uint64_t k0, uint64_t k1, int from, int cnt) {
    const uint64_t mask = (1ull << cnt) - 1ull;
    if (from + cnt <= 64) return (uint32_t)((k0 >> (64 - from - cnt)) & mask);
    if (from >= 64) return (uint32_t)((k1 >> (128 - from - cnt)) & mask);
    const int lo = from + cnt - 64;  // bits taken from k1
    return (uint32_t)((((k0 << lo) | (k1 >> (64 - lo)))) & mask);
}

// -1, 0, 1 as the top `bits` bits of (k0, k1) are below, equal to or above those of (p0, p1).
__device__ __forceinline__ int prefix_cmp(uint64_t k0, uint64_t k1, uint64_t p0, uint64_t p1, int bits) {
    if (bits <= 0) return 0;
    if (bits <= 64) {
        const uint64_t a = k0 >> (64 - bits), b = p0 >> (64 - bits);
        return a < b ? -1 : (a > b ? 1 : 0);
    }
    if (k0 != p0) return k0 < p0 ? -1 : 1;
    const uint64_t a = k1 >> (128 - bits), b = p1 >> (128 - bits);
    return a < b ? -1 : (a > b ? 1 : 0);
}

// The k heaviest of the emitted records: their row keys to `out`, in no
// particular order, their number to ctl->n_sel.
//
// First every record's (slot | part << 62 | parity << 63, row) becomes its
// rank key (~weight bits, ~order << order_shift): the reference's exact FP64
// weight and its visiting order (term index, then row).  Orders are below
// 2^(64 - order_shift), so the key's leading key_bits_total bits decide it.
// Records of zero weight (the reference drops them) get the all-ones weight
// key, which sorts after every other record, and are never taken.
//
// Then a radix select finds the k-th smallest rank key (keys are unique
// because visiting orders are): level by level a histogram of the next 11 key
// bits of the records that share the prefix chosen so far, whose digit every
// block picks for itself, so that a level is one grid barrier.  It stops as
// soon as the records of a digit are exactly the ones still needed.  Bins of
// three levels in turn: those of the next level are cleared while a level is
// counted, two barriers after they were last read.
//
// Nothing is done when the emission has to be repeated (more records than
// places, or fewer than k above a threshold): the host sees the same counts.
template <int W>
__global__ void __launch_bounds__(kTailThreads)
    find_select_kernel(uint64_t* __restrict__ rank, const uint64_t* __restrict__ keys, int64_t cap, PartView off,
                       PartView diag, const double2* __restrict__ psi, int64_t n_i, int order_shift,
                       int key_bits_total, int64_t k, FindCtl* ctl, unsigned int* bins, uint64_t* __restrict__ out) {
    __shared__ unsigned int s_bins[kSelectBins];
    __shared__ long long s_warp[32];
    __shared__ long long s_pick[3];  // digit, records below it, records at it
    const cg::grid_group grid = cg::this_grid();
    const int64_t e = (int64_t)ctl->n_emit;
    if (ctl->overflow || e > cap || e == 0 || (ctl->emit_from > 0 && e < k)) return;  // (the same for every block)
    const int lane = threadIdx.x & 31;
    const int64_t first = (int64_t)blockIdx.x * kTailThreads + threadIdx.x, step = (int64_t)gridDim.x * kTailThreads;
    const int64_t rounded = (e + 31) / 32 * 32;  // whole warps
    for (int64_t i = first; i < rounded; i += step) {
        bool zero = false;
        if (i < e) {
            const uint64_t info = rank[2 * i], row = rank[2 * i + 1];
            const int64_t slot = (int64_t)(info & ((1ull << 62) - 1));
            const bool in_diag = (info >> 62) & 1;
            const double w = exact_weight(__ldg((in_diag ? diag.coef : off.coef) + slot), __ldg(psi + row), (int)(info >> 63));
            const uint64_t order = (uint64_t)__ldg((in_diag ? diag.orig : off.orig) + slot) * (uint64_t)n_i + row;
            zero = w == 0.0;
            rank[2 * i] = zero ? ~0ull : ~(uint64_t)__double_as_longlong(w);
            rank[2 * i + 1] = (~order) << order_shift;
        }
        const unsigned z = __ballot_sync(0xffffffffu, zero);
        if (z != 0 && lane == 0) atomicAdd(&ctl->n_zero, (unsigned long long)__popc(z));
    }
    grid.sync();
    const int64_t valid = e - (int64_t)*(volatile unsigned long long*)&ctl->n_zero;
    int64_t need = k < valid ? k : valid;
    uint64_t p0 = 0, p1 = 0;
    int fixed = 0;
    // all of the valid records: those below the all-ones weight key
    const bool every = need == valid;
    for (int level = 0; !every && need > 0 && fixed < key_bits_total; ++level) {
        unsigned int* const mine = bins + level % 3 * kSelectBins;
        unsigned int* const next = bins + (level + 1) % 3 * kSelectBins;
        for (int64_t b = first; b < kSelectBins; b += step) next[b] = 0;
        const int cnt = key_bits_total - fixed < kSelectBits ? key_bits_total - fixed : kSelectBits;
        for (int b = threadIdx.x; b < kSelectBins; b += kTailThreads) s_bins[b] = 0;
        __syncthreads();
        for (int64_t i = first; i < e; i += step) {
            const uint64_t k0 = rank[2 * i], k1 = rank[2 * i + 1];
            if (prefix_cmp(k0, k1, p0, p1, fixed) == 0) atomicAdd(&s_bins[key_bits(k0, k1, fixed, cnt)], 1u);
        }
        __syncthreads();
        for (int b = threadIdx.x; b < kSelectBins; b += kTailThreads) {
            const unsigned int v = s_bins[b];
            if (v) atomicAdd(mine + b, v);
        }
        grid.sync();
        // the digit where the remaining count is reached: two bins a thread (2^31 records and more are summed)
        static_assert(kSelectBins == 2 * kTailThreads, "two bins a thread");
        const long long c0 = ((volatile unsigned int*)mine)[2 * threadIdx.x], c1 = ((volatile unsigned int*)mine)[2 * threadIdx.x + 1];
        const long long run = block_inclusive_scan(c0 + c1, s_warp);
        const long long before = run - c0 - c1;
        if (run >= need && before < need) {
            const bool second = before + c0 < need;
            s_pick[0] = 2 * threadIdx.x + (second ? 1 : 0);
            s_pick[1] = second ? before + c0 : before;
            s_pick[2] = second ? c1 : c0;
        }
        __syncthreads();
        const uint64_t d = (uint64_t)s_pick[0];
        if (fixed + cnt <= 64) {
            p0 |= d << (64 - fixed - cnt);
        } else if (fixed >= 64) {
            p1 |= d << (128 - fixed - cnt);
        } else {
            const int lo_bits = fixed + cnt - 64;
            p0 |= d >> lo_bits;
            p1 |= d << (64 - lo_bits);
        }
        need -= s_pick[1];
        fixed += cnt;
        if (s_pick[2] == need) break;
        __syncthreads();  // s_pick is written again
    }
    // the records up to the chosen prefix
    if (need <= 0) return;
    for (int64_t i = first; i < rounded; i += step) {
        bool take = false;
        if (i < e) {
            const uint64_t k0 = rank[2 * i], k1 = rank[2 * i + 1];
            take = every ? k0 != ~0ull : prefix_cmp(k0, k1, p0, p1, fixed) <= 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, take);
        unsigned long long base = 0;
        if (lane == 0 && m) base = atomicAdd(&ctl->n_sel, (unsigned long long)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (take) {
            const unsigned long long at = base + __popc(m & ((1u << lane) - 1u));
#pragma unroll
            for (int q = 0; q < W; ++q) out[at * W + q] = keys[i * W + q];
        }
    }
}

// Blocks of the sort for up to k rows: one per SM, fewer for few rows.
int64_t sort_blocks_for(int64_t k) {
    const int64_t b = (k + 255) / 256;
    return b < 1 ? 1 : b > 152 ? 152 : b;
}

// Sort ctl->n_sel keys (LSD radix, a row byte a pass, least significant
// first), keep the distinct ones and write them as rows of nq bytes.  Block b
// owns the b-th contiguous share of the keys and its warps contiguous pieces
// of that, so a pass is stable: count digits per warp; (barrier) every digit's
// counts are summed over the blocks by one warp; (barrier) every key goes
// behind the smaller digits, the same digit of earlier blocks and warps, and
// its own place within the warp; (barrier).  Keys travel alone, in two
// buffers.  counts: 256 x gridDim.x + 256 values.
template <int W>
__global__ void __launch_bounds__(kTailThreads)
    find_sort_kernel(uint64_t* keys, uint64_t* other, int32_t* counts, FindCtl* ctl, int nq, uint8_t* __restrict__ out) {
    __shared__ int32_t s_cnt[kTailWarps][256];
    __shared__ int32_t s_base[256];
    __shared__ int s_warp[32];
    const cg::grid_group grid = cg::this_grid();
    const int64_t n = (int64_t)ctl->n_sel;
    if (n == 0) return;  // (the same for every block)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int blocks = (int)gridDim.x, me = (int)blockIdx.x;
    int32_t* const totals = counts + 256 * (int64_t)blocks;
    const int64_t chunk = (n + blocks - 1) / blocks;
    const int64_t lo = (int64_t)me * chunk < n ? (int64_t)me * chunk : n;
    const int64_t hi = lo + chunk < n ? lo + chunk : n;
    const int64_t piece = ((hi - lo + kTailWarps - 1) / kTailWarps + 31) / 32 * 32;
    const int64_t wlo = lo + warp * piece < hi ? lo + warp * piece : hi;
    const int64_t whi = wlo + piece < hi ? wlo + piece : hi;
    uint64_t* src = keys;
    uint64_t* dst = other;
    for (int byte = nq - 1; byte >= 0; --byte) {
        const int word = byte >> 3, shift = 8 * (7 - (byte & 7));
        for (int d = lane; d < 256; d += 32) s_cnt[warp][d] = 0;
        __syncwarp();
        for (int64_t i = wlo + lane; i < whi; i += 32) atomicAdd(&s_cnt[warp][(unsigned)(src[i * W + word] >> shift) & 0xffu], 1);
        __syncthreads();
        if (threadIdx.x < 256) {
            int32_t run = 0;
            for (int w = 0; w < kTailWarps; ++w) {
                const int32_t c = s_cnt[w][threadIdx.x];
                s_cnt[w][threadIdx.x] = run;
                run += c;
            }
            counts[(int64_t)threadIdx.x * blocks + me] = run;
        }
        grid.sync();
        for (int d = me + warp * blocks; d < 256; d += kTailWarps * blocks) {
            int32_t before = 0;
            for (int b = 0; b < blocks; b += 32) {
                const int32_t c = b + lane < blocks ? counts[(int64_t)d * blocks + b + lane] : 0;
                int32_t x = c;
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const int32_t y = __shfl_up_sync(0xffffffffu, x, s);
                    if (lane >= s) x += y;
                }
                if (b + lane < blocks) counts[(int64_t)d * blocks + b + lane] = before + x - c;
                before += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) totals[d] = before;
        }
        grid.sync();
        const int total = threadIdx.x < 256 ? totals[threadIdx.x] : 0;
        const int up_to = block_inclusive_scan(total, s_warp);
        if (threadIdx.x < 256) s_base[threadIdx.x] = up_to - total + counts[(int64_t)threadIdx.x * blocks + me];
        __syncthreads();
        for (int64_t base = wlo; base < whi; base += 32) {
            const int64_t i = base + lane;
            const bool in = i < whi;
            uint64_t key[W];
#pragma unroll
            for (int q = 0; q < W; ++q) key[q] = in ? src[i * W + q] : 0;
            const unsigned d = in ? (unsigned)(src[i * W + word] >> shift) & 0xffu : 256u;
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            const int leader = __ffs(peers) - 1;
            int at = 0;
            if (in && lane == leader) {
                at = s_cnt[warp][d];
                s_cnt[warp][d] = at + __popc(peers);
            }
            at = __shfl_sync(0xffffffffu, at, leader);
            if (in) {
                const int64_t to = (int64_t)s_base[d] + at + __popc(peers & lt);
#pragma unroll
                for (int q = 0; q < W; ++q) dst[to * W + q] = key[q];
            }
            __syncwarp();
        }
        uint64_t* const t = src;
        src = dst;
        dst = t;
        grid.sync();
    }
    // the first of every run of equal keys
    auto head = [&](int64_t i) {
        bool h = i == 0;
#pragma unroll
        for (int q = 0; q < W; ++q) h = h || src[i * W + q] != src[(i - 1) * W + q];
        return h;
    };
    int heads = 0;
    for (int64_t base = wlo; base < whi; base += 32) {
        heads += __popc(__ballot_sync(0xffffffffu, base + lane < whi && head(base + lane)));
    }
    // places: heads of earlier blocks (counts[b]), of earlier warps, of earlier lanes
    const int in_block = block_inclusive_scan(lane == 0 ? heads : 0, s_warp);
    if (threadIdx.x == kTailThreads - 1) counts[me] = in_block;
    grid.sync();
    int earlier = 0, all = 0;
    for (int b = lane; b < blocks; b += 32) {
        const int c = counts[b];
        all += c;
        if (b < me) earlier += c;
    }
    earlier = (int)__reduce_add_sync(0xffffffffu, (unsigned)earlier);
    all = (int)__reduce_add_sync(0xffffffffu, (unsigned)all);
    int64_t at = earlier + __shfl_sync(0xffffffffu, in_block, 0) - heads;
    for (int64_t base = wlo; base < whi; base += 32) {
        const int64_t i = base + lane;
        const bool h = i < whi && head(i);
        const unsigned m = __ballot_sync(0xffffffffu, h);
        if (h) {
            uint8_t* r = out + (at + __popc(m & lt)) * nq;
            for (int b = 0; b < nq; ++b) r[b] = (uint8_t)(src[i * W + (b >> 3)] >> (8 * (7 - (b & 7))));
        }
        at += __popc(m);
    }
    if (me == 0 && threadIdx.x == 0) ctl->n_unique = (unsigned long long)all;
}

__global__ void zero_u64_kernel(unsigned long long* p, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = 0;
}

struct FindArgs {
    const void* table_host;
    const void* table_dev;
    const uint8_t* configs_i;
    const double* psi_i;
    int64_t n_i;
    int64_t k;
    const uint8_t* configs_ex;
    int64_t n_ex;
    uint8_t* out;
    int64_t* n_out;
};

// Workspace layout: fixed part (exclude set, packed rows, histogram, control
// block, the selected rows and their sort), then the emission area of cap
// records.
template <int W>
struct FindLayout {
    HashRows excl;
    uint64_t* keys_i;
    uint64_t* keys_s;       // every kSampleStride-th row of keys_i
    double2* psi_s;         // and its amplitude
    unsigned long long* hist;  // bucket counts; the selection's bins afterwards
    FindCtl* ctl;
    unsigned long long* deep;
    LongGroup* queue;
    uint64_t* sel_keys;     // the selected rows' keys, and the buffer they are sorted with
    uint64_t* sort_keys;
    int32_t* sort_counts;
    // emission area
    uint64_t* emit_rank;
    uint64_t* emit_keys;
};

// Places for rests of groups: a few rows with most of the weight have one in each of their groups.
unsigned int queue_places(int64_t n_i) {
    const int64_t places = 64 * n_i;
    return (unsigned int)(places < 1024 ? 1024 : places < (1 << 18) ? places : 1 << 18);
}

template <int W>
FindLayout<W> take_find(Arena& ws, int64_t n_i, int64_t k, int64_t n_ex, int64_t cap) {
    FindLayout<W> L;
    L.excl = take_hashrows<W>(ws, n_ex);
    L.keys_i = ws.take<uint64_t>((uint64_t)(n_i > 0 ? n_i : 1) * W);
    const int64_t n_s = n_i / kSampleStride + 1;
    L.keys_s = ws.take<uint64_t>((uint64_t)n_s * W);
    L.psi_s = ws.take<double2>((uint64_t)n_s);
    L.hist = ws.take<unsigned long long>(kBuckets);
    L.ctl = ws.take<FindCtl>(1);
    L.deep = ws.take<unsigned long long>(kBuckets);
    L.queue = ws.take<LongGroup>(queue_places(n_i));
    int64_t kk = k > 0 ? k : 1;
    L.sel_keys = ws.take<uint64_t>((uint64_t)kk * W);
    L.sort_keys = ws.take<uint64_t>((uint64_t)kk * W);
    L.sort_counts = ws.take<int32_t>(256 * (uint64_t)sort_blocks_for(kk) + 256);
    int64_t c = cap > 0 ? cap : 1;
    L.emit_rank = ws.take<uint64_t>((uint64_t)c * 2);
    L.emit_keys = ws.take<uint64_t>((uint64_t)c * W);
    return L;
}

template <int W>
int find_impl(const FindArgs& a, void* workspace, uint64_t workspace_bytes, uint64_t* needed, cudaStream_t s) {
    const qmbx_table_header* h = header_of(a.table_host);
    const int nq = h->n_qubytes;
    const int64_t k = a.k;
    // emission capacity: the most records the workspace can hold (the
    // layout grows monotonically with the capacity, so bisect), such that a
    // workspace sized for c records by this layout holds at least c
    auto fits = [&](int64_t c) {
        Arena trial(nullptr, 0);
        take_find<W>(trial, a.n_i, k, a.n_ex, c);
        return trial.used <= workspace_bytes;
    };
    int64_t cap = 1;
    if (fits(1)) {
        int64_t hi = (int64_t)(workspace_bytes / 16) + 2;  // a record takes more than 16 bytes
        while (cap < hi) {
            const int64_t mid = cap + (hi - cap + 1) / 2;
            if (fits(mid)) {
                cap = mid;
            } else {
                hi = mid - 1;
            }
        }
    }
    Arena ws(workspace, workspace_bytes);
    FindLayout<W> L = take_find<W>(ws, a.n_i, k, a.n_ex, cap);
    if (workspace == nullptr || !ws.fits()) {
        if (needed) *needed = ws.used;
        return fail(QMBX_ERR_WORKSPACE, "find_relative needs at least %llu bytes of workspace",
                    (unsigned long long)ws.used);
    }
    *a.n_out = 0;
    g_find_stats = FindStats{};
    if (k == 0 || a.n_i == 0) return QMBX_OK;
    int st;
    // the exclusion set is only looked up: no first rows, no list of distinct ones
    if ((st = build_hashset<W>(a.configs_ex, nq, L.excl, s)) != QMBX_OK) return st;
    const uint64_t* keys_i = L.excl.keys;
    if (a.configs_i != a.configs_ex || a.n_i > a.n_ex) {
        if ((st = pack_rows<W>(a.configs_i, a.n_i, nq, L.keys_i, s)) != QMBX_OK) return st;
        keys_i = L.keys_i;
    }
    // hist, ctl and deep lie one behind the other
    QMBX_CUDA_TRY(cudaMemsetAsync(L.hist, 0, (size_t)(reinterpret_cast<char*>(L.deep + kBuckets) - reinterpret_cast<char*>(L.hist)), s));

    RelativeArgs r{};
    r.psi = reinterpret_cast<const double2*>(a.psi_i);
    r.n_i = a.n_i;
    r.excl = L.excl.hash();
    r.off = part_view(a.table_host, a.table_dev, QMBX_PART_FWD);
    r.diag = part_view(a.table_host, a.table_dev, QMBX_PART_DIAG);
    r.hist = L.hist;
    r.hist_exact = 1;
    r.deep = L.deep;
    r.queue = L.queue;
    r.queue_cap = queue_places(a.n_i);
    r.ctl = L.ctl;
    r.cap_emit = cap;
    r.emit_rank = L.emit_rank;
    r.emit_keys = L.emit_keys;
    auto need_bytes = [&](unsigned long long records) {
        Arena want(nullptr, 0);
        take_find<W>(want, a.n_i, k, a.n_ex, (int64_t)records);
        return want.used;
    };

    // pass 1: bucket counts over every row, or every kSampleStride-th row of
    // large inputs; the threshold is chosen on the device (no host round trip)
    const bool sampled = a.n_i >= kSampleMinRows;
    const bool bounded = relative_bounded(r.off);
    if (sampled) {
        const int64_t n_s = (a.n_i + kSampleStride - 1) / kSampleStride;
        QMBX_KERNEL(kGroupOther, s, sample_rows_kernel<W><<<grid_for(n_s, kThreads), kThreads, 0, s>>>(keys_i, r.psi, n_s, L.keys_s, L.psi_s));
        QMBX_LAUNCH_CHECK("sample_rows_kernel");
        RelativeArgs rs = r;
        rs.psi = L.psi_s;
        rs.n_i = n_s;
        rs.hist_exact = 0;  // an estimate: every record counted, no exclusion lookups
        // aim at about twice k records above the chosen bucket, one more bucket of slack
        if (bounded) {
            if ((st = launch_threshold<W>(rs, L.keys_s, n_s, k, a.n_i, 2.0 * (double)k, s)) != QMBX_OK) return st;
        } else {
            if ((st = launch_relative<W, false>(rs, L.keys_s, n_s, s)) != QMBX_OK) return st;
            QMBX_KERNEL(kGroupSelect, s, choose_emit_kernel<<<1, kChooseThreads, 0, s>>>(L.hist, (double)a.n_i / (double)n_s, 2.0 * (double)k, L.ctl));
        }
    } else {
        RelativeArgs r1 = r;
        r1.hist_exact = 0;
        if (bounded) {
            if ((st = launch_threshold<W>(r1, keys_i, a.n_i, k, a.n_i, (double)k, s)) != QMBX_OK) return st;
        } else {
            if ((st = launch_relative<W, false>(r1, keys_i, a.n_i, s)) != QMBX_OK) return st;
            QMBX_KERNEL(kGroupSelect, s, choose_emit_kernel<<<1, kChooseThreads, 0, s>>>(L.hist, 1.0, (double)k, L.ctl));
        }
    }
    ++g_find_stats.walks;
    QMBX_LAUNCH_CHECK("find_relative threshold");

    // bits of the visiting order (term index * n_i + row < n_terms * n_i), in whole bytes
    int order_bytes = 1;
    {
        const double span = (double)(h->n_terms > 0 ? h->n_terms : 1) * (double)a.n_i;
        while (order_bytes < 8 && span > std::ldexp(1.0, 8 * order_bytes)) ++order_bytes;
    }
    int order_shift = 64 - 8 * order_bytes;
    int key_bits_total = 64 + 8 * order_bytes;
    const int sms = pivot_grid() / 4;
    // pass 2: emit the records at or above emit_from, select and sort.  Every
    // record down to the k-th was emitted when at least k were (or the
    // threshold is the lowest bucket); otherwise the sample put the threshold
    // too high, nothing is selected, and an unsampled histogram pass gives the
    // exact one for a second round (never seen on the benchmark shapes; the
    // tests drive it).
    FindCtl ctl{};
    for (int attempt = 0;; ++attempt) {
        st = bounded ? launch_emit<W>(r, keys_i, a.n_i, k, s) : launch_relative<W, true>(r, keys_i, a.n_i, s);
        if (st != QMBX_OK) return st;
        ++g_find_stats.walks;
        unsigned int* bins = reinterpret_cast<unsigned int*>(L.hist);  // left cleared by the threshold
        {
            int64_t n_i = a.n_i, want = k, places = cap;
            const double2* psi = r.psi;
            void* args[] = {&L.emit_rank, &L.emit_keys, &places, &r.off, &r.diag, &psi, &n_i, &order_shift,
                            &key_bits_total, &want, &L.ctl, &bins, &L.sel_keys};
            QMBX_KERNEL(kGroupSelect, s, QMBX_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)find_select_kernel<W>, dim3(sms), dim3(kTailThreads), args, 0, s)));
        }
        {
            int bytes = nq;
            uint8_t* out = a.out;
            void* args[] = {&L.sel_keys, &L.sort_keys, &L.sort_counts, &L.ctl, &bytes, &out};
            const int64_t blocks = sort_blocks_for(k) < sms ? sort_blocks_for(k) : sms;
            QMBX_KERNEL(kGroupSort, s, QMBX_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)find_sort_kernel<W>, dim3((unsigned)blocks), dim3(kTailThreads), args, 0, s)));
        }
        QMBX_CUDA_TRY(cudaMemcpyAsync(&ctl, L.ctl, sizeof(FindCtl), cudaMemcpyDeviceToHost, s));
        QMBX_CUDA_TRY(cudaStreamSynchronize(s));
        if (ctl.overflow || (int64_t)ctl.n_emit > cap) {
            if (needed) *needed = need_bytes(ctl.n_emit);
            return fail(QMBX_ERR_WORKSPACE, "find_relative needs %llu bytes of workspace for %llu records near the threshold",
                        (unsigned long long)need_bytes(ctl.n_emit), ctl.n_emit);
        }
        if (ctl.emit_from == 0 || (int64_t)ctl.n_emit >= k) break;  // every record down to the k-th was kept
        if (attempt > 0) return fail(QMBX_ERR_DEVICE, "find_relative threshold did not settle");
        // the exact threshold from the counts of every record
        QMBX_KERNEL(kGroupOther, s, zero_u64_kernel<<<grid_for(kBuckets, kThreads), kThreads, 0, s>>>(L.hist, kBuckets));
        if ((st = launch_relative<W, false>(r, keys_i, a.n_i, s)) != QMBX_OK) return st;
        ++g_find_stats.walks;
        QMBX_CUDA_TRY(cudaMemsetAsync(L.ctl, 0, sizeof(FindCtl), s));
        QMBX_KERNEL(kGroupSelect, s, choose_emit_kernel<<<1, kChooseThreads, 0, s>>>(L.hist, 1.0, (double)k, L.ctl));
        QMBX_LAUNCH_CHECK("choose_emit_kernel");
    }
    const int64_t keep = (int64_t)ctl.n_sel;
    if (keep > k) return fail(QMBX_ERR_DEVICE, "find_relative selected %lld records for %lld places", (long long)keep, (long long)k);
    g_find_stats.records = (int64_t)ctl.n_emit;
    g_find_stats.selected = keep;
    if (keep > 0) {
        // per pass: the selected keys read and written
        g_find_stats.sort_passes = nq;
        g_find_stats.sort_bytes = (int64_t)nq * 2 * keep * 8 * W;
    }
    *a.n_out = (int64_t)ctl.n_unique;
    g_find_stats.rows_out = (int64_t)ctl.n_unique;
    return QMBX_OK;
}

// ---------------------------------------------------------------------------
// single_relative
// ---------------------------------------------------------------------------

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// key factor log(u_t) / |coef_t| of every changing term (-inf for zero coefficients)
__global__ void es_factor_kernel(const double2* __restrict__ coef, const int32_t* __restrict__ orig, int64_t n,
                                 uint64_t seed, double* __restrict__ kf) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double2 c = coef[i];
    double w = sqrt(c.x * c.x + c.y * c.y);
    uint64_t bits = splitmix64(seed ^ splitmix64((uint64_t)orig[i]));
    double u = (double)((bits >> 11) + 1) * (1.0 / 9007199254740992.0);
    kf[i] = w > 0.0 ? log(u) / w : -INFINITY;
}

template <int W>
struct SingleVisitor : VisitorBase {
    static constexpr bool kProbe = true;
    HashView lookup;  // the input rows
    const double* kf;
    const int32_t* orig;
    uint8_t* out;
    int nq;
    const int32_t* rows;  // walked rows (NULL: every row)
    struct Acc {
        double key;
        int32_t term;
        Key<W> best;
    };
    __device__ __forceinline__ void init(Acc& a, int64_t, const Key<W>&, int*) const {
        a.key = -INFINITY;
        a.term = -1;
#pragma unroll
        for (int q = 0; q < W; ++q) a.best.w[q] = 0;
    }
    __device__ __forceinline__ bool take(Acc& a, const Key<W>&, const Key<W>& img, int, int64_t slot, int64_t pos,
                                         int2&) const {
        if (pos >= 0) return false;
        const double key = __ldg(kf + slot);
        const int32_t t = __ldg(orig + slot);
        if (a.term < 0 || key > a.key || (key == a.key && t < a.term)) {
            a.key = key;
            a.term = t;
            a.best = img;
        }
        return false;
    }
    __device__ __forceinline__ void visit(Acc& a, const Key<W>&, const Key<W>& img, int, int64_t slot) const {
        const double key = __ldg(kf + slot);
        const int32_t t = __ldg(orig + slot);
        const bool better = a.term < 0 || key > a.key || (key == a.key && t < a.term);
        if (!better) return;
        if (hash_find<W>(lookup, img) >= 0) return;
        a.key = key;
        a.term = t;
        a.best = img;
    }
    __device__ __forceinline__ void visit_diag(Acc&, const Key<W>&, int, int64_t) const {}
    // warp argmax of (key, lowest term) carrying the image
    __device__ __forceinline__ void reduce(Acc& a) const {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            double k2 = __shfl_xor_sync(0xffffffffu, a.key, d);
            int32_t t2 = __shfl_xor_sync(0xffffffffu, a.term, d);
            Key<W> b2;
#pragma unroll
            for (int q = 0; q < W; ++q) b2.w[q] = __shfl_xor_sync(0xffffffffu, a.best.w[q], d);
            bool take = t2 >= 0 && (a.term < 0 || k2 > a.key || (k2 == a.key && t2 < a.term));
            if (take) {
                a.key = k2;
                a.term = t2;
                a.best = b2;
            }
        }
    }
    __device__ __forceinline__ void finish(Acc& a, int64_t row, const Key<W>&) const {
        uint8_t* r = out + (rows != nullptr ? (int64_t)__ldg(rows + row) : row) * nq;
        for (int b = 0; b < nq; ++b) r[b] = (uint8_t)(a.best.w[b >> 3] >> (8 * (7 - (b & 7))));
    }
};

// ---------------------------------------------------------------------------
// single_relative by the terms in key order.  A term's key is the same for
// every row, so a row's neighbour is given by the first term, in descending
// key order, that applies and leads outside the input.  Terms apply to a few
// per cent of the rows, so a row finds it among the first hundred or so: the
// best thousand terms are gathered and sorted once, and a warp takes a
// row through them 32 at a time.  Rows that find none there are walked.
//   20,000 rows under 55,371 terms: walk 648 us; bins, gather, sort and rows 26 us
// ---------------------------------------------------------------------------

constexpr int kBestTerms = 1024;
constexpr int kKeyBins = 1 << 14;  // exponent and three mantissa bits of |key|: bins of a ratio of at most 1.125

struct BestTerm {
    unsigned long long key;  // |key| as ordered bits: the smallest is the best
    int32_t orig, slot;      // input order breaks ties
};

struct SingleCtl {
    int gathered;   // terms in the list
    int unresolved; // rows to walk
};

__device__ __forceinline__ unsigned long long single_key(double kf) {
    return (unsigned long long)__double_as_longlong(fabs(kf));  // keys are log(u) / |coef| <= 0
}

__global__ void single_bins_kernel(const double* __restrict__ kf, int64_t n, int* __restrict__ bins) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int bin = i < n ? (int)(single_key(kf[i]) >> 49) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    if (bin >= 0 && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(bins + bin, __popc(peers));
}

// The terms of the lowest bins that together hold at most kBestTerms.  Every
// block finds the last such bin for itself.
__global__ void __launch_bounds__(kTailThreads) single_gather_kernel(const double* __restrict__ kf,
                                                                     const int32_t* __restrict__ orig, int64_t n,
                                                                     const int* __restrict__ bins,
                                                                     BestTerm* __restrict__ best,
                                                                     SingleCtl* __restrict__ ctl) {
    __shared__ int s_warp[32];
    __shared__ int s_end;  // first bin left out
    constexpr int kPer = kKeyBins / kTailThreads;
    if (threadIdx.x == 0) s_end = kKeyBins;
    int mine[kPer];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; k += 4) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(bins + kPer * threadIdx.x + k));
        mine[k] = v.x;
        mine[k + 1] = v.y;
        mine[k + 2] = v.z;
        mine[k + 3] = v.w;
        sum += v.x + v.y + v.z + v.w;
    }
    const int run = block_inclusive_scan(sum, s_warp);
    if (run > kBestTerms && run - sum <= kBestTerms) {
        int upto = run - sum, end = kPer * threadIdx.x;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            upto += mine[k];
            if (upto <= kBestTerms) end = kPer * threadIdx.x + k + 1;
        }
        s_end = end;
    }
    __syncthreads();
    const int end = s_end;
    for (int64_t i = (int64_t)blockIdx.x * kTailThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kTailThreads) {
        const unsigned long long key = single_key(kf[i]);
        if ((int)(key >> 49) >= end) continue;
        BestTerm t;
        t.key = key;
        t.orig = __ldg(orig + i);
        t.slot = (int32_t)i;
        best[atomicAdd(&ctl->gathered, 1)] = t;
    }
}

// Sort the gathered terms by (key, input order), which no two share: a warp
// counts the terms ahead of one.  (A bitonic sort of 4,096 terms in one block
// took 112 us; the counts of 1,024 take a few.)
// The terms' tests go with them: word q of the k-th term at tests[q kBestTerms + k].
__global__ void __launch_bounds__(kThreads) single_sort_kernel(const BestTerm* __restrict__ best,
                                                               const SingleCtl* __restrict__ ctl, PartView off, int words,
                                                               BestTerm* __restrict__ sorted,
                                                               ulonglong2* __restrict__ tests) {
    __shared__ unsigned long long s_key[kBestTerms];
    __shared__ int32_t s_orig[kBestTerms];
    const int n = ctl->gathered;
    if ((int)blockIdx.x * kWarpsPerBlock >= n) return;
    for (int i = threadIdx.x; i < n; i += kThreads) {
        s_key[i] = best[i].key;
        s_orig[i] = best[i].orig;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int me = (int)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (me >= n) return;
    const unsigned long long key = s_key[me];
    const int32_t orig = s_orig[me];
    unsigned ahead = 0;
    for (int i = lane; i < n; i += 32) ahead += s_key[i] < key || (s_key[i] == key && s_orig[i] < orig) ? 1u : 0u;
    ahead = __reduce_add_sync(0xffffffffu, ahead);
    if (lane == 0) sorted[ahead] = best[me];
    if (lane < words) tests[lane * kBestTerms + ahead] = __ldg(off.test + (int64_t)lane * off.stride + best[me].slot);
}

// A warp takes a row through the terms in order, 32 at first and up to
// kSingleStep at a time: those that apply queue up, and the images of 32 of
// them are looked up at once.  The terms' tests lie in order, so that a warp
// reads 32 in four lines.  On sets whose rows have no relative the terms are
// tried in vain: on every determinant of 3 + 3 electrons in 14 orbitals (the
// walk alone 2.43 ms) 2,048 terms gathered from the table's own places took
// the call to 3.24 ms, in order to 2.91, and 1,024 in order to 2.74.
constexpr int kSingleStep = 256;

template <int W>
__global__ void __launch_bounds__(kThreads) single_first_kernel(const uint64_t* __restrict__ keys, int64_t n, HashView set,
                                                                PartView off, const BestTerm* __restrict__ best,
                                                                const ulonglong2* __restrict__ tests,
                                                                SingleCtl* __restrict__ ctl,
                                                                int32_t* __restrict__ unresolved, int nq,
                                                                uint8_t* __restrict__ out) {
    __shared__ int32_t s_term[kWarpsPerBlock][kSingleStep];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int32_t* queue = s_term[threadIdx.x >> 5];
    const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (row >= n) return;
    const int terms = ctl->gathered;
    const Key<W> c = load_key<W>(keys, row);
    for (int base = 0, step = 32; base < terms; base += step, step = base < kSingleStep ? base : kSingleStep) {
        int waiting = 0;
        __syncwarp();  // the queue has been read
        for (int at = base; at < base + step && at < terms; at += 32) {
            bool on = at + lane < terms;
            if (on) {
                uint64_t bad = 0;
#pragma unroll
                for (int q = 0; q < W; ++q) {
                    const ulonglong2 test = __ldg(tests + q * kBestTerms + at + lane);
                    bad |= (c.w[q] ^ test.y) & test.x;
                }
                on = bad == 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) queue[waiting + __popc(m & lt)] = at + lane;
            waiting += __popc(m);
        }
        __syncwarp();
        for (int k = 0; k < waiting; k += 32) {
            bool out_of_set = false;
            Key<W> img{};
            if (k + lane < waiting) {
                TermRec<W> rec;
                load_apply<W>(rec, off, __ldg(&best[queue[k + lane]].slot));
                rec.image(c, img);
                out_of_set = hash_find<W>(set, img) < 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, out_of_set);
            if (m != 0) {
                if (lane == __ffs(m) - 1) {
                    uint8_t* r = out + row * nq;
                    for (int b = 0; b < nq; ++b) r[b] = (uint8_t)(img.w[b >> 3] >> (8 * (7 - (b & 7))));
                }
                return;
            }
        }
    }
    if (lane == 0) unresolved[atomicAdd(&ctl->unresolved, 1)] = (int32_t)row;
}

// The rows of a list.
template <int W>
struct ListedRows {
    const uint64_t* keys;
    const int32_t* rows;
    __device__ __forceinline__ Key<W> get(int64_t i) const { return load_key<W>(keys, __ldg(rows + i)); }
};

template <int W>
struct SingleLayout {
    HashRows set;
    double* kf;
};

// Behind it, for calls by the terms in key order.
struct SingleOrder {
    SingleCtl* ctl;  // followed by the bins, cleared together
    int* bins;
    BestTerm* best;
    BestTerm* sorted;
    ulonglong2* tests;
    int32_t* unresolved;
};

SingleOrder take_single_order(Arena& ws, int64_t n, int words) {
    SingleOrder o;
    o.ctl = ws.take<SingleCtl>(1);
    o.bins = ws.take<int>(kKeyBins);
    o.best = ws.take<BestTerm>(kBestTerms);
    o.sorted = ws.take<BestTerm>(kBestTerms);
    o.tests = ws.take<ulonglong2>((uint64_t)words * kBestTerms);
    o.unresolved = ws.take<int32_t>((uint64_t)(n > 0 ? n : 1));
    return o;
}

// Whether rows are taken through the terms in key order: where the walks would
// visit enough terms to outweigh ordering them.  (rows x terms, whole calls by
// the walk and in order, us: 400 x 55,371, rows of 10, 175 and 84, of 4, 68
// and 82; 1,500 x 14,251 100 and 90; 6,000 x 14,251 121 and 91; below the line
// 200 x 55,371 171 by the walk.)
bool single_ordered(const PartView& off, int64_t n) {
    const char* e = getenv("QMBX_WALK");
    const char f = e != nullptr ? e[0] : 0;
    if (f == 't' || f == 'g' || f == 'p') return false;
    return off.n >= kGroupedMinTerms && (double)n * (double)off.n > 2e7;
}

template <int W>
SingleLayout<W> take_single(Arena& ws, int64_t n, int64_t n_off) {
    SingleLayout<W> L;
    L.set = take_hashrows<W>(ws, n);
    L.kf = ws.take<double>((uint64_t)(n_off > 0 ? n_off : 1));
    return L;
}

template <int W>
int single_impl(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n, uint64_t seed,
                uint8_t* out, Arena& ws, cudaStream_t s) {
    const qmbx_table_header* h = header_of(table_host);
    PartView off = part_view(table_host, table_dev, QMBX_PART_FWD);
    SingleLayout<W> L = take_single<W>(ws, n, h->part[QMBX_PART_FWD].n);
    if (ws.base == nullptr) return QMBX_OK;
    if (!ws.fits()) return fail(QMBX_ERR_WORKSPACE, "single_relative needs %llu bytes of workspace", (unsigned long long)ws.used);
    if (n == 0) return QMBX_OK;
    int st;
    // the set is only looked up: no first rows, no list of distinct ones
    if ((st = build_hashset<W>(configs, h->n_qubytes, L.set, s)) != QMBX_OK) return st;
    if (off.n > 0) {
        QMBX_KERNEL(kGroupOther, s, es_factor_kernel<<<grid_for(off.n, kThreads), kThreads, 0, s>>>(off.coef, off.orig, off.n, seed, L.kf));
        QMBX_LAUNCH_CHECK("es_factor_kernel");
    }
    PartView none = off;
    none.n = 0;
    SingleVisitor<W> v{{}, L.set.hash(), L.kf, off.orig, out, h->n_qubytes, nullptr};
    Arena behind = ws;
    const SingleOrder o = take_single_order(behind, n, W);
    if (single_ordered(off, n) && behind.fits()) {
        QMBX_CUDA_TRY(cudaMemsetAsync(o.ctl, 0, (size_t)(reinterpret_cast<char*>(o.bins + kKeyBins) - reinterpret_cast<char*>(o.ctl)), s));
        const unsigned blocks = grid_for(off.n, kTailThreads) < 152u ? grid_for(off.n, kTailThreads) : 152u;
        QMBX_KERNEL(kGroupSelect, s, single_bins_kernel<<<grid_for(off.n, kThreads), kThreads, 0, s>>>(L.kf, off.n, o.bins));
        QMBX_KERNEL(kGroupSelect, s, single_gather_kernel<<<blocks, kTailThreads, 0, s>>>(L.kf, off.orig, off.n, o.bins, o.best, o.ctl));
        QMBX_KERNEL(kGroupSort, s, single_sort_kernel<<<kBestTerms / kWarpsPerBlock, kThreads, 0, s>>>(o.best, o.ctl, off, W, o.sorted, o.tests));
        QMBX_KERNEL(kGroupEnumerate, s, single_first_kernel<W><<<grid_for(n, kWarpsPerBlock), kThreads, 0, s>>>(L.set.keys, n, L.set.hash(), off, o.sorted, o.tests, o.ctl, o.unresolved, h->n_qubytes, out));
        // rows that none of these terms serves: the walk over all terms
        v.rows = o.unresolved;
        ListedRows<W> rest{L.set.keys, o.unresolved};
        QMBX_KERNEL(kGroupOther, s, grouped_kernel<W><<<grouped_grid(n), kThreads, 0, s>>>(v, rest, &o.ctl->unresolved, n, off, none));
        QMBX_LAUNCH_CHECK("single_relative by terms in key order");
        return QMBX_OK;
    }
    KeyRows<W> src{L.set.keys};
    if (choose_walk(off, n, false) == Walk::kGrouped) {
        QMBX_KERNEL(kGroupEnumerate, s, grouped_kernel<W><<<grouped_grid(n), kThreads, 0, s>>>(v, src, nullptr, n, off, none));
    } else {
        QMBX_KERNEL(kGroupEnumerate, s, enumerate_kernel<W><<<grid_for(n, kThreads), kThreads, 0, s>>>(v, src, nullptr, n, off, none));
    }
    QMBX_LAUNCH_CHECK("single_relative enumeration");
    return QMBX_OK;
}

int check_ws(void* workspace) {
    if (workspace != nullptr && reinterpret_cast<uintptr_t>(workspace) % QMBX_ALIGN != 0) {
        return fail(QMBX_ERR_ARGUMENT, "workspace must be %d-byte aligned", QMBX_ALIGN);
    }
    return QMBX_OK;
}

}  // namespace
}  // namespace qmbx

using namespace qmbx;

extern "C" int qmbx_find_relative_workspace(const void* table_host, int64_t n_i, int64_t count_selected,
                                            int64_t n_exclude, uint64_t* bytes) {
    clear_error();
    const qmbx_table_header* h = header_of(table_host);
    if (h == nullptr || h->magic != QMBX_MAGIC) return fail(QMBX_ERR_ARGUMENT, "not a compiled qmbx table");
    if (bytes == nullptr) return fail(QMBX_ERR_ARGUMENT, "bytes must not be NULL");
    int64_t k = count_selected > 0 ? count_selected : 0;
    int64_t cap = 4 * k + (1 << 16);
    Arena probe(nullptr, 0);
    switch (h->n_words) {
        case 1: take_find<1>(probe, n_i, k, n_exclude, cap); break;
        case 2: take_find<2>(probe, n_i, k, n_exclude, cap); break;
        case 3: take_find<3>(probe, n_i, k, n_exclude, cap); break;
        case 4: take_find<4>(probe, n_i, k, n_exclude, cap); break;
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
    *bytes = probe.used;
    return QMBX_OK;
}

extern "C" int qmbx_find_relative(const void* table_host, const void* table_dev, const uint8_t* configs_i,
                                  const double* psi_i, int64_t n_i, int64_t count_selected,
                                  const uint8_t* configs_exclude, int64_t n_exclude, uint8_t* out, int64_t* n_out,
                                  void* workspace, uint64_t workspace_bytes, uint64_t* workspace_needed,
                                  qmbx_stream_t stream) {
    clear_error();
    int st = check_table(table_host, table_dev);
    if (st != QMBX_OK) return st;
    if (n_out == nullptr) return fail(QMBX_ERR_ARGUMENT, "n_out must not be NULL");
    if (count_selected < 0) return fail(QMBX_ERR_ARGUMENT, "count_selected must not be negative");
    if (count_selected >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "count_selected too large");
    if (n_i < 0 || n_i >= (int64_t(1) << 31) || n_exclude < 0 || n_exclude >= (int64_t(1) << 31)) {
        return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    }
    if ((n_i > 0 && (configs_i == nullptr || psi_i == nullptr)) || (n_exclude > 0 && configs_exclude == nullptr)) {
        return fail(QMBX_ERR_ARGUMENT, "input pointers must not be NULL");
    }
    if (count_selected > 0 && out == nullptr) return fail(QMBX_ERR_ARGUMENT, "out must not be NULL");
    if ((st = check_ws(workspace)) != QMBX_OK) return st;
    if (workspace == nullptr) workspace_bytes = 0;
    FindArgs a{table_host, table_dev, configs_i, psi_i, n_i, count_selected, configs_exclude, n_exclude, out, n_out};
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    switch (header_of(table_host)->n_words) {
        case 1: return find_impl<1>(a, workspace, workspace_bytes, workspace_needed, s);
        case 2: return find_impl<2>(a, workspace, workspace_bytes, workspace_needed, s);
        case 3: return find_impl<3>(a, workspace, workspace_bytes, workspace_needed, s);
        case 4: return find_impl<4>(a, workspace, workspace_bytes, workspace_needed, s);
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
}

extern "C" int qmbx_find_relative_stats(int64_t stats[6]) {
    clear_error();
    if (stats == nullptr) return fail(QMBX_ERR_ARGUMENT, "stats must not be NULL");
    const FindStats& f = g_find_stats;
    stats[0] = f.records;
    stats[1] = f.walks;
    stats[2] = f.sort_passes;
    stats[3] = f.sort_bytes;
    stats[4] = f.selected;
    stats[5] = f.rows_out;
    return QMBX_OK;
}

extern "C" int qmbx_single_relative_workspace(const void* table_host, int64_t n, uint64_t* bytes) {
    clear_error();
    const qmbx_table_header* h = header_of(table_host);
    if (h == nullptr || h->magic != QMBX_MAGIC) return fail(QMBX_ERR_ARGUMENT, "not a compiled qmbx table");
    if (bytes == nullptr) return fail(QMBX_ERR_ARGUMENT, "bytes must not be NULL");
    Arena probe(nullptr, 0);
    int64_t n_off = h->part[QMBX_PART_FWD].n;
    switch (h->n_words) {
        case 1: take_single<1>(probe, n, n_off); break;
        case 2: take_single<2>(probe, n, n_off); break;
        case 3: take_single<3>(probe, n, n_off); break;
        case 4: take_single<4>(probe, n, n_off); break;
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
    take_single_order(probe, n, h->n_words);
    *bytes = probe.used;
    return QMBX_OK;
}

extern "C" int qmbx_single_relative(const void* table_host, const void* table_dev, const uint8_t* configs, int64_t n,
                                    uint64_t seed, uint8_t* out, void* workspace, uint64_t workspace_bytes,
                                    qmbx_stream_t stream) {
    clear_error();
    int st = check_table(table_host, table_dev);
    if (st != QMBX_OK) return st;
    if (n < 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (n > 0 && (configs == nullptr || out == nullptr)) return fail(QMBX_ERR_ARGUMENT, "pointers must not be NULL");
    if ((st = check_ws(workspace)) != QMBX_OK) return st;
    if (workspace == nullptr) return fail(QMBX_ERR_WORKSPACE, "single_relative needs a workspace");
    Arena ws(workspace, workspace_bytes);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    switch (header_of(table_host)->n_words) {
        case 1: return single_impl<1>(table_host, table_dev, configs, n, seed, out, ws, s);
        case 2: return single_impl<2>(table_host, table_dev, configs, n, seed, out, ws, s);
        case 3: return single_impl<3>(table_host, table_dev, configs, n, seed, out, ws, s);
        case 4: return single_impl<4>(table_host, table_dev, configs, n, seed, out, ws, s);
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
}

// ---------------------------------------------------------------------------
// The Epstein-Nesbet PT2 step of qmb/pert.py:37-61 in one call:
//   E0 = Re<psi|H|psi> / <psi|psi> over configs,
//   other = find_relative(configs, psi, count_selected, configs),
//   E2 = sum_j |(H psi)_j|^2 / <psi|psi> / (E0 - Re H_jj) over other.
// The reference walks the terms four times: apply_within for E0,
// find_relative, apply_within onto other, and diagonal_term.  Here
// find_relative runs as on its own, and one apply_within from configs onto
// configs and the selected rows together gives both E0's H psi and the
// selected rows' (configs and the selected rows are disjoint).  The
// selected rows' diagonal terms follow.  E0 never leaves the device.
// ---------------------------------------------------------------------------

namespace qmbx {
namespace {

constexpr int kPt2Blocks = 1024;

// Deterministic block sum of one double per thread (blockDim.x a multiple of 32, at most 1024).
__device__ __forceinline__ double block_sum(double x, double* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    x = warp_sum(x);
    if (lane == 0) s_warp[warp] = x;
    __syncthreads();
    double t = lane < nwarps ? s_warp[lane] : 0.0;
    if (warp == 0) t = warp_sum(t);
    __syncthreads();
    return t;  // valid in warp 0
}

// sums[0] = E0 = Re<psi|H psi> / norm over the n configs, sums[1] = norm = <psi|psi>
__global__ void pt2_e0_kernel(const double2* __restrict__ psi, const double2* __restrict__ hpsi, int64_t n,
                              double* __restrict__ sums) {
    __shared__ double s_warp[32];
    double num = 0.0, norm = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double2 p = psi[i], h = hpsi[i];
        num += p.x * h.x + p.y * h.y;
        norm += p.x * p.x + p.y * p.y;
    }
    num = block_sum(num, s_warp);
    norm = block_sum(norm, s_warp);
    if (threadIdx.x == 0) {
        sums[0] = num / norm;
        sums[1] = norm;
    }
}

// partials[b] = sum over the rows of block b of |h_j|^2 / norm / (E0 - Re d_j)
__global__ void pt2_terms_kernel(const double2* __restrict__ hpsi, const double2* __restrict__ diag, int64_t m,
                                 const double* __restrict__ sums, double* __restrict__ partials) {
    __shared__ double s_warp[32];
    const double e0 = sums[0], norm = sums[1];
    double acc = 0.0;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const double2 h = hpsi[j];
        acc += (h.x * h.x + h.y * h.y) / norm / (e0 - diag[j].x);
    }
    acc = block_sum(acc, s_warp);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

__global__ void pt2_sum_kernel(const double* __restrict__ partials, int nb, double* __restrict__ sums) {
    __shared__ double s_warp[32];
    double acc = 0.0;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) acc += partials[k];
    acc = block_sum(acc, s_warp);
    if (threadIdx.x == 0) sums[2] = acc;
}

struct Pt2Layout {
    uint8_t* rows;  // configs (n rows), then the selected rows (at most k)
    double2* hpsi;  // H psi on the same rows
    double2* diag;  // the selected rows' diagonal terms
    double* sums;
    double* partials;
};

Pt2Layout take_pt2(Arena& ws, int64_t n, int64_t k, int nq) {
    Pt2Layout L;
    const uint64_t kk = (uint64_t)(k > 0 ? k : 1);
    L.rows = ws.take<uint8_t>((uint64_t)(n + kk) * (uint64_t)nq);
    L.hpsi = ws.take<double2>((uint64_t)n + kk);
    L.diag = ws.take<double2>(kk);
    L.sums = ws.take<double>(4);
    L.partials = ws.take<double>(kPt2Blocks);
    return L;
}

}  // namespace
}  // namespace qmbx

extern "C" int qmbx_pt2_workspace(const void* table_host, int64_t n, int64_t count_selected, uint64_t* bytes) {
    clear_error();
    const qmbx_table_header* h = header_of(table_host);
    if (h == nullptr || h->magic != QMBX_MAGIC) return fail(QMBX_ERR_ARGUMENT, "not a compiled qmbx table");
    if (bytes == nullptr) return fail(QMBX_ERR_ARGUMENT, "bytes must not be NULL");
    Arena fixed(nullptr, 0);
    take_pt2(fixed, n, count_selected, h->n_qubytes);
    uint64_t find = 0, apply = 0;
    int st = qmbx_find_relative_workspace(table_host, n, count_selected, n, &find);
    if (st != QMBX_OK) return st;
    if ((st = qmbx_apply_within_workspace(table_host, n, n + count_selected, &apply)) != QMBX_OK) return st;
    *bytes = fixed.used + (find > apply ? find : apply);
    return QMBX_OK;
}

extern "C" int qmbx_pt2(const void* table_host, const void* table_dev, const uint8_t* configs, const double* psi,
                        int64_t n, int64_t count_selected, double* energies, int64_t* n_other, void* workspace,
                        uint64_t workspace_bytes, uint64_t* workspace_needed, qmbx_stream_t stream) {
    clear_error();
    int st = check_table(table_host, table_dev);
    if (st != QMBX_OK) return st;
    if (energies == nullptr || n_other == nullptr) return fail(QMBX_ERR_ARGUMENT, "energies and n_other must not be NULL");
    if (n <= 0 || n >= (int64_t(1) << 31)) return fail(QMBX_ERR_ARGUMENT, "row count out of range");
    if (configs == nullptr || psi == nullptr) return fail(QMBX_ERR_ARGUMENT, "input pointers must not be NULL");
    if (count_selected <= 0 || count_selected >= (int64_t(1) << 31)) {
        return fail(QMBX_ERR_ARGUMENT, "count_selected must be positive and below 2^31");
    }
    if ((st = check_ws(workspace)) != QMBX_OK) return st;
    const qmbx_table_header* h = header_of(table_host);
    Arena fixed(workspace, workspace == nullptr ? 0 : workspace_bytes);
    Pt2Layout L = take_pt2(fixed, n, count_selected, h->n_qubytes);
    if (workspace == nullptr || !fixed.fits()) {
        uint64_t want = 0;
        qmbx_pt2_workspace(table_host, n, count_selected, &want);
        if (workspace_needed) *workspace_needed = want;
        return fail(QMBX_ERR_WORKSPACE, "pt2 needs at least %llu bytes of workspace", (unsigned long long)want);
    }
    void* scratch = static_cast<char*>(workspace) + fixed.used;
    const uint64_t scratch_bytes = workspace_bytes - fixed.used;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    *n_other = 0;
    const int nq = h->n_qubytes;
    // the configs first, the selected rows after them
    QMBX_CUDA_TRY(cudaMemcpyAsync(L.rows, configs, (size_t)n * nq, cudaMemcpyDeviceToDevice, s));
    FindArgs a{table_host, table_dev, configs, psi, n, count_selected, configs, n, L.rows + (size_t)n * nq, n_other};
    uint64_t find_needed = 0;
    switch (h->n_words) {
        case 1: st = find_impl<1>(a, scratch, scratch_bytes, &find_needed, s); break;
        case 2: st = find_impl<2>(a, scratch, scratch_bytes, &find_needed, s); break;
        case 3: st = find_impl<3>(a, scratch, scratch_bytes, &find_needed, s); break;
        case 4: st = find_impl<4>(a, scratch, scratch_bytes, &find_needed, s); break;
        default: return fail(QMBX_ERR_ARGUMENT, "unsupported word count");
    }
    if (st == QMBX_ERR_WORKSPACE && workspace_needed) *workspace_needed = fixed.used + find_needed;
    if (st != QMBX_OK) return st;
    const int64_t m = *n_other;
    // H psi onto the configs (for E0) and the selected rows at once
    if ((st = qmbx_apply_within(table_host, table_dev, configs, psi, n, L.rows, n + m, 0,
                                reinterpret_cast<double*>(L.hpsi), scratch, scratch_bytes, stream)) != QMBX_OK) {
        if (st == QMBX_ERR_WORKSPACE && workspace_needed) {
            uint64_t apply = 0;
            qmbx_apply_within_workspace(table_host, n, n + m, &apply);
            *workspace_needed = fixed.used + apply;
        }
        return st;
    }
    QMBX_KERNEL(kGroupSelect, s, pt2_e0_kernel<<<1, 1024, 0, s>>>(reinterpret_cast<const double2*>(psi), L.hpsi, n, L.sums));
    QMBX_LAUNCH_CHECK("pt2_e0_kernel");
    if (m > 0) {
        // the selected rows' diagonal terms
        if ((st = qmbx_diagonal_term(table_host, table_dev, L.rows + (size_t)n * nq, m, reinterpret_cast<double*>(L.diag),
                                     stream)) != QMBX_OK) {
            return st;
        }
        const unsigned nb = grid_for(m, 256) < (unsigned)kPt2Blocks ? grid_for(m, 256) : (unsigned)kPt2Blocks;
        QMBX_KERNEL(kGroupSelect, s, pt2_terms_kernel<<<nb, 256, 0, s>>>(L.hpsi + n, L.diag, m, L.sums, L.partials));
        QMBX_KERNEL(kGroupSelect, s, pt2_sum_kernel<<<1, 1024, 0, s>>>(L.partials, (int)nb, L.sums));
        QMBX_LAUNCH_CHECK("pt2 sums");
    } else {
        QMBX_CUDA_TRY(cudaMemsetAsync(L.sums + 2, 0, sizeof(double), s));
    }
    double out[3] = {0.0, 0.0, 0.0};
    QMBX_CUDA_TRY(cudaMemcpyAsync(out, L.sums, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
    QMBX_CUDA_TRY(cudaStreamSynchronize(s));
    energies[0] = out[0];
    energies[1] = out[2];
    return QMBX_OK;
}
