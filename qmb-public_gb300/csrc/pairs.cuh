// The pair scan: which rows of two row sets a number-conserving operator
// connects, found by comparing the rows themselves instead of walking the
// terms of every row.
//
// A term moves at most two particles, so rows a and b with equally many
// particles are connected only if at most two of a's occupied positions are
// empty in b.  The kernel counts those positions for 32 rows b at a time: the
// b side is stored as bit planes (one 32-bit word per position holds that
// position of 32 rows), and a row a adds up the complements of the planes of
// its occupied positions in a carry-save counter, 7 three-input logic
// instructions per four positions and word (the counter of Harley and Seal;
// Warren, "Hacker's Delight", section 5-1).  The few pairs that stay are
// looked up in the table's transition index (format.h), which names exactly
// the terms between the two rows.
//
// The pairs that stay go to a list in the workspace, and a second kernel looks
// them up with a thread each: the lookups' chains of dependent L2 reads then
// run at full occupancy and in balance however unevenly the rows connect,
// where lookups inside the scan held up the other warps at its barriers.
//
// Against the term walks: a walk tests every reachable term of a row and
// looks up every image, mostly in vain (65,536 random rows of 14 particles on
// 52 sites under 669,579 terms: 1.8e9 lookups for 270 hits).  The scan's cost
// does not depend on the number of terms.  On GB300, kernel times:
//   those 65,536 rows with themselves     13.2 ms walked, 0.20 ms scanned
//   20,000 x 200,000 rows of 10 on 28     0.80 ms walked, 0.31 + 0.10 ms (2.8M pairs looked up)
//   16,384 clustered rows (8.7M hits)     6.4 ms walked, 0.11 + 0.17 ms (matrix count)
// No one unit of the scan is full: the first shape keeps the ALU pipe at 62 %
// (64 lanes a clock and SM for the three-input logic, 1.75 of them per position
// and word) and L1 with shared memory at 77 %, the second 59 % and 67 %, with
// 36 % of the warps resident; DRAM and L2 are near idle.  Counting the head
// that sorted neighbours share once per run of rows gained 1 % and is not done.
// The lookups are bound by the latency of their L2 reads.
#pragma once

#include "device.cuh"

namespace qmbx {

// Words of 32 rows each lane owns: a tile of planes covers 1024 V rows.  The
// lanes read four words with one 16-byte load; three and four key words take
// half, which keeps the planes of 256 positions within shared memory.
template <int W>
__host__ __device__ constexpr int pair_words() {
    return W <= 2 ? 4 : 2;
}
template <int W>
__host__ __device__ constexpr int pair_tile() {
    return 1024 * pair_words<W>();
}
// Consecutive rows of the list side a warp stages at a time.
constexpr int kPairRun = 8;

// A row set prepared for the scan: its distinct rows ordered by particle
// number, so that a tile holds rows of one number (two at a boundary) and
// rows of another number skip it.
struct PairSet {
    uint64_t* keys;    // n x W, scan order
    int32_t* row;      // first row of every scan position
    uint32_t* planes;  // [tiles][sites][32 V]: word w of site s holds rows 32 w .. 32 w + 31 of the tile
    uint16_t* list;    // [n, a whole number of runs][sites]: occupied sites x 32 (plane offsets in units of V words),
                       // most significant position first; an odd list ends with `sites` x 32, a plane of ones
    int* hist;         // rows per particle number, then the places taken so far (2 x (64 W + 1))
    const int* count;  // distinct rows (device)
    int64_t n;         // rows of the set
};

struct PairWork {
    PairSet i, j;          // j == i for the same rows on both sides
    // work items handed out, close pairs found, choose_pairs' sums; then both sets' hist, all cleared at once
    unsigned long long* next;
    uint64_t clear_bytes;
    uint2* pairs;          // pairs that stay: scan positions of the list side and the plane side
    unsigned int cap;      // places in `pairs`; pairs past them are looked up by the scan itself,
    void* overflow;        // with a PairQueue per warp of the grid
    int* gate;             // rows for the scan's diagonal pass, rows for the walk: one of them is 0
    bool same;
};

// Blocks of the scan at most.  Three are resident on each of 152 SMs (80 registers a thread; two at 256 positions); the
// rest start behind them and mostly find every work item handed out.
constexpr int kPairBlocks = 608;
constexpr int kPairCounters = 6;
// Words of 64 bits for a set's hist (a count for each of 0 .. 64 W particles, twice, as ints).
template <int W>
constexpr int pair_hist() {
    return 64 * W + 1;
}

template <int W>
PairSet take_pair_set(Arena& ws, int64_t n, int sites, int* hist);

// Hits waiting to be applied: one a lane, or four where they are recorded,
// since every drain's atomic meets the same counter (3.6M recorded FP32 hits:
// lookups 151 us with one, 128 us with four; unrecorded FP64 99 and 107 us).
// Fewer than a drain wait while a lookup adds one a lane.
constexpr int kPairDrain = 128;
struct PairQueue {
    int4 hits[kPairDrain + 32];  // (slot | parity << 31, from row, to row, 0)
};

template <int W>
PairWork take_pair_work(Arena& ws, int64_t n_i, int64_t n_j, bool same, int sites) {
    PairWork p{};
    p.same = same;
    p.clear_bytes = (kPairCounters + 2 * pair_hist<W>()) * sizeof(unsigned long long);
    p.next = ws.take<unsigned long long>(kPairCounters + 2 * pair_hist<W>());
    int* hist = p.next != nullptr ? reinterpret_cast<int*>(p.next + kPairCounters) : nullptr;
    p.i = take_pair_set<W>(ws, n_i, sites, hist);
    p.j = same ? p.i : take_pair_set<W>(ws, n_j, sites, hist != nullptr ? hist + 2 * pair_hist<W>() : nullptr);
    // Room for a few dozen pairs a row (20,000 x 200,000 rows of 10 among 28 list 2.8M pairs).  A pair past it costs
    // up to half again as much where most pairs connect (140 against 100 ps), more where few do.
    const double rows_i = (double)(n_i > 0 ? n_i : 1), rows_j = (double)(n_j > 0 ? n_j : 1);
    const double all = same ? 0.5 * rows_i * (rows_i - 1.0) + 1.0 : rows_i * rows_j;
    const double room = (double)(1 << 22) + 32.0 * ((double)n_i + (double)n_j);
    p.cap = (unsigned int)(all < room ? all : room < 4e9 ? room : 4e9);
    p.pairs = ws.take<uint2>(p.cap);
    // a list with a place for every pair does not run over
    p.overflow = (double)p.cap < all ? ws.take<PairQueue>((uint64_t)kPairBlocks * kWarpsPerBlock) : nullptr;
    p.gate = ws.take<int>(2);
    return p;
}

// Order the distinct rows of `rows`; form their planes, their position lists, or both (nothing when *gate is 0).
template <int W>
int build_pair_set(const HashRows& rows, int sites, bool planes, bool lists, const int* gate, PairSet& out, cudaStream_t s);

// The planes are made of the larger side, whose tiles they fill better.
inline bool pairs_swapped(const PairWork& p) { return !p.same && p.i.n > p.j.n; }

// p.gate for the rows at hand, and cleared counters: the scan, or else the walk (`walked`: its row set; `terms`:
// its part).  On the host only numbers of rows and terms are known; what the scan costs also depends on how many
// pairs are close, and the walk on how many terms a row reaches, so a sample of both is taken on the device.
// Costs, fitted to whole FP64 calls (times in ps, summed over the GPU): a pair of rows 0.0075 a particle; a close
// pair 80 within one set (100 for its two lookups and hits, less 20 for the two hits a walk would find), 40 between
// two; a reached term 5 in the walk; against the grouped walk 35 us for the scan's two kernels, whose blocks are few
// and uneven on small sets (clustered sets of that size are no better in the pivot-major walk).  (scan and walk, us)
//   every determinant of 3 + 3 in 14 orbitals, 132,496 rows    11,934   4,093 (all of a row's 1,485 neighbours present)
//   a random third of them, 40,000 rows                          1,184   1,016
//   200,000 of the 4.0M of 5 + 5                                 2,783   7,914
//   16,384 and 262,144 clustered rows of 7 + 7 in 26      515, 13,740   4,610, 70,543
//   8,281 rows, all of 2 + 2 in 14                                  518     219
template <int W>
int choose_pairs(const PairWork& p, const HashRows& rows_i, const HashRows& rows_j, const HashRows& walked,
                 const PartView& terms, cudaStream_t s);

// Prepare both sides.
template <int W>
int build_pairs(const HashRows& rows_i, const HashRows& rows_j, int sites, PairWork& p, cudaStream_t s) {
    const bool swap = pairs_swapped(p);
    int st = build_pair_set<W>(rows_i, sites, p.same || swap, p.same || !swap, p.gate, p.i, s);
    if (st != QMBX_OK) return st;
    if (p.same) {
        p.j = p.i;
        return QMBX_OK;
    }
    return build_pair_set<W>(rows_j, sites, !swap, swap, p.gate, p.j, s);
}

// Whether the table can be scanned, whether a call on n_i x n_j rows has
// scratch for it, and whether it may be (pairs.cu).
bool pairs_possible(const qmbx_table_header* h);
bool pairs_scratch(const qmbx_table_header* h, int64_t n_i, int64_t n_j);
bool pairs_wanted(const qmbx_table_header* h, int64_t n_i, int64_t n_j);
bool pairs_forced();  // QMBX_WALK names the scan

// Rows of the list side per work item, for about 16 items per SM.
int pair_chunk(int64_t n_list, int64_t n_planes, int tile);

struct ClassView {
    const uint4* buckets;
    const int2* list;
    uint32_t mask;
    int shift;
};

inline ClassView class_view(const void* table_host, const void* table_dev) {
    const qmbx_table_header* h = header_of(table_host);
    const char* base = static_cast<const char*>(table_dev);
    ClassView c;
    c.buckets = reinterpret_cast<const uint4*>(base + h->off_class);
    c.list = reinterpret_cast<const int2*>(base + h->off_class_list);
    c.mask = (uint32_t)(h->n_class_buckets - 1);
    c.shift = 32;
    for (int64_t b = h->n_class_buckets; b > 1; b >>= 1) --c.shift;
    return c;
}

constexpr uint32_t kNoClass = 0xffffffffu;

__device__ __forceinline__ uint32_t class_find(const ClassView& c, uint32_t key) {
    uint32_t b = qmbx_class_bucket(key, c.shift);
    for (uint32_t probe = 0; probe <= c.mask; ++probe) {
        const uint4 e = __ldg(c.buckets + b);
        if (e.x == key) return e.y;
        if (e.z == key) return e.w;
        if (e.x == 0u || e.z == 0u) return kNoClass;
        b = (b + 1) & c.mask;
    }
    return kNoClass;
}

// Transition keys from a to b and back; false when no term can connect them
// (more than two positions differ on a side, or not equally many).
template <int W>
__device__ __forceinline__ bool transition(const Key<W>& a, const Key<W>& b, uint32_t& there, uint32_t& back) {
    int gone = 0, come = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) {
        gone += __popcll(a.w[q] & ~b.w[q]);
        come += __popcll(b.w[q] & ~a.w[q]);
    }
    if (gone != come || gone < 1 || gone > 2) return false;
    uint32_t lo[2] = {0, 0}, hi[2] = {0, 0};  // lowest and highest position that a alone, b alone holds
#pragma unroll
    for (int q = W - 1; q >= 0; --q) {
        const uint64_t m0 = a.w[q] & ~b.w[q], m1 = b.w[q] & ~a.w[q];
        if (m0) lo[0] = 64 * q + (__ffsll((long long)m0) - 1);
        if (m1) lo[1] = 64 * q + (__ffsll((long long)m1) - 1);
    }
#pragma unroll
    for (int q = 0; q < W; ++q) {
        const uint64_t m0 = a.w[q] & ~b.w[q], m1 = b.w[q] & ~a.w[q];
        if (m0) hi[0] = 64 * q + 63 - __clzll((long long)m0);
        if (m1) hi[1] = 64 * q + 63 - __clzll((long long)m1);
    }
    const uint32_t from = lo[0] | hi[0] << 8, to = lo[1] | hi[1] << 8;
    there = from | to << 16;
    back = to | from << 16;
    return true;
}

template <int W, class H>
struct PairContext {
    H h;
    ClassView cls;
    PartView fwd;
    const uint64_t *a_keys, *b_keys;  // list side, plane side
    const int32_t *a_row, *b_row;
    int same, swap;  // swap: the list side holds the rows the terms lead to
};

template <int W, class H>
struct PairWorker {
    const PairContext<W, H>& x;
    PairQueue& q;
    int hcount;
    int lane;

    __device__ __forceinline__ void drain(int n) {
        x.h.record(q.hits, n, lane);
        for (int k = lane; k < n; k += 32) x.h.apply(q.hits[k]);
        __syncwarp();
        if (lane < hcount - n) q.hits[lane] = q.hits[n + lane];  // fewer than 32
        __syncwarp();
        hcount -= n;
    }
    __device__ __forceinline__ void push(bool hit, int4 v) {
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m == 0) return;
        if (hit) q.hits[hcount + __popc(m & ((1u << lane) - 1u))] = v;
        hcount += __popc(m);
        __syncwarp();
        const int full = x.h.recording() ? kPairDrain : 32;
        if (hcount >= full) drain(full);
    }
    __device__ __forceinline__ uint32_t parity_of(const Key<W>& c, int64_t slot) const {
        int par = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) par += __popcll(c.w[w] & __ldg(x.fwd.apply + (int64_t)w * x.fwd.stride + slot).y);
        return (uint32_t)(par & 1) << 31;
    }
    // the terms of the transition v from row `from` (key c) to row `to`, one transition a lane
    __device__ __forceinline__ void connect(uint32_t v, const Key<W>& c, int from, int to) {
        const bool only = v != kNoClass && !(v >> 31), several = v != kNoClass && (v >> 31);
        // the parity of the only term, or of the run's first
        uint32_t slot = v;
        if (several) slot = (uint32_t)__ldg(x.cls.list + (v & 0x7fffffffu)).x & 0x7fffffffu;
        const uint32_t par = only || several ? parity_of(c, slot) : 0u;
        push(only, make_int4((int)(v | par), from, to, 0));
        // transitions of several terms: the lanes over the terms
        unsigned lists = __ballot_sync(0xffffffffu, several);
        while (lists) {
            const int src = __ffs(lists) - 1;
            lists &= lists - 1;
            int at = (int)(__shfl_sync(0xffffffffu, v, src) & 0x7fffffffu);
            const int f = __shfl_sync(0xffffffffu, from, src), t = __shfl_sync(0xffffffffu, to, src);
            const uint32_t p = __shfl_sync(0xffffffffu, par, src);
            Key<W> k;
#pragma unroll
            for (int w = 0; w < W; ++w) k.w[w] = __shfl_sync(0xffffffffu, c.w[w], src);
            for (;; at += 32) {
                const int2 e = __ldg(x.cls.list + at + lane);
                const unsigned end = __ballot_sync(0xffffffffu, e.x < 0);
                const uint32_t s = (uint32_t)e.x & 0x7fffffffu;
                bool on = end == 0 || lane < __ffs(end);
                uint32_t sign = p;
                if (on && e.y >= 0) on = has_position<W>(k, e.y);
                if (on && e.y == -2) {
                    TermRec<W> rec;
                    load_test<W>(rec, x.fwd, s);
                    on = rec.applies(k);
                    if (on) sign = parity_of(k, s);
                }
                push(on, make_int4((int)(s | sign), f, t, 0));
                if (end) break;
            }
        }
    }
};

// Look up pairs, one a lane (live lanes): the terms from the rows of
// configs_i to those of configs_j, or both ways within one set.
template <int W, class H>
__device__ __forceinline__ void pair_lookup(PairWorker<W, H>& work, bool live, uint32_t pa, uint32_t pb) {
    const PairContext<W, H>& x = work.x;
    bool ok = false;
    Key<W> ka{}, kb{};
    uint32_t there = 0, back = 0;
    int ra = 0, rb = 0;
    if (live) {
        ka = load_key<W>(x.a_keys, pa);
        kb = load_key<W>(x.b_keys, pb);
        ra = __ldg(x.a_row + pa);
        rb = __ldg(x.b_row + pb);
        ok = transition<W>(ka, kb, there, back);
    }
    // swap: the terms lead from b to a; same rows: both ways
#pragma unroll 1
    for (int way = 0; way < (x.same ? 2 : 1); ++way) {
        const bool rev = x.swap || way == 1;
        Key<W> c;
#pragma unroll
        for (int w = 0; w < W; ++w) c.w[w] = rev ? kb.w[w] : ka.w[w];
        work.connect(ok ? class_find(x.cls, rev ? back : there) : kNoClass, c, rev ? rb : ra, rev ? ra : rb);
    }
}

// The list of pairs is full: look up a warp's pairs in the scan.
template <int W, class H>
__device__ __noinline__ void pair_overflow(const PairContext<W, H>* x, PairQueue* q, bool live, uint32_t pa, uint32_t pb) {
    PairWorker<W, H> work{*x, *q, 0, (int)(threadIdx.x & 31)};
    pair_lookup<W, H>(work, live, pa, pb);
    work.drain(work.hcount);
}

template <int W, class H>
__global__ void __launch_bounds__(kThreads) pair_lookup_kernel(const __grid_constant__ PairContext<W, H> context,
                                                               const uint2* __restrict__ pairs,
                                                               const unsigned long long* __restrict__ listed,
                                                               unsigned int cap) {
    __shared__ PairQueue s_queue[kWarpsPerBlock];
    const unsigned int n = *listed < cap ? (unsigned int)*listed : cap;
    const int lane = threadIdx.x & 31;
    PairWorker<W, H> work{context, s_queue[threadIdx.x >> 5], 0, lane};
    const uint64_t step = (uint64_t)gridDim.x * kThreads;
    for (uint64_t base = (uint64_t)blockIdx.x * kThreads + (threadIdx.x & ~31u); base < n; base += step) {
        const bool live = base + lane < n;
        const uint2 p = live ? __ldg(pairs + base + lane) : make_uint2(0, 0);
        pair_lookup<W, H>(work, live, p.x, p.y);
    }
    work.drain(work.hcount);
}

// What a warp of the scan has found and not yet listed: a lane's words of a
// row's pairs that stay, and single pairs waiting for all lanes to have one.
// Up to 31 of either wait while 32 more are added.
template <int W>
struct PairFound {
    static constexpr int kTileBits = pair_words<W>() == 4 ? 12 : 11;
    alignas(16) uint32_t near[64][pair_words<W>()];
    uint32_t tag[64];    // list row (from the item's first) << 5 | lane
    uint32_t pairs[64];  // list row << kTileBits | plane row of the tile
};

// Where found pairs go.
template <int W, class H>
struct PairOut {
    const PairContext<W, H>* context;
    uint2* pairs;
    unsigned long long* listed;  // counts on past the list's end; two sets can hold more than 2^32 close pairs
    unsigned int cap;
    PairQueue* overflow;
};

// Append the newest n (<= 32) waiting pairs of f to the list.
template <int W, class H>
__device__ __forceinline__ void pair_list(const PairOut<W, H>& out, const PairFound<W>& f, int64_t a0, int64_t b0,
                                          int waiting, int n, int lane) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(out.listed, (unsigned long long)n);
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t e = f.pairs[lane < n ? waiting - n + lane : 0];
    const uint32_t pa = (uint32_t)a0 + (e >> PairFound<W>::kTileBits);
    const uint32_t pb = (uint32_t)b0 + (e & ((1u << PairFound<W>::kTileBits) - 1u));
    const bool late = lane < n && base + lane >= out.cap;
    if (lane < n && !late) out.pairs[base + lane] = make_uint2(pa, pb);
    if (__any_sync(0xffffffffu, late)) {
        pair_overflow<W, H>(out.context, out.overflow + blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5), late, pa, pb);
    }
    __syncwarp();
}

// Split the newest n (<= 32) of `rows` waiting entries into single pairs and
// list those that fill a warp, at the end all of them.  Returns the pairs
// that wait.  Not inlined: the counting loop keeps its registers.
template <int W, class H>
__device__ __noinline__ int pair_split(const PairOut<W, H>& out, PairFound<W>& f, int64_t a0, int64_t b0, int rows, int n,
                                       int waiting, bool end) {
    constexpr int V = pair_words<W>();
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t near[V];
    uint32_t tag = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) near[v] = 0;
    if (lane < n) {
        tag = f.tag[rows - n + lane];
#pragma unroll
        for (int v = 0; v < V; ++v) near[v] = f.near[rows - n + lane][v];
    }
    __syncwarp();
    const uint32_t first = (tag & 31u) * 32 * V;  // the lane's first plane row
    const uint32_t e = (tag >> 5) << PairFound<W>::kTileBits | first;
    // within one set only pairs with the list row first
    const int64_t behind = out.context->same ? a0 + (tag >> 5) - b0 - first : -1;
    for (;;) {
        int bit = -1;
#pragma unroll
        for (int v = V - 1; v >= 0; --v) bit = near[v] != 0u ? 32 * v + __ffs(near[v]) - 1 : bit;
        if (!__any_sync(0xffffffffu, bit >= 0)) break;
#pragma unroll
        for (int v = 0; v < V; ++v) near[v] &= bit >> 5 == v ? near[v] - 1u : 0xffffffffu;
        const bool take = bit >= 0 && bit > behind;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) f.pairs[waiting + __popc(m & lt)] = e + (uint32_t)bit;
        waiting += __popc(m);
        __syncwarp();
        if (waiting >= 32) {
            pair_list<W, H>(out, f, a0, b0, waiting, 32, lane);
            waiting -= 32;
        }
    }
    if (end && waiting > 0) {
        pair_list<W, H>(out, f, a0, b0, waiting, waiting, lane);
        waiting = 0;
    }
    return waiting;
}

template <int V>
struct PlaneWords;
template <>
struct PlaneWords<4> {
    static __device__ __forceinline__ void get(const uint32_t* p, uint32_t (&w)[4]) {
        const uint4 x = *reinterpret_cast<const uint4*>(p);
        w[0] = x.x;
        w[1] = x.y;
        w[2] = x.z;
        w[3] = x.w;
    }
    static __device__ __forceinline__ void put(uint32_t* p, const uint32_t (&w)[4]) {
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};
template <>
struct PlaneWords<2> {
    static __device__ __forceinline__ void get(const uint32_t* p, uint32_t (&w)[2]) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        w[0] = x.x;
        w[1] = x.y;
    }
    static __device__ __forceinline__ void put(uint32_t* p, const uint32_t (&w)[2]) {
        *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    }
};

// One three-input logic instruction; `Table` is the function's value at
// (a, b, c) = (0xf0, 0xcc, 0xaa).
template <int Table>
__device__ __forceinline__ uint32_t logic3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(r) : "r"(a), "r"(b), "r"(c), "n"(Table));
    return r;
}
constexpr int kXor3 = 0x96;         // a ^ b ^ c
constexpr int kMajority = 0xe8;     // at least two of a, b, c
constexpr int kMajorityNot = 0x71;  // at least two of a, ~b, ~c
constexpr int kOrAnd = 0xf8;        // a | (b & c)
constexpr int kNotOrAnd = 0x07;     // ~(a | (b & c))

// How many of a list's positions are empty in each plane row: ones + 2 twos,
// or more.
template <int V>
struct EmptyCount {
    uint32_t ones[V], twos[V], more[V];
    // count a list of `pairs` pairs of positions; more starts as `absent`
    __device__ __forceinline__ void count(const uint32_t* planes, const uint16_t* list, int pairs, int lane,
                                          const uint32_t (&absent)[V]) {
        int k = 0;
        if (pairs & 1) {
            // an odd pair first: nothing is counted yet
            const uint32_t at = *reinterpret_cast<const uint32_t*>(list + 2 * (pairs - 1));
            uint32_t p0[V], p1[V];
            PlaneWords<V>::get(planes + ((at & 0xffffu) + lane) * V, p0);
            PlaneWords<V>::get(planes + ((at >> 16) + lane) * V, p1);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                ones[v] = p0[v] ^ p1[v];
                twos[v] = ~(p0[v] | p1[v]);
                more[v] = absent[v];
            }
        } else if (pairs != 0) {
            uint32_t p0[V], p1[V], p2[V], p3[V];
            four(planes, list, lane, p0, p1, p2, p3);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint32_t c0 = ~(p0[v] | p1[v]);
                const uint32_t s0 = p0[v] ^ p1[v];
                const uint32_t c1 = logic3<kMajorityNot>(s0, p2[v], p3[v]);
                ones[v] = logic3<kXor3>(s0, p2[v], p3[v]);
                more[v] = logic3<kOrAnd>(absent[v], c0, c1);
                twos[v] = c0 ^ c1;
            }
            k = 2;
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                ones[v] = twos[v] = 0u;
                more[v] = absent[v];
            }
        }
#pragma unroll 2
        for (; k + 2 <= pairs; k += 2) {
            uint32_t p0[V], p1[V], p2[V], p3[V];
            four(planes, list + 2 * k, lane, p0, p1, p2, p3);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint32_t c0 = logic3<kMajorityNot>(ones[v], p0[v], p1[v]);
                const uint32_t s0 = logic3<kXor3>(ones[v], p0[v], p1[v]);
                const uint32_t c1 = logic3<kMajorityNot>(s0, p2[v], p3[v]);
                ones[v] = logic3<kXor3>(s0, p2[v], p3[v]);
                more[v] |= logic3<kMajority>(twos[v], c0, c1);
                twos[v] = logic3<kXor3>(twos[v], c0, c1);
            }
        }
    }
    static __device__ __forceinline__ void four(const uint32_t* planes, const uint16_t* list, int lane, uint32_t (&p0)[V],
                                                uint32_t (&p1)[V], uint32_t (&p2)[V], uint32_t (&p3)[V]) {
        const uint2 at = *reinterpret_cast<const uint2*>(list);
        PlaneWords<V>::get(planes + ((at.x & 0xffffu) + lane) * V, p0);
        PlaneWords<V>::get(planes + ((at.x >> 16) + lane) * V, p1);
        PlaneWords<V>::get(planes + ((at.y & 0xffffu) + lane) * V, p2);
        PlaneWords<V>::get(planes + ((at.y >> 16) + lane) * V, p3);
    }
};

// Shared memory of a block: the planes of a tile (and an all-ones plane for
// odd lists) and the staged position lists.
template <int W>
int pair_shared_bytes(int sites) {
    return (sites + 1) * 32 * pair_words<W>() * 4 + kWarpsPerBlock * kPairRun * sites * 2;
}

template <int W, class H>
__global__ void __launch_bounds__(kThreads, 3)
    pair_scan_kernel(const __grid_constant__ PairContext<W, H> context, const uint32_t* __restrict__ planes,
                     const uint16_t* __restrict__ lists, const int* __restrict__ a_count,
                     const int* __restrict__ b_count, int sites, int chunk,
                     unsigned long long* __restrict__ next, uint2* __restrict__ pairs, unsigned int cap, PairQueue* overflow,
                     const int* __restrict__ gate) {
    constexpr int V = pair_words<W>();
    constexpr int kWords = 32 * V;
    constexpr int kTile = pair_tile<W>();
    extern __shared__ uint4 pair_sm[];
    uint32_t* s_planes = reinterpret_cast<uint32_t*>(pair_sm);
    __shared__ PairFound<W> s_found[kWarpsPerBlock];
    __shared__ unsigned long long s_item;
    if (gate != nullptr && *gate == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    uint16_t* s_list = reinterpret_cast<uint16_t*>(s_planes + (sites + 1) * kWords) + warp * kPairRun * sites;
    const uint64_t* a_keys = context.a_keys;
    const uint64_t* b_keys = context.b_keys;
    const bool same = context.same != 0;
    const int64_t na = *a_count, nb = *b_count;
    const int64_t tiles = (nb + kTile - 1) / kTile, chunks = (na + chunk - 1) / chunk;
    const PairOut<W, H> out{&context, pairs, next + 1, cap, overflow};
    PairFound<W>& found = s_found[warp];
    int rows = 0, single = 0;  // entries and pairs waiting in `found`
    for (;;) {
        __syncthreads();  // the last item's planes and number have been read
        if (threadIdx.x == 0) s_item = atomicAdd(next, 1ull);
        __syncthreads();
        const int64_t item = (int64_t)s_item;
        if (item >= tiles * chunks) break;
        const int64_t tile = item / chunks;
        const int64_t first = (item - tile * chunks) * chunk;
        int64_t last = first + chunk < na ? first + chunk : na;
        const int64_t b0 = tile * kTile;
        const int64_t b1 = b0 + kTile < nb ? b0 + kTile : nb;
        if (same && last > b1) last = b1;  // only pairs with the list row first
        if (first >= last) continue;
        int lowest = 0, highest = 0;       // particle numbers of the tile
        {
            const Key<W> k0 = load_key<W>(b_keys, b0), k1 = load_key<W>(b_keys, b1 - 1);
#pragma unroll
            for (int q = 0; q < W; ++q) {
                lowest += __popcll(k0.w[q]);
                highest += __popcll(k1.w[q]);
            }
        }
        const uint4* src = reinterpret_cast<const uint4*>(planes + tile * (int64_t)sites * kWords);
        for (int k = threadIdx.x; k < sites * kWords / 4; k += kThreads) reinterpret_cast<uint4*>(s_planes)[k] = __ldg(src + k);
        for (int k = threadIdx.x; k < kWords; k += kThreads) s_planes[sites * kWords + k] = 0xffffffffu;
        uint32_t absent[V];  // rows past the last one never match
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int rows = (int)(b1 - b0) - 32 * (lane * V + v);
            absent[v] = rows >= 32 ? 0u : rows <= 0 ? 0xffffffffu : 0xffffffffu << rows;
        }
        __syncthreads();  // planes stored
        for (int64_t run = first + warp * kPairRun; run < last; run += kWarpsPerBlock * kPairRun) {
            // stage the run's lists
            for (int k = lane; k < kPairRun * sites / 8; k += 32) {
                reinterpret_cast<uint4*>(s_list)[k] = __ldg(reinterpret_cast<const uint4*>(lists + run * sites) + k);
            }
            int number = 0;
            if (lane < kPairRun && run + lane < last) {
                const Key<W> k = load_key<W>(a_keys, run + lane);
#pragma unroll
                for (int q = 0; q < W; ++q) number += __popcll(k.w[q]);
            }
            const bool valid = lane < kPairRun && run + lane < last && number >= lowest && number <= highest;
            const int twos = (number + 1) / 2;
            unsigned todo = __ballot_sync(0xffffffffu, valid);
            __syncwarp();
#pragma unroll 1
            for (; todo != 0; todo &= todo - 1) {
                const int r = __ffs(todo) - 1;
                EmptyCount<V> c;
                c.count(s_planes, s_list + r * sites, __shfl_sync(0xffffffffu, twos, r), lane, absent);
                uint32_t near[V], any = 0;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    near[v] = logic3<kNotOrAnd>(c.more[v], c.ones[v], c.twos[v]);  // at most two
                    any |= near[v];
                }
                const unsigned m = __ballot_sync(0xffffffffu, any != 0u);
                if (m == 0) continue;
                if (any != 0u) {
                    const int at = rows + __popc(m & lt);
                    PlaneWords<V>::put(found.near[at], near);
                    found.tag[at] = (uint32_t)(run - first + r) << 5 | (uint32_t)lane;
                }
                rows += __popc(m);
                __syncwarp();
                if (rows >= 32) {
                    single = pair_split<W, H>(out, found, first, b0, rows, 32, single, false);
                    rows -= 32;
                }
            }
            __syncwarp();  // the run's lists have been read
        }
        if (rows > 0 || single > 0) {
            pair_split<W, H>(out, found, first, b0, rows, rows, single, true);
            rows = single = 0;
        }
    }
}

// Scan every pair of rows of i and j: hits of terms that lead from a row of i
// to a row of j.  The counters are cleared (choose_pairs).
template <int W, class H>
int launch_pair_scan(const H& h, const PairWork& p, const void* table_host, const void* table_dev, const int* gate,
                     cudaStream_t s, int group) {
    const int sites = header_of(table_host)->n_sites;
    const bool swap = pairs_swapped(p);
    const PairSet& a = swap ? p.j : p.i;
    const PairSet& b = swap ? p.i : p.j;
    const int shared = pair_shared_bytes<W>(sites);
    // Beside the static queues the planes of more than about 40 positions pass the default limit.  The limit is the
    // kernel's, not the call's: every call sets what the longest rows of W words need, so that no thread lowers it
    // between another's setting and launch.
    QMBX_CUDA_TRY(cudaFuncSetAttribute(pair_scan_kernel<W, H>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       pair_shared_bytes<W>(64 * W)));
    const PairContext<W, H> context{h, class_view(table_host, table_dev), part_view(table_host, table_dev, QMBX_PART_FWD),
                                    a.keys, b.keys, a.row, b.row, p.same ? 1 : 0, swap ? 1 : 0};
    const int grid = pivot_grid() < kPairBlocks ? pivot_grid() : kPairBlocks;
    QMBX_KERNEL(group, s, pair_scan_kernel<W, H><<<grid, kThreads, shared, s>>>(
        context, b.planes, a.list, a.count, b.count, sites, pair_chunk(a.n, b.n, pair_tile<W>()), p.next, p.pairs, p.cap,
        static_cast<PairQueue*>(p.overflow), gate));
    QMBX_KERNEL(kGroupOther, s, pair_lookup_kernel<W, H><<<2 * pivot_grid(), kThreads, 0, s>>>(context, p.pairs, p.next + 1, p.cap));
    QMBX_LAUNCH_CHECK("pair scan");
    return QMBX_OK;
}

}  // namespace qmbx
