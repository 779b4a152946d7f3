// sgd_small.cu - the deterministic layout of small graphs (n_vertices x dim
// within kSmallLayoutFloats): optimize_layout_training
// (rust_umap/src/lib.rs:5137-5321) with the same result on every run.
//
// The edges are coloured greedily in graph order so that no two edges of a
// colour share a vertex.  An epoch updates the due edges as if the colours
// ran one after another (Gauss-Seidel by colour); negative samples read the
// positions at the epoch's start.  A due edge therefore depends only on the
// earlier due edges at its own two vertices, and any execution order that
// keeps each vertex's order gives the same positions bit for bit.
//
// Which edges are due, their negative counts and the negatives themselves do
// not depend on the positions, so they are worked out for a block of epochs
// at a time on the whole GPU:
//   due_kernel     one thread per edge replays its schedule and writes its
//                  negative count (or kNotDue) for every epoch of the block;
//   order_kernel   one CTA per epoch walks the colours once, gives every due
//                  edge its rank among its head's and its tail's due edges and
//                  the earliest time it could start, and writes one 48-byte
//                  event per due edge, sorted by that time, in batches of up
//                  to 32 that could start together (0.24 ms a block of epochs
//                  at 1,000 rows, 0.6 at 4,200);
//   layout_kernel  one CTA holds the embedding in shared memory and runs the
//                  batches of the block's epochs.  A warp takes a batch, waits
//                  until each event's two vertices have reached its ranks,
//                  updates, and advances their counts (the tail's right after
//                  the attractive step, the head's after its last negative).
// What bounds it is the serial chain of the busiest vertex: about 390 cycles
// for an attractive step and 270 for a negative (logarithm 64, exponential,
// division 40 and a dozen dependent operations), behind about 200 cycles from
// one warp's store to the next one's start.  At 1,000 x 32 rows of noise (22,500
// edges, 6,900 due in an epoch; by the rows drawn, a vertex with 37 to 55 due
// edges at its head and as many at its tail) the arithmetic of that chain is 41
// to 61 us an epoch; layout_kernel takes 119 to 164.  The three kernels
// together, against one CTA with a barrier after every colour that reads its
// schedule and draws its random numbers on the chain: 200 epochs of 1,000 x 32
// (55 due edges) 33.4 and 272 ms, 100 epochs of 4,200 x 96 34.9 and 282, of
// 8,192 x 32 42.9 and 286.
//
// Measured and not kept (1,000 x 32 / 4,200 x 96, against 27 / 40 ms on the same
// rows): the events in colour order, one per lane (53 / 62); each ready lane at
// once instead of the whole batch together (36 / 48); a state machine that runs
// one sample of every lane's event a step (44 / 60: its polls, votes and branches
// cost more than the step); smaller batches (38 / 50 at half the size).
//
// A wait always ends: batches are in an order that respects the dependencies
// and a warp takes its own in that order, so the first batch that is not done
// waits only for batches that are.  It is bounded all the same: a warp stops
// the layout after kSpinLimit polls during which no warp of the CTA has got any
// further (the vertices' counts, and `beat` within a long run of negatives).
// How long a batch may wait has no bound of its own: at a negative rate of
// 8,000,000 one event takes 1.5 s.
#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "sgd_math.cuh"

namespace umapb {
namespace {

constexpr int kMaxDim = 16;
constexpr int kSmallThreads = 512;  // 16 warps: 256 and 768 threads were 10 to 30% slower
constexpr int kWarps = kSmallThreads / 32;
constexpr int kOrderThreads = 1024;
constexpr uint32_t kNotDue = 0xffffffffu;
constexpr int kInlineNeg = 14;      // negatives stored in the event (rate 5 draws 3 to 9)
constexpr int kStartBuckets = 4096;  // distinct start times an epoch is sorted by
constexpr uint32_t kByColor = 0x80000000u;  // flag on n_batches: the events are in colour order
constexpr uint32_t kSpinLimit = 1u << 23;  // polls while no warp updates anything (about 1 s)
constexpr uint32_t kBeatEvery = 4096;      // negatives
constexpr size_t kBlockBytes = static_cast<size_t>(256) << 20;  // work space of one block of epochs
constexpr size_t kBlockStep = static_cast<size_t>(32) << 20;
constexpr int64_t kBlockEpochs = 148;  // one order_kernel CTA per SM

// One due edge of one epoch.
struct alignas(16) Event {
    uint32_t ends;    // head | tail << 16
    uint32_t rank_h;  // due edges before this one at its head and at its tail
    uint32_t rank_t;
    uint32_t n_neg;
    uint32_t edge;    // graph-order id: keys the negative stream
    uint16_t neg[kInlineNeg];
};
static_assert(sizeof(Event) == 48, "three 16-byte loads");

struct SmallArgs {
    float* emb;               // n x dim, global
    int64_t m;
    uint32_t n_vertices;
    int dim;
    // edges in colour order
    const int32_t* order;     // graph-order id
    const int32_t* heads;
    const int32_t* tails;
    const float* eps;
    float* next;
    float* next_neg;
    const int32_t* color_ptr;  // n_colors + 1 offsets
    int n_colors;
    // the block of epochs
    int64_t epoch0;
    int n_block;
    uint32_t* n_neg;          // n_block x m
    uint32_t* start;          // n_block x m: earliest start, ranks at head and tail
    uint32_t* rank_h;
    uint32_t* rank_t;
    Event* events;            // n_block x m
    uint32_t* batches;        // n_block x batch_cap: first event of each batch, then the total
    uint32_t* n_batches;      // n_block; kByColor set where the events are in colour order
    int64_t batch_cap;
    unsigned long long* samples;  // attractive samples over all epochs
    int* err;
    // layout
    int64_t n_epochs;
    float lr, a, b, att_factor, rep_factor, neg_rate_f;
    uint64_t seed;
};

// The edges in colour order with their schedule at epoch 0
// (make_epochs_per_sample, lib.rs:4937-4960).
__global__ void gather_kernel(const int32_t* __restrict__ order, const int32_t* __restrict__ gh,
                              const int32_t* __restrict__ gt, const float* __restrict__ w,
                              float max_w, float n_epochs_f, float neg_rate_f, int64_t m,
                              int32_t* __restrict__ heads, int32_t* __restrict__ tails,
                              float* __restrict__ eps, float* __restrict__ next,
                              float* __restrict__ next_neg) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int32_t e = order[i];
    heads[i] = gh[e];
    tails[i] = gt[e];
    const float v = epochs_per_sample(w[e], max_w, n_epochs_f);
    eps[i] = v;
    next[i] = v;
    next_neg[i] = __fdiv_rn(v, neg_rate_f);
}

__global__ void __launch_bounds__(256) due_kernel(SmallArgs p) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= p.m) return;
    const float eps = p.eps[i];
    float nxt = p.next[i], nn = p.next_neg[i];
    const float en = __fdiv_rn(eps, p.neg_rate_f);
    const bool has_neg = isfinite(en) && en > 0.0f;
    for (int b = 0; b < p.n_block; ++b) {
        const float ef = static_cast<float>(p.epoch0 + b);
        uint32_t c = kNotDue;
        if (!(nxt > ef)) {
            nxt = __fadd_rn(nxt, eps);
            c = 0;
            if (has_neg) {
                c = floor_count(__fdiv_rn(__fsub_rn(ef, nn), en));
                nn = __fadd_rn(nn, __fmul_rn(static_cast<float>(c), en));
                if (c == kNotDue) c = kNotDue - 1;
            }
        }
        p.n_neg[static_cast<int64_t>(b) * p.m + i] = c;
    }
    p.next[i] = nxt;
    p.next_neg[i] = nn;
}

// The order of one epoch's due edges.  Times are in units of an attractive
// step: a tail is released one unit after its edge starts, a head after its
// negatives too (7/16 of a unit each; 4/16 to 11/16 were tried).  A dependent edge
// starts at least one unit after the edge it waits for, so sorting by start
// time keeps every dependency; the order within one start time is free, and
// a batch never spans two start times.  Epochs that run past kStartBuckets
// units keep the colour order instead; their batches may hold edges that
// depend on one another, so a batch's ready lanes go first there.
__global__ void __launch_bounds__(kOrderThreads, 1) order_kernel(SmallArgs p) {
    extern __shared__ uint32_t osm[];
    uint32_t* avail = osm;                     // per vertex: earliest start of its next edge
    uint32_t* seen = avail + p.n_vertices;     // per vertex: due edges so far
    uint32_t* base = seen + p.n_vertices;      // start-time histogram, then write offsets
    __shared__ uint64_t warp_sum[32];
    __shared__ uint32_t latest;
    const int tid = threadIdx.x;
    const int64_t off = static_cast<int64_t>(blockIdx.x) * p.m;
    const uint32_t* nn = p.n_neg + off;
    for (uint32_t v = tid; v < 2 * p.n_vertices + kStartBuckets; v += kOrderThreads) osm[v] = 0;
    if (tid == 0) latest = 0;
    __syncthreads();

    // the next colour's first strip is loaded while this one is worked on
    uint32_t c_next = kNotDue;
    int32_t h_next = 0, t_next = 0;
    auto prefetch = [&](int c) {
        c_next = kNotDue;
        if (c < p.n_colors) {
            const int32_t e = p.color_ptr[c] + tid;
            if (e < p.color_ptr[c + 1]) {
                c_next = nn[e];
                h_next = p.heads[e];
                t_next = p.tails[e];
            }
        }
    };
    prefetch(0);
    uint32_t last = 0;
    for (int c = 0; c < p.n_colors; ++c) {
        uint32_t cnt = c_next;
        int32_t h = h_next, t = t_next;
        prefetch(c + 1);
        const int32_t end = p.color_ptr[c + 1];
        for (int32_t e = p.color_ptr[c] + tid; e < end; e += kOrderThreads) {
            if (cnt != kNotDue) {
                const uint32_t st = max(avail[h], avail[t]);
                p.start[off + e] = st;
                p.rank_h[off + e] = seen[h]++;
                if (t != h) {
                    p.rank_t[off + e] = seen[t]++;
                    avail[t] = min(st + 1u, 0x3fffffffu);
                }
                avail[h] = min(st + 1u + (min(cnt, 4096u) * 7u) / 16u, 0x3fffffffu);
                last = max(last, st);
                atomicAdd(&base[min(st, static_cast<uint32_t>(kStartBuckets - 1))], 1u);
            }
            if (e + kOrderThreads < end) {
                cnt = nn[e + kOrderThreads];
                h = p.heads[e + kOrderThreads];
                t = p.tails[e + kOrderThreads];
            }
        }
        __syncthreads();
    }
    atomicMax(&latest, last);
    // exclusive scans of the histogram (events) and of the batches it makes
    // (up to 32 events of one start time each), kPer start times a thread
    constexpr int kPer = kStartBuckets / kOrderThreads;
    uint32_t v[kPer];
    uint64_t sum = 0;  // batches << 32 | events
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        v[k] = base[tid * kPer + k];
        sum += static_cast<uint64_t>((v[k] + 31) / 32) << 32 | v[k];
    }
    uint64_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if ((tid & 31) >= o) inc += u;
    }
    if ((tid & 31) == 31) warp_sum[tid >> 5] = inc;
    __syncthreads();
    if (tid < 32) {
        uint64_t w = warp_sum[tid];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t u = __shfl_up_sync(0xffffffffu, w, o);
            if (tid >= o) w += u;
        }
        warp_sum[tid] = w;
    }
    __syncthreads();
    const bool by_start = latest < static_cast<uint32_t>(kStartBuckets);
    const uint64_t excl = inc - sum + (tid >= 32 ? warp_sum[(tid >> 5) - 1] : 0u);
    const uint32_t total = static_cast<uint32_t>(warp_sum[31]);
    uint32_t at = static_cast<uint32_t>(excl), batch = static_cast<uint32_t>(excl >> 32);
    uint32_t* batches = p.batches + blockIdx.x * p.batch_cap;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        base[tid * kPer + k] = at;
        if (by_start)
            for (uint32_t e = 0; e < v[k]; e += 32) batches[batch++] = at + e;
        at += v[k];
    }
    uint32_t n_batches = static_cast<uint32_t>(warp_sum[31] >> 32);
    if (!by_start) {
        n_batches = (total + 31) / 32;
        for (uint32_t k = tid; k < n_batches; k += kOrderThreads) batches[k] = 32 * k;
    }
    if (tid == 0) {
        batches[n_batches] = total;
        p.n_batches[blockIdx.x] = n_batches | (by_start ? 0u : kByColor);
        if (total) atomicAdd(p.samples, static_cast<unsigned long long>(total));
        if (!by_start) base[0] = 0;  // one counter, filled colour by colour
    }
    __syncthreads();

    Event* out = p.events + off;
    const uint64_t epoch = static_cast<uint64_t>(p.epoch0 + blockIdx.x);
    auto emit = [&](int64_t e, uint32_t cnt) {
        const uint32_t st = by_start ? p.start[off + e] : 0u;
        Event ev;
        ev.ends = static_cast<uint32_t>(p.heads[e]) | static_cast<uint32_t>(p.tails[e]) << 16;
        ev.rank_h = p.rank_h[off + e];
        ev.rank_t = p.rank_t[off + e];
        ev.n_neg = cnt;
        ev.edge = static_cast<uint32_t>(p.order[e]);
        const uint64_t stream = mix64(p.seed ^ mix64(static_cast<uint64_t>(ev.edge)));
#pragma unroll
        for (int s = 0; s < kInlineNeg; ++s)
            ev.neg[s] = static_cast<uint16_t>(
                rng_below(mix64(stream ^ ((epoch << 32) | static_cast<uint32_t>(s))), p.n_vertices));
        out[atomicAdd(&base[st], 1u)] = ev;
    };
    if (by_start) {
        for (int64_t e = tid; e < p.m; e += kOrderThreads) {
            const uint32_t cnt = nn[e];
            if (cnt != kNotDue) emit(e, cnt);
        }
    } else {
        for (int c = 0; c < p.n_colors; ++c) {
            for (int32_t e = p.color_ptr[c] + tid; e < p.color_ptr[c + 1]; e += kOrderThreads) {
                const uint32_t cnt = nn[e];
                if (cnt != kNotDue) emit(e, cnt);
            }
            __syncthreads();
        }
    }
}

// A vertex in shared memory: its position and its progress, the number of due
// edges of the epoch that have updated it.  Up to three dimensions both sit
// in one word that is read and written as a whole (64 bits for one dimension,
// 128 for two and three), so a poll brings the position with the counter and
// no fence orders the two.  Wider positions keep the counter beside them, with
// acquire loads and release stores.
template <int D>
struct Vertices {
    static constexpr bool kPacked = D >= 1 && D <= 3;
    static constexpr int kWords = D == 1 ? 2 : 4;
    static constexpr int kD = D > 0 ? D : kMaxDim;
    uint32_t at;      // shared address
    uint32_t n, dim;
    __device__ static uint32_t words(uint32_t n, uint32_t dim) {
        return ((kPacked ? n * kWords : n * (dim + 1)) + 3u) & ~3u;
    }
    __device__ __forceinline__ void load(uint32_t v, float* pos, uint32_t& count) const {
        if constexpr (D == 1) {
            uint64_t w;
            asm volatile("ld.relaxed.cta.shared::cta.u64 %0, [%1];" : "=l"(w) : "r"(at + v * 8) : "memory");
            pos[0] = __uint_as_float(static_cast<uint32_t>(w));
            count = static_cast<uint32_t>(w >> 32);
        } else if constexpr (kPacked) {
            uint64_t lo, hi;
            asm volatile(
                "{\n\t.reg .b128 w;\n\t"
                "ld.relaxed.cta.shared::cta.b128 w, [%2];\n\t"
                "mov.b128 {%0, %1}, w;\n\t}"
                : "=l"(lo), "=l"(hi)
                : "r"(at + v * 16)
                : "memory");
            pos[0] = __uint_as_float(static_cast<uint32_t>(lo));
            pos[1] = __uint_as_float(static_cast<uint32_t>(lo >> 32));
            if constexpr (D == 3) pos[2] = __uint_as_float(static_cast<uint32_t>(hi));
            count = static_cast<uint32_t>(hi >> 32);
        } else {
            poll(v, pos, count);
            fetch(v, pos);
        }
    }
    // What a waiting warp reads again and again: the counter, with the position
    // where both are one word.  Wider positions are fetched once the counter is
    // right: with every poll they filled the shared-memory pipe that the
    // working warps need.
    __device__ __forceinline__ void poll(uint32_t v, float* pos, uint32_t& count) const {
        if constexpr (kPacked)
            load(v, pos, count);
        else
            asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
                         : "=r"(count)
                         : "r"(at + (n * dim + v) * 4)
                         : "memory");
    }
    __device__ __forceinline__ void fetch(uint32_t v, float* pos) const {
#pragma unroll
        for (int d = 0; d < kD; ++d)
            if (D > 0 || d < static_cast<int>(dim))
                asm volatile("ld.relaxed.cta.shared::cta.f32 %0, [%1];"
                             : "=f"(pos[d])
                             : "r"(at + (v * dim + d) * 4)
                             : "memory");
    }
    __device__ __forceinline__ uint32_t count(uint32_t v) const {
        const uint32_t word = D == 1 ? v * 2 + 1 : kPacked ? v * 4 + 3 : n * dim + v;
        uint32_t c;
        asm volatile("ld.relaxed.cta.shared::cta.u32 %0, [%1];" : "=r"(c) : "r"(at + word * 4) : "memory");
        return c;
    }
    __device__ __forceinline__ void store(uint32_t v, const float* pos, uint32_t count) const {
        if constexpr (D == 1) {
            const uint64_t w = static_cast<uint64_t>(count) << 32 | __float_as_uint(pos[0]);
            asm volatile("st.relaxed.cta.shared::cta.u64 [%0], %1;" ::"r"(at + v * 8), "l"(w) : "memory");
        } else if constexpr (kPacked) {
            const uint64_t lo = static_cast<uint64_t>(__float_as_uint(pos[1])) << 32 | __float_as_uint(pos[0]);
            uint64_t hi = static_cast<uint64_t>(count) << 32;
            if constexpr (D == 3) hi |= __float_as_uint(pos[2]);
            asm volatile(
                "{\n\t.reg .b128 w;\n\t"
                "mov.b128 w, {%1, %2};\n\t"
                "st.relaxed.cta.shared::cta.b128 [%0], w;\n\t}" ::"r"(at + v * 16),
                "l"(lo), "l"(hi)
                : "memory");
        } else {
#pragma unroll
            for (int d = 0; d < kD; ++d)
                if (D > 0 || d < static_cast<int>(dim))
                    asm volatile("st.relaxed.cta.shared::cta.f32 [%0], %1;" ::"r"(
                                     at + (v * dim + d) * 4),
                                 "f"(pos[d])
                                 : "memory");
            asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(at + (n * dim + v) * 4),
                         "r"(count)
                         : "memory");
        }
    }
};

// The reference's per-edge arithmetic (lib.rs:5172-5318) on shared-memory
// positions.  D = 0 takes the dimension at run time.
//
// A warp takes a batch of up to 32 events that could start at the same time
// and runs the ones whose turn has come, until all have run.
template <int D>
__global__ void __launch_bounds__(kSmallThreads, 1) layout_kernel(SmallArgs p) {
    extern __shared__ __align__(16) float lsm[];
    __shared__ int stop;
    __shared__ uint32_t beat;  // moves on with every kBeatEvery negatives of an event
    __shared__ uint32_t counts[kBlockEpochs];
    constexpr int kD = Vertices<D>::kD;
    const int dim = D > 0 ? D : p.dim;
    const uint32_t nv = p.n_vertices;
    const Vertices<D> verts{static_cast<uint32_t>(__cvta_generic_to_shared(lsm)), nv,
                            static_cast<uint32_t>(dim)};
    float* snap = lsm + Vertices<D>::words(nv, dim);  // positions at the epoch's start
    const int tid = threadIdx.x, lane = tid & 31;
    auto each = [&](auto&& f) {  // f(d) for every dimension
#pragma unroll
        for (int d = 0; d < kD; ++d)
            if (D > 0 || d < dim) f(d);
    };
    for (uint32_t i = tid; i < nv * dim; i += kSmallThreads) snap[i] = p.emb[i];
    __syncthreads();
    for (uint32_t v = tid; v < nv; v += kSmallThreads) verts.store(v, snap + v * dim, 0);
    for (int b = tid; b < p.n_block; b += kSmallThreads) counts[b] = p.n_batches[b];
    if (tid == 0) stop = 0;
    if (tid == 0) beat = 0;
    __syncthreads();
    const float nef = static_cast<float>(p.n_epochs);
    auto reached = [&] {  // moves on whenever a warp gets further within an epoch
        uint32_t sum = lane == 0 ? *static_cast<volatile uint32_t*>(&beat) : 0u;
        for (uint32_t v = lane; v < nv; v += 32) sum += verts.count(v);
        return __reduce_add_sync(0xffffffffu, sum);
    };

    for (int b = 0; b < p.n_block; ++b) {
        const int n_batches = static_cast<int>(counts[b] & ~kByColor);
        const bool together = (counts[b] & kByColor) == 0;
        const uint32_t* start = p.batches + static_cast<int64_t>(b) * p.batch_cap;
        const uint4* ev4 = reinterpret_cast<const uint4*>(p.events + static_cast<int64_t>(b) * p.m);
        // the next batch's events and the bounds of the one after it are on
        // the way while a batch is worked on
        int j = tid >> 5;
        uint32_t first = 0, last = 0, first1 = 0, last1 = 0;
        uint4 q0 = make_uint4(0, 0, 0, 0), q1 = q0, q2 = q0;
        auto bounds = [&](int k, uint32_t& lo, uint32_t& hi) {
            lo = k < n_batches ? __ldg(start + k) : 0u;
            hi = k < n_batches ? __ldg(start + k + 1) : 0u;
        };
        auto load = [&](uint32_t lo, uint32_t hi) {
            if (lo + lane < hi) {
                q0 = __ldg(ev4 + 3 * (lo + lane));
                q1 = __ldg(ev4 + 3 * (lo + lane) + 1);
                q2 = __ldg(ev4 + 3 * (lo + lane) + 2);
            }
        };
        bounds(j, first, last);
        bounds(j + kWarps, first1, last1);
        load(first, last);
        __syncthreads();
        if (stop) return;  // a wait ran out: the host reports it
        for (uint32_t v = tid; v < nv; v += kSmallThreads) {
            float x[kD];
            uint32_t c;
            verts.load(v, x, c);
            each([&](int d) { snap[v * dim + d] = x[d]; });
            verts.store(v, x, 0);
        }
        __syncthreads();
        const int64_t epoch = p.epoch0 + b;
        const float alpha = p.lr * (1.0f - static_cast<float>(epoch) / nef);
        for (; j < n_batches; j += kWarps) {
            const uint4 e0 = q0, e1 = q1, e2 = q2;
            unsigned todo = last - first >= 32 ? 0xffffffffu : (1u << (last - first)) - 1u;
            first = first1;
            last = last1;
            load(first, last);
            bounds(j + 2 * kWarps, first1, last1);
            const uint32_t head = e0.x & 0xffffu, tail = e0.x >> 16;
            const uint32_t rank_h = e0.y, rank_t = e0.z, n_neg = e0.w;
            // negative s of the event, 16 bits each
            auto neg_of = [&](int s) {
                const uint32_t w[7] = {e1.y, e1.z, e1.w, e2.x, e2.y, e2.z, e2.w};
                return (s & 1) ? w[s >> 1] >> 16 : w[s >> 1] & 0xffffu;
            };
            uint32_t idle = 0, seen = ~0u;
            while (todo) {
                bool ready = false;
                float h[kD], t[kD];
                if ((todo >> lane) & 1u) {
                    uint32_t ch, ct;
                    verts.poll(head, h, ch);
                    verts.poll(tail, t, ct);
                    ready = ch == rank_h && (ct == rank_t || head == tail);
                }
                unsigned now = __ballot_sync(0xffffffffu, ready);
                if (together && now != todo) {
                    now = 0;
                    ready = false;
                }
                todo &= ~now;
                if (now == 0) {
                    if ((++idle & 1023u) == 0) {
                        if (idle > kSpinLimit) {
                            const uint32_t at = reached();
                            if (at != seen) idle = 0;
                            seen = at;
                        }
                        if (__any_sync(0xffffffffu,
                                       idle > kSpinLimit || *static_cast<volatile int*>(&stop))) {
                            *static_cast<volatile int*>(&stop) = 1;
                            *p.err = 1;
                            j = n_batches;
                            break;
                        }
                    }
                    continue;
                }
                if (ready) {
                    if constexpr (!Vertices<D>::kPacked) {
                        verts.fetch(head, h);
                        verts.fetch(tail, t);
                    }
                    {
                        float d2 = 0.0f;
                        each([&](int d) {
                            const float df = __fsub_rn(h[d], t[d]);
                            d2 = __fadd_rn(d2, __fmul_rn(df, df));
                        });
                        const float pb = pow_pos(d2, p.b);
                        const float gc = __fdiv_rn(__fmul_rn(p.att_factor, __fdiv_rn(pb, d2)),
                                                   __fadd_rn(__fmul_rn(p.a, pb), 1.0f));
                        const bool moves = head != tail && d2 > 0.0f;
                        each([&](int d) {
                            const float mv =
                                __fmul_rn(clip4(__fmul_rn(gc, __fsub_rn(h[d], t[d]))), alpha);
                            h[d] = moves ? __fadd_rn(h[d], mv) : h[d];
                            t[d] = moves ? __fsub_rn(t[d], mv) : t[d];
                        });
                        if (head != tail) verts.store(tail, t, rank_t + 1);
                    }
                    auto repel = [&](const float* o, bool use) {
                        float d2 = 0.0f;
                        each([&](int d) {
                            const float df = __fsub_rn(h[d], o[d]);
                            d2 = __fadd_rn(d2, __fmul_rn(df, df));
                        });
                        const float pb = pow_pos(d2, p.b);
                        const float gc = __fdiv_rn(
                            p.rep_factor, __fmul_rn(__fadd_rn(0.001f, d2),
                                                    __fadd_rn(__fmul_rn(p.a, pb), 1.0f)));
                        const bool moves = use && d2 > 0.0f && gc > 0.0f;
                        each([&](int d) {
                            const float v = __fadd_rn(
                                h[d],
                                __fmul_rn(clip4(__fmul_rn(gc, __fsub_rn(h[d], o[d]))), alpha));
                            h[d] = moves ? v : h[d];
                        });
                    };
                    if (n_neg == 0) verts.store(head, h, rank_h + 1);
                    const uint32_t most = __reduce_max_sync(now, n_neg);
                    float o[kD], on[kD];
                    each([&](int d) { o[d] = snap[neg_of(0) * dim + d]; });
#pragma unroll
                    for (int s = 0; s < kInlineNeg; ++s) {
                        if (s >= most) break;
                        // the next position is on the way while this step is worked out
                        if (s + 1 < kInlineNeg)
                            each([&](int d) { on[d] = snap[neg_of(s + 1) * dim + d]; });
                        repel(o, s < n_neg && neg_of(s) != head);
                        each([&](int d) { o[d] = on[d]; });
                        // a lane frees its head as soon as its own negatives are done
                        if (s + 1 == n_neg) verts.store(head, h, rank_h + 1);
                    }
                    for (uint32_t s = kInlineNeg; s < n_neg;) {
                        const uint32_t end = min(n_neg, s + kBeatEvery);
                        for (; s < end; ++s) {
                            const uint64_t word =
                                rng_word(p.seed, e1.x, (static_cast<uint64_t>(epoch) << 32) | s);
                            const uint32_t v = rng_below(word, nv);
                            each([&](int d) { o[d] = snap[v * dim + d]; });
                            repel(o, v != head);
                            if (s + 1 == n_neg) verts.store(head, h, rank_h + 1);
                        }
                        volatile uint32_t* const at = &beat;
                        *at = *at + 1;
                    }
                }
                __syncwarp();  // the next polls see these updates
            }
        }
    }
    __syncthreads();
    for (uint32_t v = tid; v < nv; v += kSmallThreads) {
        float x[kD];
        uint32_t c;
        verts.load(v, x, c);
        each([&](int d) { p.emb[v * dim + d] = x[d]; });
    }
}

// Greedy edge colouring in graph order: each edge takes the smallest colour
// not yet used at its head or its tail.  A vertex's used colours are a row of
// `words` 64-bit words, widened when a colour does not fit.
std::vector<int32_t> color_edges(const std::vector<int32_t>& heads,
                                 const std::vector<int32_t>& tails, int64_t n, int* n_colors) {
    const int64_t m = static_cast<int64_t>(heads.size());
    size_t words = 4;
    std::vector<uint64_t> used(n * words, 0);
    std::vector<int32_t> color(m);
    int top = 0;
    for (int64_t e = 0; e < m; ++e) {
        uint64_t* uh = used.data() + heads[e] * words;
        uint64_t* ut = used.data() + tails[e] * words;
        size_t w = 0;
        while (w < words && (uh[w] | ut[w]) == ~uint64_t{0}) ++w;
        if (w == words) {
            std::vector<uint64_t> wide(n * words * 2, 0);
            for (int64_t v = 0; v < n; ++v)
                std::copy_n(used.data() + v * words, words, wide.data() + v * words * 2);
            used.swap(wide);
            words *= 2;
            uh = used.data() + heads[e] * words;
            ut = used.data() + tails[e] * words;
        }
        const int bit = __builtin_ctzll(~(uh[w] | ut[w]));
        uh[w] |= uint64_t{1} << bit;
        ut[w] |= uint64_t{1} << bit;
        color[e] = static_cast<int32_t>(w * 64 + bit);
        top = std::max(top, color[e] + 1);
    }
    *n_colors = top;
    return color;
}

}  // namespace

double optimize_layout_small(float* emb, int64_t n_vertices, int dim, const Graph& g,
                             int64_t n_epochs, float a, float b, float lr, int64_t neg_rate,
                             float repulsion, uint64_t seed, float* kernel_ms, cudaStream_t s) {
    const int64_t m = g.n_edges;
    std::vector<int32_t> hh(m), th(m);
    UMAPB_CUDA(cudaMemcpyAsync(hh.data(), g.heads.get(), m * 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(th.data(), g.tails.get(), m * 4, cudaMemcpyDeviceToHost, s));
    const float mx = std::max(max_weight(g.weights.get(), m, s), 1e-12f);  // waits for the stream
    int n_colors = 0;
    const std::vector<int32_t> color = color_edges(hh, th, n_vertices, &n_colors);
    std::vector<int32_t> ptr(n_colors + 1, 0), order(m);
    for (int32_t c : color) ++ptr[c + 1];
    for (int c = 0; c < n_colors; ++c) ptr[c + 1] += ptr[c];
    {
        std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
        for (int64_t e = 0; e < m; ++e) order[fill[color[e]]++] = static_cast<int32_t>(e);
    }
    const float nrf = static_cast<float>(neg_rate);
    // one batch per 32 events, one more per start time, the total
    const int64_t batch_cap = m / 32 + std::min<int64_t>(m, kStartBuckets) + 1;
    const int64_t per_epoch = m * static_cast<int64_t>(sizeof(Event) + 4 * sizeof(uint32_t)) +
                              (batch_cap + 1) * static_cast<int64_t>(sizeof(uint32_t));
    const int64_t block = std::max<int64_t>(
        1, std::min({n_epochs, kBlockEpochs, static_cast<int64_t>(kBlockBytes) / per_epoch}));
    // The work space in whole steps of kBlockStep, so that graphs of like size
    // ask for the same block.  It is not the model's: 1,000 rows take 224 MB of
    // it for 148 epochs, and a new block of that size costs 3 ms.  Fewer epochs at
    // a time would need less, but every block's order_kernel (0.2 to 0.5 ms)
    // comes before its layout.
    WorkBlock work(ceil_div(block * per_epoch, static_cast<int64_t>(kBlockStep)) * kBlockStep, s);
    DevBuf<int32_t> dorder(m, s), dh(m, s), dt(m, s), dptr(n_colors + 1, s);
    DevBuf<float> deps(m, s), dnext(m, s), dneg(m, s);
    DevBuf<unsigned long long> samples(1, s);
    DevBuf<int> err(1, s);
    UMAPB_CUDA(cudaMemcpyAsync(dorder.get(), order.data(), m * 4, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(dptr.get(), ptr.data(), (n_colors + 1) * 4, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemsetAsync(samples.get(), 0, 8, s));
    UMAPB_CUDA(cudaMemsetAsync(err.get(), 0, 4, s));
    SmallArgs p{};
    p.emb = emb;
    p.m = m;
    p.n_vertices = static_cast<uint32_t>(n_vertices);
    p.dim = dim;
    p.order = dorder.get();
    p.heads = dh.get();
    p.tails = dt.get();
    p.eps = deps.get();
    p.next = dnext.get();
    p.next_neg = dneg.get();
    p.color_ptr = dptr.get();
    p.n_colors = n_colors;
    p.events = static_cast<Event*>(work.ptr);
    p.n_neg = reinterpret_cast<uint32_t*>(p.events + block * m);
    p.start = p.n_neg + block * m;
    p.rank_h = p.start + block * m;
    p.rank_t = p.rank_h + block * m;
    p.batches = p.rank_t + block * m;
    p.n_batches = p.batches + block * batch_cap;
    p.batch_cap = batch_cap;
    p.samples = samples.get();
    p.err = err.get();
    p.n_epochs = n_epochs;
    p.lr = lr;
    p.a = a;
    p.b = b;
    p.att_factor = -2.0f * a * b;
    p.rep_factor = 2.0f * repulsion * b;
    p.neg_rate_f = nrf;
    p.seed = seed;
    const unsigned grid = static_cast<unsigned>(ceil_div(m, 256));
    const int order_smem = static_cast<int>((2 * n_vertices + kStartBuckets) * sizeof(uint32_t));
    // positions with their counters (Vertices), and the epoch's starting positions
    const int64_t vertex_words = dim == 1 ? 2 : dim <= 3 ? 4 : dim + 1;
    const int layout_smem = static_cast<int>(
        (ceil_div(n_vertices * vertex_words, 4) + ceil_div(n_vertices * dim, 4)) * 16);
    auto layout = dim == 1   ? layout_kernel<1>
                  : dim == 2 ? layout_kernel<2>
                  : dim == 3 ? layout_kernel<3>
                  : dim == 4 ? layout_kernel<4>
                             : layout_kernel<0>;
    allow_shared(order_kernel, 1024);
    allow_shared(layout, 1024);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (kernel_ms) {
        UMAPB_CUDA(cudaEventCreate(&e0));
        UMAPB_CUDA(cudaEventCreate(&e1));
        UMAPB_CUDA(cudaEventRecord(e0, s));
    }
    gather_kernel<<<grid, 256, 0, s>>>(dorder.get(), g.heads.get(), g.tails.get(),
                                       g.weights.get(), mx, static_cast<float>(n_epochs), nrf, m,
                                       dh.get(), dt.get(), deps.get(), dnext.get(), dneg.get());
    UMAPB_LAUNCH_CHECK();
    for (int64_t ep = 0; ep < n_epochs; ep += block) {
        p.epoch0 = ep;
        p.n_block = static_cast<int>(std::min(block, n_epochs - ep));
        due_kernel<<<grid, 256, 0, s>>>(p);
        UMAPB_LAUNCH_CHECK();
        order_kernel<<<static_cast<unsigned>(p.n_block), kOrderThreads, order_smem, s>>>(p);
        UMAPB_LAUNCH_CHECK();
        layout<<<1, kSmallThreads, layout_smem, s>>>(p);
        UMAPB_LAUNCH_CHECK();
    }
    if (kernel_ms) {
        UMAPB_CUDA(cudaEventRecord(e1, s));
        UMAPB_CUDA(cudaEventSynchronize(e1));
        UMAPB_CUDA(cudaEventElapsedTime(kernel_ms, e0, e1));
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    unsigned long long count = 0;
    int failed = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&count, samples.get(), 8, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(&failed, err.get(), 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    work.keep(kBlockBytes);
    if (failed) throw Error(UMAPB_ERR_CUDA, "the small-graph layout stopped on a wait limit");
    return static_cast<double>(count);
}

}  // namespace umapb
