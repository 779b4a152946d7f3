// spectral.cu - spectral initialisation (rust_umap/src/lib.rs:3841-4791).
//
// The reference runs, per connected component, block subspace iteration on
// the shifted operator I + D^-1/2 W D^-1/2: 256 iterations, s = (dim+1)*6
// columns, modified Gram-Schmidt applied twice in FP64, then a Rayleigh-Ritz
// step (lib.rs:4227-4326).  Here all components of the graph that take the
// iterative path run at once: the sparse product is one pull-style SpMM over
// the CSR graph (components never share edges, so the operator is block
// diagonal), the block is kept in FP32 (N x s, L2 resident at 1M rows), and
// orthonormalisation is CholQR2 per component: the s x s Gram matrix is
// reduced in FP64, factored in FP64 on the device, and its inverse factor is
// applied in FP64.  CholQR and MGS produce the same orthonormal basis in exact
// arithmetic (the unique QR factor with positive diagonal); the MGS failure
// test (column norm^2 <= 1e-12 after projection, lib.rs:4188) is the
// Cholesky pivot test.  The block is orthonormalised after every fourth
// product instead of every product: the span of (I + A)^4 X does not depend
// on whether X was re-orthonormalised in between (exactly so in exact
// arithmetic), and over four products of an operator with spectrum in [0, 2]
// the columns' condition grows by at most 2^4 on the bulk of the spectrum,
// far inside what an FP64 Gram matrix of FP32 columns resolves.  256 is a
// multiple of 4, so the last product is followed by an orthonormalisation as
// in the reference.  The Ritz matrices are solved on the host.
//
// Small pieces follow the reference on the host: the dense Laplacian path
// (lib.rs:4007-4069, 3917-3957) for components below 128 nodes or connected
// inputs with <= 8 features and <= 2048 rows, random init for components
// with fewer than 2*dim nodes, and the meta layout of component centroids
// (lib.rs:4519-4554).  Random numbers (initial block, noise, random layouts)
// come from counter-based streams, not the reference's SmallRng sequence.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "kernels.cuh"

namespace umapb {
namespace {

constexpr int kIters = 256;             // SPECTRAL_ITERATIVE_MAX_ITERS (lib.rs:31)
constexpr int kOrthoEvery = 4;          // products between orthonormalisations
constexpr int kOversampling = 6;        // lib.rs:32
constexpr int64_t kComponentIterThreshold = 128;  // lib.rs:30
constexpr int64_t kDenseFallbackMax = 4096;       // lib.rs:33
constexpr double kOrthoEps = 1e-12;     // lib.rs:34
constexpr float kInitMaxCoord = 10.0f;  // lib.rs:22
constexpr float kInitNoise = 1e-4f;     // lib.rs:23
constexpr int kMaxS = 32;               // s <= 32 -> n_components <= 4
// Edges above which a row of a product takes a CTA: a row a short path walks
// costs about 0.09 us per edge whatever the others do, so rows are long where
// that would outlast a quarter of the whole product (10 ps per edge), but not
// below 96 edges, where a CTA costs as much as the walk.  At 1M x 64 a fixed 96
// made the products 99 ms a fit, the rule (671) 88.
constexpr int32_t kLongRowMin = 96, kLongRowMax = 1024;
constexpr int64_t kEdgesPerLongEdge = 36000;

inline unsigned grid_for(int64_t n, int t = 256) {
    return static_cast<unsigned>(ceil_div(std::max<int64_t>(n, 1), t));
}

// ---------------------------------------------------- components (device)
__device__ inline int32_t find_root(const int32_t* parent, int32_t x) {
    int32_t p = parent[x];
    while (p != x) {
        x = p;
        p = parent[x];
    }
    return x;
}

__global__ void cc_init(int32_t* parent, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) parent[i] = static_cast<int32_t>(i);
}

__global__ void cc_hook(const int32_t* __restrict__ heads, const int32_t* __restrict__ tails,
                        int64_t m, int32_t* parent, int* changed) {
    const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const int32_t u = heads[e], v = tails[e];
    if (u >= v) return;  // each undirected pair once
    const int32_t ru = find_root(parent, u), rv = find_root(parent, v);
    if (ru == rv) return;
    const int32_t hi = ru > rv ? ru : rv, lo = ru > rv ? rv : ru;
    atomicMin(&parent[hi], lo);
    *changed = 1;
}

__global__ void cc_compress(int32_t* parent, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) parent[i] = find_root(parent, static_cast<int32_t>(i));
}

__global__ void cc_is_root(const int32_t* parent, int64_t n, int32_t* flag) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) flag[i] = parent[i] == i ? 1 : 0;
}

__global__ void cc_label(const int32_t* parent, const int32_t* rank, int64_t n, int32_t* label) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) label[i] = rank[parent[i]];
}

__global__ void iota_kernel(int32_t* v, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = static_cast<int32_t>(i);
}

// --------------------------------------------------- subspace iteration --
__global__ void degree_kernel(const int32_t* __restrict__ row_ptr, const float* __restrict__ w,
                              int64_t n, double* __restrict__ deg, float* __restrict__ dinv) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int32_t e = row_ptr[i]; e < row_ptr[i + 1]; ++e) s += static_cast<double>(w[e]);
    deg[i] = s;
    dinv[i] = s > 0.0 ? static_cast<float>(1.0 / sqrt(s)) : 0.0f;
}

__global__ void norm_weight_kernel(const int32_t* __restrict__ heads,
                                   const int32_t* __restrict__ tails, const float* __restrict__ w,
                                   const double* __restrict__ deg, int64_t m,
                                   float* __restrict__ nw) {
    const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const double di = deg[heads[e]], dj = deg[tails[e]];
    const double ii = di > 0.0 ? 1.0 / sqrt(di) : 0.0, ij = dj > 0.0 ? 1.0 / sqrt(dj) : 0.0;
    nw[e] = static_cast<float>(static_cast<double>(w[e]) * ii * ij);
}

// The iterative components' rows are processed in "position" order: the
// nodes of slot 0, then slot 1, ... (slots = components on the iterative
// path).  Blocks X and Y are stored in that order, so every pass except the
// SpMM gathers streams contiguous memory.

__global__ void pos_kernel(const int32_t* __restrict__ nodes, int64_t cnt, int32_t* __restrict__ pos) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p < cnt) pos[nodes[p]] = static_cast<int32_t>(p);
}

// The CSR of the shifted operator in position order.  A row's edges start at
// a multiple of four (rows are padded to whole quads), so four tails and four
// weights arrive in one 16-byte load each.
__global__ void prow_len_kernel(const int32_t* __restrict__ nodes, int64_t cnt,
                                const int32_t* __restrict__ row_ptr, int32_t* __restrict__ len,
                                int32_t* __restrict__ quads, int32_t long_row,
                                int32_t* __restrict__ long_rows,
                                int32_t* __restrict__ n_long) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p < cnt) {
        const int32_t v = nodes[p];
        const int32_t l = row_ptr[v + 1] - row_ptr[v];
        len[p] = l;
        quads[p] = (l + 3) / 4;
        if (l > long_row) long_rows[atomicAdd(n_long, 1)] = static_cast<int32_t>(p);
    }
}

__global__ void pcsr_kernel(const int32_t* __restrict__ nodes, int64_t cnt,
                            const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ tails,
                            const float* __restrict__ nw, const int32_t* __restrict__ pos,
                            const int32_t* __restrict__ qptr, int32_t* __restrict__ ptails,
                            float* __restrict__ pnw) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= cnt) return;
    const int32_t v = nodes[p];
    int64_t o = static_cast<int64_t>(qptr[p]) * 4;
    for (int32_t e = row_ptr[v]; e < row_ptr[v + 1]; ++e, ++o) {
        ptails[o] = pos[tails[e]];
        pnw[o] = nw[e];
    }
    for (; o & 3; ++o) {  // padding: never used, but read
        ptails[o] = static_cast<int32_t>(p);
        pnw[o] = 0.0f;
    }
}

// Initial block: column 0 = sqrt(degree), the others U(-1, 1) (lib.rs:4254-4261).
__global__ void init_block_kernel(const int32_t* __restrict__ nodes, int64_t cnt,
                                  const int32_t* __restrict__ slot_of_pos,
                                  const uint64_t* __restrict__ slot_seed,
                                  const double* __restrict__ deg, int s, int sp,
                                  float* __restrict__ X) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cnt) return;
    const int32_t i = nodes[t];
    const uint64_t seed = slot_seed[slot_of_pos[t]] ^ 0x7A5B3D91CE42A117ULL;
    float* row = X + t * sp;
    row[0] = static_cast<float>(sqrt(deg[i]));
    for (int c = 1; c < sp; ++c) {
        float v = 0.0f;
        if (c < s) v = static_cast<float>(-1.0 + 2.0 * rng_unit_f64(rng_word(seed, i, c)));
        row[c] = v;
    }
}

// Y = X + A_hat X in position order.  A row's sum adds its edges in edge
// order, whatever path it takes.
//
// Short rows: SP / 4 lanes share a row, one float4 of it each, four edges at a
// time, the next four tails and weights on the way.
// Long rows: a CTA each, started first.  All threads gather the next
// kLongChunk edges' rows while one warp, a lane per column, adds the previous
// chunk from shared memory, so a hub costs about 7 cycles an edge instead of a
// memory round trip for every four.
constexpr int kSpmmThreads = 256;
constexpr int kLongChunk = 128;

// The products and the orthonormalisation are a chain of some 450 short
// launches, each reading what the one before wrote.  They are launched with
// programmatic serialisation: a kernel's CTAs may be resident while the one
// before still runs, and wait here until it has finished and its writes can
// be seen.  The next kernel is let in only after that wait, so no kernel runs
// beside the one before the last, and what the chain writes is read with
// plain loads after the wait.  1,000 rows 5.65 -> 4.75 ms, 20,000 x 192 10.9 ->
// 10.05, 100,000 20.2 -> 19.2; level at 150,000 and 200,000 rows, where the
// waiting CTAs take the places of running ones about as often as they save a
// launch, and slower at 1M (325 -> 342), so from kEarlyRows on a kernel starts
// when the one before has ended.
constexpr int64_t kEarlyRows = 131072;
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
void launch_chained(void (*kernel)(Params...), bool early, dim3 grid, int threads, cudaStream_t s,
                    Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    UMAPB_CUDA(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
    UMAPB_LAUNCH_CHECK();
}

template <int SP>
constexpr int spmm_rows_per_block() { return kSpmmThreads / 32 * (32 / (SP / 4)); }

template <int SP>
__device__ __forceinline__ void spmm_long_row(int64_t t, const int32_t* __restrict__ qptr,
                                              const int32_t* __restrict__ len,
                                              const int32_t* __restrict__ ptails,
                                              const float* __restrict__ pnw, const float* X,
                                              float* Y) {
    constexpr int V = SP / 4, GL = V <= 4 ? 4 : 8;  // lanes of a gathered row
    constexpr int kGroups = kSpmmThreads / GL;
    constexpr int kPer = kLongChunk / kGroups;  // edges a group gathers per chunk
    __shared__ __align__(16) float tile[2][kLongChunk * SP];
    __shared__ float wt[2][kLongChunk];
    const int tid = threadIdx.x, grp = tid / GL, v = tid % GL;
    const int32_t n = len[t];
    const int64_t st = static_cast<int64_t>(qptr[t]) * 4;
    float4 q[kPer];
    float w[kPer];
    int32_t id[kPer];
    auto ids = [&](int32_t e0) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int32_t e = e0 + grp + k * kGroups;
            id[k] = e < n ? __ldg(ptails + st + e) : -1;
            w[k] = e < n ? __ldg(pnw + st + e) : 0.0f;
        }
    };
    auto gather = [&] {
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (v < V && id[k] >= 0)
                q[k] = reinterpret_cast<const float4*>(X + static_cast<int64_t>(id[k]) * SP)[v];
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int e = grp + k * kGroups;
            if (v < V && id[k] >= 0) reinterpret_cast<float4*>(tile[buf] + e * SP)[v] = q[k];
            if (v == 0) wt[buf][e] = w[k];
        }
    };
    float acc = tid < SP ? X[t * SP + tid] : 0.0f;
    ids(0);
    gather();
    put(0);
    for (int32_t e0 = 0; e0 < n; e0 += kLongChunk) {
        const int buf = (e0 / kLongChunk) & 1;
        const bool more = e0 + kLongChunk < n;
        if (more) ids(e0 + kLongChunk);
        __syncthreads();
        if (more) gather();
        if (tid < SP) {
            const int32_t m = min(kLongChunk, n - e0);
            int32_t e = 0;
            for (; e + 8 <= m; e += 8) {
                float x[8], a[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    x[k] = tile[buf][(e + k) * SP + tid];
                    a[k] = wt[buf][e + k];
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) acc = fmaf(a[k], x[k], acc);
            }
            for (; e < m; ++e) acc = fmaf(wt[buf][e], tile[buf][e * SP + tid], acc);
        }
        if (more) put(buf ^ 1);
    }
    if (tid < SP) Y[t * SP + tid] = acc;
}

template <int SP>
__global__ void __launch_bounds__(kSpmmThreads, 4)
    spmm_kernel(int64_t cnt, const int32_t* __restrict__ qptr, const int32_t* __restrict__ len,
                const int32_t* __restrict__ ptails, const float* __restrict__ pnw,
                const int32_t* __restrict__ long_rows, int n_long, int32_t long_row,
                const float* X, float* Y) {
    wait_for_previous();
    if (static_cast<int>(blockIdx.x) < n_long) {
        spmm_long_row<SP>(long_rows[blockIdx.x], qptr, len, ptails, pnw, X, Y);
        return;
    }
    constexpr int V = SP / 4, RW = 32 / V;
    const int lane = threadIdx.x & 31;
    const int sub = lane / V, v = lane - sub * V;
    const int64_t t = static_cast<int64_t>(blockIdx.x - n_long) * spmm_rows_per_block<SP>() +
                      (threadIdx.x >> 5) * RW + sub;
    if (sub >= RW || t >= cnt) return;
    const int32_t n = len[t];
    if (n > long_row) return;
    const int32_t q0 = qptr[t];
    const int4* id4 = reinterpret_cast<const int4*>(ptails) + q0;
    const float4* w4 = reinterpret_cast<const float4*>(pnw) + q0;
    const float4* x4 = reinterpret_cast<const float4*>(X);
    float4 acc = x4[t * V + v];
    auto add = [&](float w, const float4& q) {
        acc.x = fmaf(w, q.x, acc.x);
        acc.y = fmaf(w, q.y, acc.y);
        acc.z = fmaf(w, q.z, acc.z);
        acc.w = fmaf(w, q.w, acc.w);
    };
    auto row = [&](int32_t i) { return x4[static_cast<int64_t>(i) * V + v]; };
    int32_t e = 0;
    if (n > 0) {
        int4 id = __ldg(id4);
        float4 w = __ldg(w4);
#pragma unroll 1  // two quads at a time were 4% slower at 1M rows
        for (; e + 4 <= n; e += 4) {
            const float4 a = row(id.x), b = row(id.y), c = row(id.z), d = row(id.w);
            const float4 wc = w;
            if (e + 4 < n) {  // the next quad's tails and weights
                id = __ldg(id4 + e / 4 + 1);
                w = __ldg(w4 + e / 4 + 1);
            }
            add(wc.x, a);
            add(wc.y, b);
            add(wc.z, c);
            add(wc.w, d);
        }
        if (e < n) {
            const float4 a = row(id.x), b = row(id.y), c = row(id.z);  // padding reads its own row
            add(w.x, a);
            if (e + 1 < n) add(w.y, b);
            if (e + 2 < n) add(w.z, c);
        }
    }
    reinterpret_cast<float4*>(Y)[t * V + v] = acc;
}

struct Chunk {
    int32_t slot;
    int32_t start;  // position range [start, end)
    int32_t end;
    int32_t first;  // index of the slot's first chunk
    int32_t of;     // chunks of the slot
    int32_t bundle; // index of the slot's first bundle of kBundle chunks
};
constexpr int kBundle = 16;

// Upper triangle of A^T B over a chunk's rows, FP64.  S is a multiple of 3
// ((dim + 1) * 6), so the upper triangle is covered by NT = T (T + 1) / 2
// tiles of 3 x 3 entries (T = S / 3).  The rows of a chunk are dealt to G
// groups (row r of each slab of R rows to group r % G) and a thread keeps one
// tile of one group; the groups' tiles are then added in order.
constexpr int kOrthoThreads = 256;

template <int S, int SP>
struct GramShape {
    static_assert(S % 3 == 0, "the block width is a multiple of 3");
    static constexpr int T = S / 3;
    static constexpr int NT = T * (T + 1) / 2;
    static constexpr int G = kOrthoThreads / NT;
    static constexpr int R = SP <= 20 ? 128 : 64;  // rows per slab
    static constexpr int kRounds = (R + G - 1) / G;  // rows of a group in a slab
    static constexpr int kStage = kRounds * G;     // rows staged at a time
    static constexpr int kTile = NT * 9;           // doubles of a group's tiles
};

template <int S, int SP>
struct GramTile {
    using Sh = GramShape<S, SP>;
    double acc[3][3];
    int tile, grp, tp, tq;
    bool worker;
    __device__ __forceinline__ void init(int groups) {
        const int tid = threadIdx.x;
        worker = tid < groups * Sh::NT;
        tile = tid % Sh::NT;
        grp = tid / Sh::NT;
        tile_at(tile, &tp, &tq);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) acc[i][j] = 0.0;
    }
    // tile t covers rows 3 p.., columns 3 q.., p <= q
    static __device__ __forceinline__ void tile_at(int t, int* p, int* q) {
        int pp = 0, qq = t;
        while (qq >= Sh::T - pp) {
            qq -= Sh::T - pp;
            ++pp;
        }
        *p = pp;
        *q = qq + pp;
    }
    __device__ __forceinline__ void add(const double* As, const double* Bs, int rows, int groups) {
        if (!worker) return;
#pragma unroll 2
        for (int r = grp; r < rows; r += groups) {
            const double* ar = As + r * SP + 3 * tp;
            const double* br = Bs + r * SP + 3 * tq;
            const double a0 = ar[0], a1 = ar[1], a2 = ar[2];
            const double b0 = br[0], b1 = br[1], b2 = br[2];
            acc[0][0] = fma(a0, b0, acc[0][0]);
            acc[0][1] = fma(a0, b1, acc[0][1]);
            acc[0][2] = fma(a0, b2, acc[0][2]);
            acc[1][0] = fma(a1, b0, acc[1][0]);
            acc[1][1] = fma(a1, b1, acc[1][1]);
            acc[1][2] = fma(a1, b2, acc[1][2]);
            acc[2][0] = fma(a2, b0, acc[2][0]);
            acc[2][1] = fma(a2, b1, acc[2][1]);
            acc[2][2] = fma(a2, b2, acc[2][2]);
        }
    }
    __device__ __forceinline__ void store(double* to) const {
        if (!worker) return;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) to[grp * Sh::kTile + tile * 9 + i * 3 + j] = acc[i][j];
    }
    // entry o of a group's tiles: row and column, false in the lower triangle
    static __device__ __forceinline__ bool entry(int o, int* row, int* col) {
        const int t = o / 9, ij = o - t * 9, i = ij / 3;
        int p, q;
        tile_at(t, &p, &q);
        *row = 3 * p + i;
        *col = 3 * q + ij - i * 3;
        return *row <= *col;
    }
};

// G = L L^T of one slot, one warp: lane i keeps row i; right-looking updates
// with the pivot column shared by shuffles.  A pivot <= 1e-12 is the MGS
// failure of the reference (column norm^2 after projection); the factor is
// then the identity.  `g` (shared memory) holds the upper triangle.
template <int S>
__device__ void chol_factor(const double* g, double* Lout, double* dinv, int* fail) {
    const int lane = threadIdx.x & 31;
    double row[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
        double v = 0.0;
        if (lane < S) v = lane <= k ? g[lane * S + k] : g[k * S + lane];
        row[k] = v;
    }
    bool ok = true;
    double diag = 1.0;
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const double pivot = __shfl_sync(0xffffffffu, row[j], j);
        if (!(pivot > kOrthoEps) || !isfinite(pivot)) {
            ok = false;
            break;
        }
        const double ljj = sqrt(pivot);
        const double lij = lane == j ? ljj : row[j] / ljj;
        if (lane == j) diag = ljj;
        if (lane >= j) row[j] = lij;
#pragma unroll
        for (int k = j + 1; k < S; ++k) {
            const double lkj = __shfl_sync(0xffffffffu, lij, k);
            if (lane > j) row[k] = fma(-lij, lkj, row[k]);
        }
    }
    if (!ok && lane == 0) *fail = 1;
    if (lane < S) {
#pragma unroll
        for (int k = 0; k < S; ++k)  // column-major: the solve reads columns
            Lout[k * S + lane] = ok ? (k <= lane ? row[k] : 0.0) : (k == lane ? 1.0 : 0.0);
        dinv[lane] = ok ? 1.0 / diag : 1.0;
    }
}

struct OrthoArgs {
    const Chunk* chunks;
    const float* Y;
    float* X;
    double* L;       // [slot][S][S], column-major
    double* dinv;    // [slot][S]: 1 / diagonal
    double* part;    // [chunk][G][kTile]: tiles of the groups, where a chunk has several CTAs
    double* sums;    // [chunk][kTile]: Gram matrices of the chunks
    double* bundle;  // [bundle][kTile]: sums of kBundle chunks each
    int* chunk_done;   // CTAs done with the chunk; 0 between launches
    int* bundle_done;  // chunks done of the bundle; 0 between launches
    int* slot_done;    // bundles done of the slot; 0 between launches
    int* fail;
    int groups;      // row groups of a CTA (blockIdx.y takes the next `groups`)
};

// One pass of CholQR2, which is gram | solve + gram | solve:
//   kSolve: X = Y L^-T by forward substitution, FP64 (else X is Y);
//   kGram:  the Gram matrix of X; the last CTA of a slot factors it.
// A chunk's row groups are dealt to several CTAs where there are few chunks;
// each solves and sums only the rows of its groups, and the sums are added in
// the same order however they are dealt (groups in order, then chunks in
// order, kBundle at a time), so the factor does not depend on the split or on
// timing.
//
// Bound by the FP64 operands' way through shared memory at 1M rows and by
// latency at 20,000 and fewer: the launch, the slabs of one CTA, and the
// factor's chain of 18 square roots and divisions.  An orthonormalisation (two
// passes) of 18 columns takes 34 us of kernels in 3 launches at 1,000 rows, 41
// at 20,000 and 255 at 1M; as eight launches (clear, Gram matrix, factor and
// solve, twice, with a chunk on one CTA) it took 56, 61 and 268.  Splitting a
// chunk is what shortens it at few rows (a CTA walks 88 to 176 rows, not 1024);
// from 149 chunks on every SM has one and the whole chunk stays on one CTA, with
// no tiles through global memory (with the split's row arithmetic the 1M rows
// took 354 us).
template <int S, int SP, bool kSolve, bool kGram, bool kSplit>
__global__ void __launch_bounds__(kOrthoThreads, 2) ortho_kernel(const OrthoArgs p) {
    using Sh = GramShape<S, SP>;
    constexpr int kVec = SP / 4;
    constexpr int kPf = (Sh::kStage * kVec + kOrthoThreads - 1) / kOrthoThreads;
    constexpr int kReduce = (Sh::G + 1) * Sh::kTile;  // the groups' tiles and their sum
    constexpr int kDoubles = Sh::kStage * SP > kReduce ? Sh::kStage * SP : kReduce;
    static_assert(Sh::kStage <= kOrthoThreads, "a thread solves one row");
    __shared__ __align__(16) float rows_f[kSolve ? Sh::kStage * SP : 4];
    __shared__ __align__(16) double Ls[S * S];
    __shared__ double di[S];
    __shared__ __align__(16) double sm[kGram ? kDoubles : 2];
    __shared__ bool last;
    const Chunk ch = p.chunks[blockIdx.x];
    wait_for_previous();
    const int tid = threadIdx.x;
    const int rows = ch.end - ch.start;
    // Staged rows are whole rounds of the CTA's groups; where a chunk is split,
    // the last round of a slab may run past the slab and is padded with zeros,
    // which change no sum.
    int g0 = 0, groups = Sh::G, local = rows, stage = Sh::R, per_slab = Sh::R;
    if (kSplit) {
        g0 = blockIdx.y * p.groups;
        groups = min(p.groups, Sh::G - g0);
        per_slab = Sh::kRounds * groups;
        local = (rows + Sh::R - 1) / Sh::R * per_slab;
        stage = Sh::kStage / groups * groups;
    }
    // staged row j -> row of the chunk; false for padding
    auto row_of = [&](int j, int* row) {
        *row = j;
        if (!kSplit) return true;
        const int slab = j / per_slab, in = j - slab * per_slab, round = in / groups;
        const int r = round * Sh::G + g0 + in - round * groups;
        *row = slab * Sh::R + r;
        return r < Sh::R && *row < rows;
    };
    float4 pf[kPf];
    const float4* y4 = reinterpret_cast<const float4*>(p.Y + static_cast<int64_t>(ch.start) * SP);
    float4* x4 = reinterpret_cast<float4*>(p.X + static_cast<int64_t>(ch.start) * SP);
    auto prefetch = [&](int j0) {
#pragma unroll
        for (int k = 0; k < kPf; ++k) {
            const int e = tid + k * kOrthoThreads, j = e / kVec;
            int row;
            pf[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (j < stage && j0 + j < local && row_of(j0 + j, &row))
                pf[k] = y4[static_cast<int64_t>(row) * kVec + e - j * kVec];
        }
    };
    prefetch(0);
    if (kSolve) {
        for (int e = tid; e < S * S; e += kOrthoThreads)
            Ls[e] = __ldcg(p.L + static_cast<int64_t>(ch.slot) * S * S + e);
        if (tid < S) di[tid] = __ldcg(p.dinv + static_cast<int64_t>(ch.slot) * S + tid);
    }
    auto widen = [&](int e, const float4& q) {
        reinterpret_cast<double2*>(sm)[2 * e] =
            make_double2(static_cast<double>(q.x), static_cast<double>(q.y));
        reinterpret_cast<double2*>(sm)[2 * e + 1] =
            make_double2(static_cast<double>(q.z), static_cast<double>(q.w));
    };
    GramTile<S, SP> gt;
    if (kGram) gt.init(groups);
    for (int j0 = 0; j0 < local; j0 += stage) {
        const int n = min(stage, local - j0);
        __syncthreads();  // the previous stage is done with
#pragma unroll
        for (int k = 0; k < kPf; ++k) {
            const int e = tid + k * kOrthoThreads;
            if (e >= n * kVec) break;
            if (kSolve) {
                reinterpret_cast<float4*>(rows_f)[e] = pf[k];
            } else {
                widen(e, pf[k]);
            }
        }
        __syncthreads();
        if (j0 + stage < local) prefetch(j0 + stage);
        if (kSolve) {
            if (tid < n) {
                float4* r4 = reinterpret_cast<float4*>(rows_f) + tid * kVec;
                double v[SP];
#pragma unroll
                for (int q = 0; q < kVec; ++q) {
                    const float4 y = r4[q];
                    v[4 * q] = static_cast<double>(y.x);
                    v[4 * q + 1] = static_cast<double>(y.y);
                    v[4 * q + 2] = static_cast<double>(y.z);
                    v[4 * q + 3] = static_cast<double>(y.w);
                }
                // column by column: every entry still gets its terms in order
#pragma unroll
                for (int a = 0; a < S; ++a) {
                    v[a] *= di[a];
#pragma unroll
                    for (int c = a & ~1; c < S; c += 2) {
                        if (c + 1 <= a) continue;
                        const double2 l = *reinterpret_cast<const double2*>(Ls + a * S + c);
                        if (c > a) v[c] = fma(-v[a], l.x, v[c]);
                        v[c + 1] = fma(-v[a], l.y, v[c + 1]);
                    }
                }
#pragma unroll
                for (int q = 0; q < kVec; ++q) {
                    float o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        o[k] = 4 * q + k < S ? static_cast<float>(v[4 * q + k]) : 0.0f;
                    r4[q] = make_float4(o[0], o[1], o[2], o[3]);
                }
            }
            __syncthreads();
            for (int e = tid; e < n * kVec; e += kOrthoThreads) {
                const int j = e / kVec;
                const float4 x = reinterpret_cast<const float4*>(rows_f)[e];
                int row;
                if (row_of(j0 + j, &row)) x4[static_cast<int64_t>(row) * kVec + e - j * kVec] = x;
                if (kGram) widen(e, x);
            }
            if (kGram) __syncthreads();
        }
        if (kGram) gt.add(sm, sm, n, groups);
    }
    if (!kGram) return;
    // true in the last of `of` CTAs to get here; its reads then see their writes
    auto last_of = [&](int* counter, int of) {
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            last = atomicAdd(counter, 1) == of - 1;
            if (last) *counter = 0;
        }
        __syncthreads();
        __threadfence();
        return last;
    };
    // `to` = the sum of `of` tile sets from `from`, in order
    auto sum = [&](const double* from, int of, double* to) {
        for (int o = tid; o < Sh::kTile; o += kOrthoThreads) {
            double v = 0.0;
#pragma unroll 16
            for (int k = 0; k < of; ++k) v += __ldcg(from + static_cast<int64_t>(k) * Sh::kTile + o);
            to[o] = v;
        }
    };
    // the chunk's matrix: its groups in order
    const int64_t chunk = blockIdx.x;
    const int bundles = (ch.of + kBundle - 1) / kBundle;
    const int in_slot = static_cast<int>(chunk) - ch.first, bundle = in_slot / kBundle;
    double* const mat = sm + (kSplit ? 0 : Sh::G * Sh::kTile);
    double* to = ch.of == 1 ? mat : p.sums + chunk * Sh::kTile;
    if (kSplit) {
        double* part = p.part + chunk * Sh::G * Sh::kTile;
        gt.store(part + static_cast<int64_t>(g0) * Sh::kTile);
        if (!last_of(p.chunk_done + chunk, gridDim.y)) return;
        sum(part, Sh::G, to);
    } else {
        __syncthreads();  // the staging buffer becomes the reduction buffer
        gt.store(sm);
        __syncthreads();
        for (int o = tid; o < Sh::kTile; o += kOrthoThreads) {
            double v = 0.0;
#pragma unroll
            for (int g = 0; g < Sh::G; ++g) v += sm[g * Sh::kTile + o];
            to[o] = v;
        }
    }
    if (ch.of > 1) {  // its bundle's chunks in order, then the slot's bundles
        if (!last_of(p.bundle_done + ch.bundle + bundle, min(kBundle, ch.of - bundle * kBundle))) return;
        to = bundles == 1 ? mat : p.bundle + static_cast<int64_t>(ch.bundle + bundle) * Sh::kTile;
        sum(p.sums + static_cast<int64_t>(ch.first + bundle * kBundle) * Sh::kTile,
            min(kBundle, ch.of - bundle * kBundle), to);
        if (bundles > 1) {
            if (!last_of(p.slot_done + ch.slot, bundles)) return;
            sum(p.bundle + static_cast<int64_t>(ch.bundle) * Sh::kTile, bundles, mat);
        }
    }
    __syncthreads();
    for (int o = tid; o < Sh::kTile; o += kOrthoThreads) {
        int row, col;
        if (GramTile<S, SP>::entry(o, &row, &col)) Ls[row * S + col] = mat[o];
    }
    __syncthreads();
    if (tid < 32)
        chol_factor<S>(Ls, p.L + static_cast<int64_t>(ch.slot) * S * S,
                       p.dinv + static_cast<int64_t>(ch.slot) * S, p.fail + ch.slot);
}

// A^T B of every slot (the Ritz step, once a run), added to a cleared G.
template <int S, int SP>
__global__ void __launch_bounds__(kOrthoThreads)
    ritz_gram_kernel(const Chunk* __restrict__ chunks, const float* __restrict__ A,
                     const float* __restrict__ B, double* __restrict__ G) {
    using Sh = GramShape<S, SP>;
    constexpr int kDoubles = 2 * Sh::R * SP > Sh::G * Sh::kTile ? 2 * Sh::R * SP : Sh::G * Sh::kTile;
    static_assert(kDoubles * 8 <= 48 * 1024, "static shared memory");
    __shared__ double sm[kDoubles];
    const Chunk ch = chunks[blockIdx.x];
    GramTile<S, SP> gt;
    gt.init(Sh::G);
    for (int r0 = ch.start; r0 < ch.end; r0 += Sh::R) {
        const int rows = min(Sh::R, ch.end - r0);
        __syncthreads();  // the previous slab is done with
        for (int e = threadIdx.x; e < rows * SP; e += kOrthoThreads) {
            sm[e] = static_cast<double>(A[static_cast<int64_t>(r0) * SP + e]);
            sm[Sh::R * SP + e] = static_cast<double>(B[static_cast<int64_t>(r0) * SP + e]);
        }
        __syncthreads();
        gt.add(sm, sm + Sh::R * SP, rows, Sh::G);
    }
    __syncthreads();
    gt.store(sm);
    __syncthreads();
    for (int o = threadIdx.x; o < Sh::kTile; o += kOrthoThreads) {
        int row, col;
        if (!GramTile<S, SP>::entry(o, &row, &col)) continue;
        double v = 0.0;
        for (int g = 0; g < Sh::G; ++g) v += sm[g * Sh::kTile + o];
        atomicAdd(&G[static_cast<int64_t>(ch.slot) * S * S + row * S + col], v);
    }
}

// coords = X V (V: s x dim per slot), FP64; and per-slot max |coord|.
__global__ void project_kernel(const int32_t* __restrict__ nodes, int64_t cnt,
                               const int32_t* __restrict__ slot_of_pos,
                               const double* __restrict__ V, int s, int sp, int dim,
                               const float* __restrict__ X, float* __restrict__ out,
                               unsigned* __restrict__ max_abs_bits) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cnt) return;
    const int64_t i = nodes[t];
    const int slot = slot_of_pos[t];
    const double* v = V + static_cast<int64_t>(slot) * s * dim;
    float mx = 0.0f;
    for (int oc = 0; oc < dim; ++oc) {
        double acc = 0.0;
        for (int b = 0; b < s; ++b) acc += static_cast<double>(X[t * sp + b]) * v[b * dim + oc];
        const float f = static_cast<float>(acc);
        out[i * dim + oc] = f;
        mx = fmaxf(mx, fabsf(f));
    }
    atomicMax(&max_abs_bits[slot], __float_as_uint(mx));
}

// coord = coord * expansion + N(0, noise) + anchor (noisy_scale_coords,
// lib.rs:4766-4791, and the per-component placement of lib.rs:4713-4752).
__global__ void finish_kernel(const int32_t* __restrict__ nodes, int64_t cnt,
                              const int32_t* __restrict__ slot_of_node,
                              const float* __restrict__ expansion,
                              const float* __restrict__ anchors, const uint64_t* __restrict__ nseed,
                              int dim, float noise, float* __restrict__ out) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cnt) return;
    const int64_t i = nodes[t];
    const int slot = slot_of_node[t];
    for (int c = 0; c < dim; ++c) {
        const uint64_t w1 = rng_word(nseed[slot], static_cast<uint64_t>(i), 2 * c);
        const uint64_t w2 = rng_word(nseed[slot], static_cast<uint64_t>(i), 2 * c + 1);
        double u1 = rng_unit_f64(w1);
        if (u1 < 1e-300) u1 = 1e-300;
        const double z = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * rng_unit_f64(w2));
        const float v = out[i * dim + c] * expansion[slot] + static_cast<float>(noise * z);
        out[i * dim + c] = v + anchors[slot * dim + c];
    }
}

__global__ void random_init_kernel(int64_t n, int dim, uint64_t seed, float low, float high,
                                   float* out) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * dim) return;
    const float u = rng_unit_f32(rng_word(seed, static_cast<uint64_t>(t / dim), t % dim));
    out[t] = low + u * (high - low);
}

__global__ void scatter_rows_kernel(const int32_t* __restrict__ nodes, int64_t cnt, int dim,
                                    const float* __restrict__ vals, float* __restrict__ out) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cnt * dim) return;
    out[static_cast<int64_t>(nodes[t / dim]) * dim + t % dim] = vals[t];
}

// Centroid sums per component (FP64) over the component-sorted node list, a
// chunk of rows and 64 features a CTA.  Bound by the latency of row loads:
// sixteen groups of rows with eight loads in flight each, added in order,
// take 20 us for ten components of 2,000 x 192; one thread a feature that
// walked a whole chunk took 690.
constexpr int kCentroidFeatures = 64;
constexpr int kCentroidGroups = 16;
__global__ void __launch_bounds__(kCentroidFeatures* kCentroidGroups)
    centroid_kernel(const Chunk* __restrict__ chunks, const int32_t* __restrict__ nodes,
                    const float* __restrict__ X, int d, int f_tiles, double* __restrict__ cent) {
    __shared__ double part[kCentroidGroups][kCentroidFeatures];
    const Chunk ch = chunks[blockIdx.x / f_tiles];
    const int lf = threadIdx.x % kCentroidFeatures, g = threadIdx.x / kCentroidFeatures;
    const int f = static_cast<int>(blockIdx.x % f_tiles) * kCentroidFeatures + lf;
    double acc = 0.0;
    if (f < d) {
#pragma unroll 8
        for (int r = ch.start + g; r < ch.end; r += kCentroidGroups)
            acc += static_cast<double>(__ldg(X + static_cast<int64_t>(__ldg(nodes + r)) * d + f));
    }
    part[g][lf] = acc;
    __syncthreads();
    if (g != 0 || f >= d) return;
    acc = 0.0;
#pragma unroll
    for (int k = 0; k < kCentroidGroups; ++k) acc += part[k][lf];
    atomicAdd(&cent[static_cast<int64_t>(ch.slot) * d + f], acc);
}

// the same sums from CSR rows (component_centroids_sparse, lib.rs:4487-4505)
__global__ void centroid_csr_kernel(const Chunk* __restrict__ chunks,
                                    const int32_t* __restrict__ nodes,
                                    const int64_t* __restrict__ indptr,
                                    const int32_t* __restrict__ indices,
                                    const float* __restrict__ values, int d,
                                    double* __restrict__ cent) {
    const Chunk ch = chunks[blockIdx.x];
    for (int r = ch.start + static_cast<int>(threadIdx.x); r < ch.end; r += blockDim.x) {
        const int64_t v = nodes[r];
        for (int64_t e = indptr[v]; e < indptr[v + 1]; ++e)
            atomicAdd(&cent[static_cast<int64_t>(ch.slot) * d + indices[e]],
                      static_cast<double>(values[e]));
    }
}

// ------------------------------------------------------------ host side --
using HostCoords = std::vector<float>;  // row-major n x dim

bool finite_all(const std::vector<float>& v) {
    for (float x : v)
        if (!std::isfinite(x)) return false;
    return true;
}

// normalized_laplacian_from_edges + spectral_embedding_from_laplacian
// (lib.rs:4007-4069, 3917-3957) for a small component given its local edges.
bool dense_spectral(int64_t n, int dim, const std::vector<std::array<int64_t, 2>>& pairs,
                    const std::vector<float>& w, HostCoords& out) {
    if (n <= dim + 1 || pairs.empty()) return false;
    std::vector<double> L(n * n, 0.0), deg(n, 0.0);
    for (int64_t i = 0; i < n; ++i) L[i * n + i] = 1.0;
    std::vector<std::pair<int64_t, int64_t>> und;
    for (size_t e = 0; e < pairs.size(); ++e) {
        const int64_t h = pairs[e][0], t = pairs[e][1];
        if (h == t) continue;
        const double wv = static_cast<double>(std::max(w[e], 0.0f));
        if (wv <= 0.0) continue;
        const int64_t i = std::min(h, t), j = std::max(h, t);
        const double prev = L[i * n + j];
        if (wv > prev) {
            if (prev == 0.0) und.emplace_back(i, j);
            const double delta = wv - prev;
            L[i * n + j] = wv;
            L[j * n + i] = wv;
            deg[i] += delta;
            deg[j] += delta;
        }
    }
    bool any = false;
    for (double v : deg) any |= v > 0.0;
    if (!any) return false;
    std::vector<double> inv(n);
    for (int64_t i = 0; i < n; ++i) inv[i] = deg[i] > 0 ? 1.0 / std::sqrt(deg[i]) : 0.0;
    for (auto [i, j] : und) {
        const double v = L[i * n + j] * inv[i] * inv[j];
        L[i * n + j] = -v;
        L[j * n + i] = -v;
    }
    for (int64_t i = 0; i < n; ++i) L[i * n + i] = 1.0;
    std::vector<double> ev, V;
    symmetric_eigen(L, static_cast<int>(n), ev, V);
    if (n <= dim + 1) return false;
    out.assign(n * dim, 0.0f);
    for (int c = 0; c < dim; ++c)
        for (int64_t r = 0; r < n; ++r) out[r * dim + c] = static_cast<float>(V[r * n + c + 1]);
    return finite_all(out);
}

void host_random(int64_t n, int dim, uint64_t seed, float low, float high, HostCoords& out) {
    out.resize(n * dim);
    for (int64_t t = 0; t < n * dim; ++t) {
        const float u = rng_unit_f32(rng_word(seed, static_cast<uint64_t>(t / dim), t % dim));
        out[t] = low + u * (high - low);
    }
}

double host_normal(uint64_t seed, uint64_t a, uint64_t b) {
    double u1 = rng_unit_f64(rng_word(seed, a, 2 * b));
    if (u1 < 1e-300) u1 = 1e-300;
    return std::sqrt(-2.0 * std::log(u1)) *
           std::cos(6.283185307179586 * rng_unit_f64(rng_word(seed, a, 2 * b + 1)));
}

// meta_component_layout_from_centroids (lib.rs:4519-4554)
bool meta_layout(const std::vector<double>& cents, int64_t m, int d, int dim, uint64_t seed,
                 HostCoords& out) {
    if (m == 0) return false;
    if (m == 1) {
        out.assign(dim, 0.0f);
        return true;
    }
    if (m <= 2 * dim) {
        const int64_t k = (m + 1) / 2;
        out.assign(m * dim, 0.0f);
        for (int64_t i = 0; i < m; ++i) out[i * dim + (i % k)] = i < k ? 1.0f : -1.0f;
        return true;
    }
    std::vector<double> aff(m * m, 0.0), deg(m, 0.0);
    for (int64_t i = 0; i < m; ++i) {
        aff[i * m + i] = 1.0;
        for (int64_t j = i + 1; j < m; ++j) {
            double d2 = 0.0;
            for (int f = 0; f < d; ++f) {
                const double dd = cents[i * d + f] - cents[j * d + f];
                d2 += dd * dd;
            }
            const double wv = std::exp(-d2);
            aff[i * m + j] = wv;
            aff[j * m + i] = wv;
        }
    }
    for (int64_t i = 0; i < m; ++i)
        for (int64_t j = 0; j < m; ++j) deg[i] += aff[i * m + j];
    std::vector<double> inv(m), L(m * m, 0.0);
    for (int64_t i = 0; i < m; ++i) inv[i] = deg[i] > 0 ? 1.0 / std::sqrt(deg[i]) : 0.0;
    for (int64_t i = 0; i < m; ++i) L[i * m + i] = 1.0;
    for (int64_t i = 0; i < m; ++i) {
        if (deg[i] <= 0) continue;
        for (int64_t j = 0; j < m; ++j) {
            if (deg[j] <= 0) continue;
            if (aff[i * m + j] > 0.0) L[i * m + j] -= aff[i * m + j] * inv[i] * inv[j];
        }
    }
    std::vector<double> ev, V;
    symmetric_eigen(L, static_cast<int>(m), ev, V);
    if (m <= dim + 1) return false;
    out.assign(m * dim, 0.0f);
    for (int c = 0; c < dim; ++c)
        for (int64_t r = 0; r < m; ++r) out[r * dim + c] = static_cast<float>(V[r * m + c + 1]);
    // noisy_scale_coords(seed ^ 0xC85E7D6ADA318F21, 10, 1e-4)
    float mx = 0.0f;
    for (float v : out) mx = std::max(mx, std::fabs(v));
    const float expansion = mx > 0.0f ? kInitMaxCoord / mx : 1.0f;
    const uint64_t ns = seed ^ 0xC85E7D6ADA318F21ULL;
    for (int64_t r = 0; r < m; ++r)
        for (int c = 0; c < dim; ++c)
            out[r * dim + c] = out[r * dim + c] * expansion +
                               static_cast<float>(kInitNoise * host_normal(ns, r, c));
    return finite_all(out);
}

// Block subspace iteration for every iterative component at once; writes
// the scaled, noised and anchored coordinates of their nodes into `out`.
// Returns false where the reference would return None (an orthonormalisation
// failure or a non-finite result).
template <int S, int SP>
bool run_iterative(const std::vector<int64_t>& it_comps, const std::vector<int64_t>& cstart,
                   const std::vector<int32_t>& order_h, const std::vector<uint64_t>& cseed,
                   const std::vector<float>& data_range, const std::vector<float>& anchors,
                   bool multi, uint64_t seed, int dim, int64_t n, const Graph& g, float* out,
                   cudaStream_t s) {
    const int64_t m = g.n_edges;
    const int64_t n_slots = static_cast<int64_t>(it_comps.size());
    std::vector<int32_t> nodes_h, slot_h;
    std::vector<int32_t> slot_end;
    std::vector<Chunk> chunks;
    std::vector<uint64_t> slot_seed(n_slots), noise_seed(n_slots);
    std::vector<float> expand_target(n_slots), slot_anchor(n_slots * dim);
    for (int64_t sl = 0; sl < n_slots; ++sl) {
        const int64_t c = it_comps[sl];
        const int32_t base = static_cast<int32_t>(nodes_h.size());
        for (int64_t q = cstart[c]; q < cstart[c + 1]; ++q) {
            nodes_h.push_back(order_h[q]);
            slot_h.push_back(static_cast<int32_t>(sl));
        }
        const int32_t end = static_cast<int32_t>(nodes_h.size());
        slot_end.push_back(end);
        slot_seed[sl] = cseed[c];
        noise_seed[sl] = multi ? seed ^ (static_cast<uint64_t>(c + 1) * 0x94D049BBULL)
                               : seed ^ 0x5DEECE66DULL;
        expand_target[sl] = multi ? data_range[c] : kInitMaxCoord;
        for (int k = 0; k < dim; ++k) slot_anchor[sl * dim + k] = multi ? anchors[c * dim + k] : 0.0f;
    }
    const int64_t cnt = static_cast<int64_t>(nodes_h.size());
    // Chunks of 1024 rows, of more where that would make over two an SM (a
    // slot's last CTA adds its chunks' matrices one after the other).
    constexpr int64_t kOrthoCtas = 2 * 148;
    int32_t n_bundles = 0;
    const int32_t per_chunk =
        static_cast<int32_t>(std::max<int64_t>(1024, ceil_div(ceil_div(cnt, kOrthoCtas), 128) * 128));
    for (int64_t sl = 0; sl < n_slots; ++sl) {
        const int32_t base = sl ? slot_end[sl - 1] : 0, end = slot_end[sl];
        const int32_t of = static_cast<int32_t>(ceil_div(end - base, per_chunk));
        const int32_t first = static_cast<int32_t>(chunks.size());
        for (int32_t st = base; st < end; st += per_chunk)
            chunks.push_back({static_cast<int32_t>(sl), st, std::min(end, st + per_chunk), first, of,
                              n_bundles});
        n_bundles += static_cast<int32_t>(ceil_div(of, kBundle));
    }
    DevBuf<int32_t> nodes(cnt, s), slots(cnt, s), pos(n, s), plen(cnt, s), quads(cnt + 1, s),
        qptr(cnt + 1, s), long_rows(cnt, s), n_long(1, s);
    DevBuf<Chunk> dch(chunks.size(), s);
    DevBuf<uint64_t> dseed(n_slots, s), dnseed(n_slots, s);
    UMAPB_CUDA(cudaMemcpyAsync(nodes.get(), nodes_h.data(), cnt * 4, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(slots.get(), slot_h.data(), cnt * 4, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(dch.get(), chunks.data(), chunks.size() * sizeof(Chunk),
                               cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(dseed.get(), slot_seed.data(), n_slots * 8, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(dnseed.get(), noise_seed.data(), n_slots * 8, cudaMemcpyHostToDevice, s));

    // degrees and normalised weights in node space
    DevBuf<double> deg(n, s);
    DevBuf<float> dinvn(n, s), nw(std::max<int64_t>(m, 1), s);
    degree_kernel<<<grid_for(n), 256, 0, s>>>(g.row_ptr.get(), g.weights.get(), n, deg.get(),
                                              dinvn.get());
    UMAPB_LAUNCH_CHECK();
    norm_weight_kernel<<<grid_for(m), 256, 0, s>>>(g.heads.get(), g.tails.get(), g.weights.get(),
                                                   deg.get(), m, nw.get());
    UMAPB_LAUNCH_CHECK();
    // position-ordered CSR
    pos_kernel<<<grid_for(cnt), 256, 0, s>>>(nodes.get(), cnt, pos.get());
    UMAPB_LAUNCH_CHECK();
    const int32_t long_row = static_cast<int32_t>(
        std::max<int64_t>(kLongRowMin, std::min<int64_t>(kLongRowMax, m / kEdgesPerLongEdge)));
    UMAPB_CUDA(cudaMemsetAsync(n_long.get(), 0, 4, s));
    UMAPB_CUDA(cudaMemsetAsync(quads.get() + cnt, 0, 4, s));
    prow_len_kernel<<<grid_for(cnt), 256, 0, s>>>(nodes.get(), cnt, g.row_ptr.get(), plen.get(),
                                                  quads.get(), long_row, long_rows.get(),
                                                  n_long.get());
    UMAPB_LAUNCH_CHECK();
    {
        size_t tb = 0;
        UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, quads.get(), qptr.get(), cnt + 1, s));
        DevBuf<unsigned char> tmp(tb, s);
        UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tb, quads.get(), qptr.get(), cnt + 1, s));
    }
    int32_t n_quads = 0, n_long_h = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&n_quads, qptr.get() + cnt, 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(&n_long_h, n_long.get(), 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    const int64_t m_it = static_cast<int64_t>(n_quads) * 4;
    DevBuf<int32_t> ptails(std::max<int64_t>(m_it, 4), s);
    DevBuf<float> pnw(std::max<int64_t>(m_it, 4), s);
    pcsr_kernel<<<grid_for(cnt), 256, 0, s>>>(nodes.get(), cnt, g.row_ptr.get(), g.tails.get(),
                                              nw.get(), pos.get(), qptr.get(), ptails.get(), pnw.get());
    UMAPB_LAUNCH_CHECK();

    DevBuf<float> Xb(cnt * SP, s), Yb(cnt * SP, s);
    using Sh = GramShape<S, SP>;
    const unsigned nch = static_cast<unsigned>(chunks.size());
    const unsigned gr = grid_for(cnt);
    // few chunks: a chunk's row groups on as many CTAs as keep two an SM
    const int split = static_cast<int>(
        std::max<int64_t>(1, std::min<int64_t>(Sh::G, kOrthoCtas / static_cast<int64_t>(nch))));
    const int groups = static_cast<int>(ceil_div(Sh::G, split));
    const dim3 ortho_grid(nch, static_cast<unsigned>(ceil_div(Sh::G, groups)));
    DevBuf<double> G(n_slots * S * S, s), L(n_slots * S * S, s), dinv(n_slots * S, s),
        sums(static_cast<int64_t>(nch) * Sh::kTile, s),
        bundle_sums(static_cast<int64_t>(n_bundles) * Sh::kTile, s),
        part(ortho_grid.y > 1 ? static_cast<int64_t>(nch) * Sh::G * Sh::kTile : 1, s);
    DevBuf<int> fail(n_slots, s), chunk_done(nch, s), bundle_done(n_bundles, s), slot_done(n_slots, s);
    UMAPB_CUDA(cudaMemsetAsync(fail.get(), 0, n_slots * 4, s));
    UMAPB_CUDA(cudaMemsetAsync(chunk_done.get(), 0, nch * 4, s));
    UMAPB_CUDA(cudaMemsetAsync(bundle_done.get(), 0, n_bundles * 4, s));
    UMAPB_CUDA(cudaMemsetAsync(slot_done.get(), 0, n_slots * 4, s));
    init_block_kernel<<<grid_for(cnt), 256, 0, s>>>(nodes.get(), cnt, slots.get(), dseed.get(),
                                                    deg.get(), S, SP, Xb.get());
    UMAPB_LAUNCH_CHECK();
    const bool early = cnt <= kEarlyRows;
    // CholQR2: src -> dst -> src; the orthonormal block ends in src
    auto cholqr = [&](float* src, float* dst) {
        OrthoArgs oa{dch.get(),          src,        nullptr,           L.get(),
                     dinv.get(),         part.get(), sums.get(),        bundle_sums.get(),
                     chunk_done.get(),   bundle_done.get(), slot_done.get(), fail.get(), groups};
        auto pass = [&](auto kernel, auto split_kernel, const float* y, float* x) {
            oa.Y = y;
            oa.X = x;
            launch_chained(ortho_grid.y > 1 ? split_kernel : kernel, early, ortho_grid, kOrthoThreads,
                           s, oa);
        };
        pass(ortho_kernel<S, SP, false, true, false>, ortho_kernel<S, SP, false, true, true>, src,
             nullptr);
        pass(ortho_kernel<S, SP, true, true, false>, ortho_kernel<S, SP, true, true, true>, src, dst);
        pass(ortho_kernel<S, SP, true, false, false>, ortho_kernel<S, SP, true, false, true>, dst, src);
    };
    const unsigned gr_spmm = static_cast<unsigned>(
        n_long_h + ceil_div(cnt, static_cast<int64_t>(spmm_rows_per_block<SP>())));
    auto spmm = [&](const float* x, float* y) {
        launch_chained(spmm_kernel<SP>, early, dim3(gr_spmm), kSpmmThreads, s, cnt, qptr.get(),
                       plen.get(), ptails.get(), pnw.get(), long_rows.get(), n_long_h, long_row, x,
                       y);
    };
    static_assert(kIters % kOrthoEvery == 0, "the last product must be orthonormalised");
    cholqr(Xb.get(), Yb.get());
    for (int it = 0; it < kIters; ++it) {
        spmm(Xb.get(), Yb.get());  // Y = (I + A) X
        std::swap(Xb, Yb);
        if ((it + 1) % kOrthoEvery == 0) cholqr(Xb.get(), Yb.get());  // orthonormal in X
    }
    spmm(Xb.get(), Yb.get());
    UMAPB_CUDA(cudaMemsetAsync(G.get(), 0, n_slots * S * S * 8, s));
    ritz_gram_kernel<S, SP><<<nch, kOrthoThreads, 0, s>>>(dch.get(), Xb.get(), Yb.get(), G.get());
    UMAPB_LAUNCH_CHECK();
    std::vector<double> G_h(n_slots * S * S);
    std::vector<int> fail_h(n_slots);
    UMAPB_CUDA(cudaMemcpyAsync(G_h.data(), G.get(), G_h.size() * 8, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(fail_h.data(), fail.get(), n_slots * 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    for (int64_t sl = 0; sl < n_slots; ++sl)
        if (fail_h[sl]) return false;  // orthonormalize_columns failed (lib.rs:4262-4273)
    // Rayleigh-Ritz: eigenvectors by descending eigenvalue, skipping the first
    std::vector<double> Vsel(n_slots * S * dim);
    for (int64_t sl = 0; sl < n_slots; ++sl) {
        std::vector<double> R(S * S);
        const double* gs = G_h.data() + sl * S * S;
        for (int i = 0; i < S; ++i)
            for (int j = i; j < S; ++j) {
                R[i * S + j] = gs[i * S + j];
                R[j * S + i] = gs[i * S + j];
            }
        std::vector<double> ev, V;
        symmetric_eigen(R, S, ev, V);
        std::vector<int> ord(S);
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return ev[a] > ev[b]; });
        for (int oc = 0; oc < dim; ++oc)
            for (int b = 0; b < S; ++b) Vsel[(sl * S + b) * dim + oc] = V[b * S + ord[oc + 1]];
    }
    DevBuf<double> dV(Vsel.size(), s);
    DevBuf<unsigned> maxbits(n_slots, s);
    UMAPB_CUDA(cudaMemcpyAsync(dV.get(), Vsel.data(), Vsel.size() * 8, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemsetAsync(maxbits.get(), 0, n_slots * 4, s));
    project_kernel<<<gr, 256, 0, s>>>(nodes.get(), cnt, slots.get(), dV.get(), S, SP, dim, Xb.get(),
                                      out, maxbits.get());
    UMAPB_LAUNCH_CHECK();
    std::vector<unsigned> mb(n_slots);
    UMAPB_CUDA(cudaMemcpyAsync(mb.data(), maxbits.get(), n_slots * 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    std::vector<float> expansion(n_slots);
    for (int64_t sl = 0; sl < n_slots; ++sl) {
        float mx;
        std::memcpy(&mx, &mb[sl], 4);
        if (!std::isfinite(mx)) return false;
        expansion[sl] = mx > 0.0f ? expand_target[sl] / mx : 1.0f;
    }
    DevBuf<float> dexp(n_slots, s), danch(n_slots * dim, s);
    UMAPB_CUDA(cudaMemcpyAsync(dexp.get(), expansion.data(), n_slots * 4, cudaMemcpyHostToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(danch.get(), slot_anchor.data(), n_slots * dim * 4,
                               cudaMemcpyHostToDevice, s));
    finish_kernel<<<gr, 256, 0, s>>>(nodes.get(), cnt, slots.get(), dexp.get(), danch.get(),
                                     dnseed.get(), dim, kInitNoise, out);
    UMAPB_LAUNCH_CHECK();
    UMAPB_CUDA(cudaStreamSynchronize(s));
    return true;
}

}  // namespace

void random_init(int64_t n, int dim, uint64_t seed, float low, float high, float* out,
                 cudaStream_t s) {
    if (n == 0) return;
    random_init_kernel<<<grid_for(n * dim), 256, 0, s>>>(n, dim, seed, low, high, out);
    UMAPB_LAUNCH_CHECK();
}

SpectralResult spectral_init(const float* X, int64_t n, int d, const Graph& g, int dim,
                             uint64_t seed, float* out, cudaStream_t s, const CsrDevice* csr) {
    SpectralResult res;
    const int64_t m = g.n_edges;
    if (n <= dim + 1 || m == 0) return res;
    const int sdim = std::max((dim + 1) * kOversampling, dim + 1);
    if (sdim > kMaxS) invalid("spectral init supports n_components <= 4 on the GPU path");

    // ---- connected components (union-find with atomicMin hooking)
    DevBuf<int32_t> parent(n, s);
    cc_init<<<grid_for(n), 256, 0, s>>>(parent.get(), n);
    UMAPB_LAUNCH_CHECK();
    DevBuf<int> changed(1, s);
    for (int round = 0; round < 64; ++round) {
        UMAPB_CUDA(cudaMemsetAsync(changed.get(), 0, 4, s));
        cc_hook<<<grid_for(m), 256, 0, s>>>(g.heads.get(), g.tails.get(), m, parent.get(),
                                            changed.get());
        UMAPB_LAUNCH_CHECK();
        cc_compress<<<grid_for(n), 256, 0, s>>>(parent.get(), n);
        UMAPB_LAUNCH_CHECK();
        int h = 0;
        UMAPB_CUDA(cudaMemcpyAsync(&h, changed.get(), 4, cudaMemcpyDeviceToHost, s));
        UMAPB_CUDA(cudaStreamSynchronize(s));
        if (!h) break;
    }
    DevBuf<int32_t> isroot(n, s), rank(n, s), label(n, s), order(n, s), lab_sorted(n, s),
        iota(n, s);
    cc_is_root<<<grid_for(n), 256, 0, s>>>(parent.get(), n, isroot.get());
    UMAPB_LAUNCH_CHECK();
    {
        size_t tb = 0;
        UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, isroot.get(), rank.get(), n, s));
        DevBuf<unsigned char> tmp(tb, s);
        UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tb, isroot.get(), rank.get(), n, s));
    }
    int32_t last_rank = 0, last_root = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&last_rank, rank.get() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(&last_root, isroot.get() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    const int64_t n_comp = static_cast<int64_t>(last_rank) + last_root;
    res.n_components = n_comp;
    cc_label<<<grid_for(n), 256, 0, s>>>(parent.get(), rank.get(), n, label.get());
    UMAPB_LAUNCH_CHECK();
    iota_kernel<<<grid_for(n), 256, 0, s>>>(iota.get(), n);
    UMAPB_LAUNCH_CHECK();
    {
        int bits = 1;
        while ((int64_t(1) << bits) < n_comp + 1) ++bits;
        size_t tb = 0;
        UMAPB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, label.get(), lab_sorted.get(),
                                                   iota.get(), order.get(), n, 0, bits, s));
        DevBuf<unsigned char> tmp(tb, s);
        UMAPB_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), tb, label.get(), lab_sorted.get(),
                                                   iota.get(), order.get(), n, 0, bits, s));
    }
    // component sizes on the host from the sorted labels
    std::vector<int32_t> lab_h(n), order_h;
    UMAPB_CUDA(cudaMemcpyAsync(lab_h.data(), lab_sorted.get(), n * 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));
    std::vector<int64_t> cstart(n_comp + 1, 0);
    for (int64_t i = 0; i < n; ++i) cstart[lab_h[i] + 1]++;
    for (int64_t c = 0; c < n_comp; ++c) cstart[c + 1] += cstart[c];

    // ---- decide the path of every component
    enum Kind { kIter, kDense, kRandom };
    std::vector<Kind> kind(n_comp);
    std::vector<uint64_t> cseed(n_comp);
    const bool multi = n_comp > 1;
    for (int64_t c = 0; c < n_comp; ++c) {
        const int64_t sz = cstart[c + 1] - cstart[c];
        if (!multi) {
            const int64_t thr = d <= 8 ? 2049 : 0;  // spectral_iterative_connected_threshold
            kind[c] = (sz >= thr && sz > sdim) ? kIter : kDense;
            cseed[c] = seed;
        } else {
            if (sz < 2 * dim || sz <= dim + 1)
                kind[c] = kRandom;
            else
                kind[c] = (sz >= kComponentIterThreshold && sz > sdim) ? kIter : kDense;
            cseed[c] = seed ^ (static_cast<uint64_t>(c + 1) * 0xBF58476D1CE4E5B9ULL);
        }
    }
    if (!multi && kind[0] == kDense && n > kDenseFallbackMax && n >= (d <= 8 ? 2049 : 0))
        return res;

    // ---- meta layout (anchors) and per-component ranges
    std::vector<float> anchors(n_comp * dim, 0.0f), data_range(n_comp, 1.0f);
    if (multi) {
        std::vector<double> cents;
        if (n_comp > 2 * dim) {
            std::vector<Chunk> chunks;
            for (int64_t c = 0; c < n_comp; ++c)
                for (int64_t st = cstart[c]; st < cstart[c + 1]; st += 4096)
                    chunks.push_back({static_cast<int32_t>(c), static_cast<int32_t>(st),
                                      static_cast<int32_t>(std::min(cstart[c + 1], st + 4096))});
            DevBuf<Chunk> dch(chunks.size(), s);
            DevBuf<double> dcent(n_comp * d, s);
            UMAPB_CUDA(cudaMemcpyAsync(dch.get(), chunks.data(), chunks.size() * sizeof(Chunk),
                                       cudaMemcpyHostToDevice, s));
            UMAPB_CUDA(cudaMemsetAsync(dcent.get(), 0, n_comp * d * 8, s));
            const int f_tiles = static_cast<int>(ceil_div(d, kCentroidFeatures));
            if (csr)
                centroid_csr_kernel<<<static_cast<unsigned>(chunks.size()), 128, 0, s>>>(
                    dch.get(), order.get(), csr->indptr.get(), csr->indices.get(),
                    csr->values.get(), d, dcent.get());
            else
                centroid_kernel<<<static_cast<unsigned>(chunks.size() * f_tiles),
                                  kCentroidFeatures * kCentroidGroups, 0, s>>>(
                    dch.get(), order.get(), X, d, f_tiles, dcent.get());
            UMAPB_LAUNCH_CHECK();
            cents.resize(n_comp * d);
            UMAPB_CUDA(cudaMemcpyAsync(cents.data(), dcent.get(), n_comp * d * 8,
                                       cudaMemcpyDeviceToHost, s));
            UMAPB_CUDA(cudaStreamSynchronize(s));
            for (int64_t c = 0; c < n_comp; ++c) {
                const double sc = 1.0 / static_cast<double>(cstart[c + 1] - cstart[c]);
                for (int f = 0; f < d; ++f) cents[c * d + f] *= sc;
            }
        }
        HostCoords layout;
        if (!meta_layout(cents, n_comp, d, dim, seed ^ 0xA13F52A92D4CB801ULL, layout)) return res;
        anchors = layout;
        for (int64_t c = 0; c < n_comp; ++c) {
            float r = INFINITY;
            for (int64_t o = 0; o < n_comp; ++o) {
                if (o == c) continue;
                float d2 = 0.0f;
                for (int k = 0; k < dim; ++k) {
                    const float df = anchors[c * dim + k] - anchors[o * dim + k];
                    d2 += df * df;
                }
                const float dist = std::sqrt(d2);
                if (dist > 0.0f) r = std::min(r, dist / 2.0f);
            }
            if (!std::isfinite(r) || r <= 0.0f) r = 1.0f;
            data_range[c] = r;
        }
    }

    // ---- host components (dense spectral / random)
    bool need_host_graph = false;
    for (int64_t c = 0; c < n_comp; ++c) need_host_graph |= kind[c] == kDense;
    std::vector<int32_t> rp_h, tl_h;
    std::vector<float> w_h;
    if (need_host_graph) {
        rp_h.resize(n + 1);
        tl_h.resize(m);
        w_h.resize(m);
        order_h.resize(n);
        UMAPB_CUDA(cudaMemcpyAsync(rp_h.data(), g.row_ptr.get(), (n + 1) * 4, cudaMemcpyDeviceToHost, s));
        UMAPB_CUDA(cudaMemcpyAsync(tl_h.data(), g.tails.get(), m * 4, cudaMemcpyDeviceToHost, s));
        UMAPB_CUDA(cudaMemcpyAsync(w_h.data(), g.weights.get(), m * 4, cudaMemcpyDeviceToHost, s));
    }
    if (order_h.empty()) order_h.resize(n);
    UMAPB_CUDA(cudaMemcpyAsync(order_h.data(), order.get(), n * 4, cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaStreamSynchronize(s));

    std::vector<int32_t> host_nodes;
    std::vector<float> host_vals;
    std::vector<int64_t> local_of(need_host_graph ? n : 0, -1);
    for (int64_t c = 0; c < n_comp; ++c) {
        if (kind[c] == kIter) continue;
        const int64_t sz = cstart[c + 1] - cstart[c];
        HostCoords local;
        if (kind[c] == kRandom) {
            host_random(sz, dim, seed ^ (static_cast<uint64_t>(c + 1) * 0x9E3779B9ULL),
                        -data_range[c], data_range[c], local);
        } else {
            for (int64_t li = 0; li < sz; ++li) local_of[order_h[cstart[c] + li]] = li;
            std::vector<std::array<int64_t, 2>> pairs;
            std::vector<float> pw;
            for (int64_t li = 0; li < sz; ++li) {
                const int64_t node = order_h[cstart[c] + li];
                for (int32_t e = rp_h[node]; e < rp_h[node + 1]; ++e) {
                    pairs.push_back({li, local_of[tl_h[e]]});
                    pw.push_back(w_h[e]);
                }
            }
            if (!dense_spectral(sz, dim, pairs, pw, local)) return res;
            float mx = 0.0f;
            for (float v : local) mx = std::max(mx, std::fabs(v));
            const float target = multi ? data_range[c] : kInitMaxCoord;
            const float expansion = mx > 0.0f ? target / mx : 1.0f;
            const uint64_t ns = multi ? seed ^ (static_cast<uint64_t>(c + 1) * 0x94D049BBULL)
                                      : seed ^ 0x5DEECE66DULL;
            for (int64_t li = 0; li < sz; ++li)
                for (int k = 0; k < dim; ++k)
                    local[li * dim + k] = local[li * dim + k] * expansion +
                                          static_cast<float>(kInitNoise * host_normal(ns, li, k));
        }
        for (int64_t li = 0; li < sz; ++li) {
            host_nodes.push_back(order_h[cstart[c] + li]);
            for (int k = 0; k < dim; ++k)
                host_vals.push_back(local[li * dim + k] + (multi ? anchors[c * dim + k] : 0.0f));
        }
    }
    if (!host_nodes.empty()) {
        const int64_t cnt = static_cast<int64_t>(host_nodes.size());
        DevBuf<int32_t> hn(cnt, s);
        DevBuf<float> hv(cnt * dim, s);
        UMAPB_CUDA(cudaMemcpyAsync(hn.get(), host_nodes.data(), cnt * 4, cudaMemcpyHostToDevice, s));
        UMAPB_CUDA(cudaMemcpyAsync(hv.get(), host_vals.data(), cnt * dim * 4, cudaMemcpyHostToDevice, s));
        scatter_rows_kernel<<<grid_for(cnt * dim), 256, 0, s>>>(hn.get(), cnt, dim, hv.get(), out);
        UMAPB_LAUNCH_CHECK();
        UMAPB_CUDA(cudaStreamSynchronize(s));
    }

    // ---- iterative components on the device
    std::vector<int64_t> it_comps;
    for (int64_t c = 0; c < n_comp; ++c)
        if (kind[c] == kIter) it_comps.push_back(c);
    if (!it_comps.empty()) {
        bool ok = false;
        switch (sdim) {
            case 12: ok = run_iterative<12, 12>(it_comps, cstart, order_h, cseed, data_range, anchors,
                                               multi, seed, dim, n, g, out, s); break;
            case 18: ok = run_iterative<18, 20>(it_comps, cstart, order_h, cseed, data_range, anchors,
                                               multi, seed, dim, n, g, out, s); break;
            case 24: ok = run_iterative<24, 24>(it_comps, cstart, order_h, cseed, data_range, anchors,
                                               multi, seed, dim, n, g, out, s); break;
            case 30: ok = run_iterative<30, 32>(it_comps, cstart, order_h, cseed, data_range, anchors,
                                               multi, seed, dim, n, g, out, s); break;
            default: invalid("unsupported spectral block width");
        }
        if (!ok) return res;
    }
    res.used_spectral = true;
    return res;
}

}  // namespace umapb
