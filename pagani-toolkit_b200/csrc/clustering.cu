// clustering.cu -- clustering coefficients.
//   binary: Cp (U/Cp/Cp/Cp.cpp:21-116) from exact per-node triangle counts;
//   Onnela: Cp_2 (W/Cp/Cp/Cp_2.cpp:23-130).
//
// One CTA per node u (grid-stride).  The neighbour set of u is marked in a
// shared-memory bitmap of the node range (n bits), so every membership test
// of a neighbour's neighbour is one shared-memory load; the neighbour lists
// themselves are read coalesced, one warp per neighbour.  Binary counting
// only visits neighbours v > u and credits the pair count to both u and v,
// which halves the work (each triangle is then counted twice at each of its
// three nodes).
#include "pg_internal.cuh"
#include "clustering.cuh"
#include <cuda.h>
#include <algorithm>
#include <cmath>

namespace {
constexpr int THREADS = 256;

__global__ void __launch_bounds__(THREADS)
k_triangles(const int32_t* __restrict__ R, const int32_t* __restrict__ C, int32_t n,
            unsigned long long* __restrict__ tri2, int* __restrict__ next_node)
{
    extern __shared__ unsigned int bm[];
    __shared__ int s_u;
    __shared__ unsigned long long s_acc[THREADS / 32];
    const int W = (n + 31) >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = THREADS / 32;
    for (int w = threadIdx.x; w < W; w += THREADS) bm[w] = 0u;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_u = atomicAdd(next_node, 1);
        __syncthreads();
        const int u = s_u;
        if (u >= n) break;
        const int32_t s = R[u], e = R[u + 1];
        if (e - s < 2) continue;
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) atomicOr(&bm[C[q] >> 5], 1u << (C[q] & 31));
        __syncthreads();
        // first neighbour index with v > u (columns ascend)
        int32_t lo = s, hi = e;
        while (lo < hi) {
            int32_t mid = (lo + hi) >> 1;
            if (C[mid] > u) hi = mid; else lo = mid + 1;
        }
        unsigned long long acc_u = 0;
        for (int32_t q = lo + warp; q < e; q += nwarp) {
            const int v = C[q];
            unsigned int c = 0;
            for (int32_t f = R[v] + lane; f < R[v + 1]; f += 32) {
                int w = C[f];
                c += (bm[w >> 5] >> (w & 31)) & 1u;
            }
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0 && c) {
                atomicAdd(&tri2[v], (unsigned long long)c);
                acc_u += c;
            }
        }
        if (lane == 0) s_acc[warp] = acc_u;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t = 0;
            for (int w = 0; w < nwarp; w++) t += s_acc[w];
            if (t) atomicAdd(&tri2[u], t);
        }
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) bm[C[q] >> 5] = 0u;
    }
}

// Cp[k] = (double)t / k / (k-1) * 2 rounded to float (Cp.cpp:110), 0 for k < 2.
__global__ void k_cp_binary(const int32_t* __restrict__ R, int32_t n, const unsigned long long* __restrict__ tri2,
                            float* __restrict__ cp, long long* __restrict__ tri)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        int k = R[u + 1] - R[u];
        unsigned long long t = tri2[u] >> 1;
        float c = 0.0f;
        if (k >= 2) {
            double x = (double)t;
            x = __ddiv_rn(x, (double)k);
            x = __ddiv_rn(x, (double)(k - 1));
            x = __dmul_rn(x, 2.0);
            c = __double2float_rn(x);
        }
        cp[u] = c;
        if (tri) tri[u] = (long long)t;
    }
}

// Deterministic FP64 mean of a float vector: one block, fixed order (strided
// per-thread sums, a shuffle tree per warp, one over the warps).  Bound by the
// latency of one block's loads; a chain of n adds in one thread took 645 us
// at 25k values, this 14 us.
__global__ void __launch_bounds__(1024) k_mean_f32(const float* __restrict__ x, int32_t n, double* __restrict__ out)
{
    __shared__ double sh[32];
    double a = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += (double)x[i];
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) *out = n > 0 ? t / n : 0.0;
    }
}

// ---------------------------------------------------------------- Onnela
// Order-preserving map from float to uint32 (larger float -> larger value;
// 0 lies below every float), for the atomic maximum.
__device__ __forceinline__ unsigned fkey(float x)
{
    const unsigned u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(unsigned k)
{
    return k == 0u ? -INFINITY : __uint_as_float((k & 0x80000000u) ? (k & ~0x80000000u) : ~k);
}

// Weight maximum over V[0..lim) (lim = n for the reference CPU rule, nnz
// otherwise), NaN ignored.  One grid-stride pass over all SMs (bound by the
// read of V); the one-block form it replaces took 11.1 ms for 6.4M weights, this 12 us.
__global__ void k_vmax(const float* __restrict__ V, long long lim, OnnelaState* __restrict__ st)
{
    float m = -INFINITY;
    const long long nt = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < lim; q += nt) m = fmaxf(m, V[q]);
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&st->vmax, fkey(m));
}

// Per edge: the cube root of the normalised weight w = V / vmax (float
// division as Cp_2.cpp:37), in FP64; per row: its first entry with a column
// above the row's own index.  Raises st->general when the fast kernel's
// rules do not hold: a normalised weight that is negative or not finite
// (the cube root of the product then differs from the product of the cube
// roots), or columns of a row that do not strictly ascend (an entry's place
// in the row is then not its rank in the neighbour bitmap).
__global__ void __launch_bounds__(THREADS)
k_onnela_roots(const int32_t* __restrict__ R, const int32_t* __restrict__ C, const float* __restrict__ V, int32_t n,
               double* __restrict__ cw, int32_t* __restrict__ up, OnnelaState* __restrict__ st)
{
    const float vm = fkey_inv(st->vmax);
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    bool bad = false;
    for (int u = gw; u < n; u += nw) {
        const int32_t s = R[u], e = R[u + 1];
        int below = 0;
        for (int32_t q = s + lane; q < e; q += 32) {
            const int c = C[q];
            const float w = __fdiv_rn(V[q], vm);
            bad |= !(w >= 0.0f && w < INFINITY) || (q > s && C[q - 1] >= c);
            below += c <= u;
            cw[q] = cbrt((double)w);
        }
        below = __reduce_add_sync(0xffffffffu, below);
        if (lane == 0) up[u] = s + below;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) st->general = 1;
}

// Per node u: sum over connected neighbour pairs j < h of
// (w_jh w_uj w_uh)^(1/3) as the product of the per-edge cube roots (FP64).
// One CTA per node (dynamic scheduler).  The neighbour set is a
// shared-memory table of (bits, neighbours below) per 32 nodes, so one
// 8-byte load both tests h and gives its place in u's row, whose roots lie
// in shared memory too.  A warp takes every eighth neighbour j; it reads the
// ranges of 32 of them at once and scans each row from its first column
// above j, four chunks in flight.  Bound by the shared-memory lookups and
// the L2 reads of the rows: 25,211 nodes / 6.4M entries in 2.1 ms,
// against 16.0 ms when each hit did a binary search and an FP64 pow.
constexpr int ONNELA_ROW = 1536;   // roots of a row kept in shared memory (longer rows: read from L2)

__global__ void __launch_bounds__(THREADS)
k_onnela(const int32_t* __restrict__ R, const int32_t* __restrict__ C, int32_t n, const double* __restrict__ cw,
         const int32_t* __restrict__ up, float* __restrict__ cp, OnnelaState* __restrict__ st)
{
    if (st->general) return;
    extern __shared__ uint2 tab[];       // x: neighbour bits, y: neighbours before these 32 nodes
    __shared__ double rowv[ONNELA_ROW];
    __shared__ int s_u, s_scan[THREADS / 32];
    __shared__ double s_acc[THREADS / 32];
    constexpr int nwarp = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = (n + 31) >> 5, per = (W + THREADS - 1) / THREADS;
    for (int w = threadIdx.x; w < W; w += THREADS) tab[w].x = 0u;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_u = atomicAdd(&st->next, 1);
        __syncthreads();
        const int u = s_u;
        if (u >= n) break;
        const int32_t s = R[u], e = R[u + 1];
        const int k = e - s;
        if (k < 2) {
            if (threadIdx.x == 0) cp[u] = 0.0f;
            continue;
        }
        const bool in_smem = k <= ONNELA_ROW;
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) {
            const int c = C[q];
            atomicOr(&tab[c >> 5].x, 1u << (c & 31));
            if (in_smem) rowv[q - s] = cw[q];
        }
        __syncthreads();
        // exclusive popcount prefix: each thread a run of words, then the block
        const int w0 = min(W, (int)threadIdx.x * per), w1 = min(W, w0 + per);
        int cnt = 0;
        for (int w = w0; w < w1; w++) cnt += __popc(tab[w].x);
        int x = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_scan[warp] = x;
        __syncthreads();
        int run = x - cnt;
        for (int w = 0; w < warp; w++) run += s_scan[w];
        for (int w = w0; w < w1; w++) {
            tab[w].y = run;
            run += __popc(tab[w].x);
        }
        __syncthreads();
        double acc = 0.0;
        for (int q0 = s + warp; q0 < e; q0 += 32 * nwarp) {
            const int q = q0 + lane * nwarp;
            int f0 = 0, f1 = 0;
            double cuj = 0.0;
            if (q < e) {
                const int j = C[q];
                f0 = up[j];
                f1 = R[j + 1];
                cuj = in_smem ? rowv[q - s] : cw[q];
            }
            const int cnt_j = min(32, (e - q0 + nwarp - 1) / nwarp);
            for (int t = 0; t < cnt_j; t++) {
                const int a = __shfl_sync(0xffffffffu, f0, t), b = __shfl_sync(0xffffffffu, f1, t);
                double part = 0.0;
                for (int f = a + lane; f < b; f += 128) {
                    int h[4];
#pragma unroll
                    for (int z = 0; z < 4; z++) h[z] = f + 32 * z < b ? C[f + 32 * z] : -1;
#pragma unroll
                    for (int z = 0; z < 4; z++) {
                        if (h[z] < 0) continue;
                        const uint2 m = tab[h[z] >> 5];
                        if ((m.x >> (h[z] & 31)) & 1u) {
                            const int at = m.y + __popc(m.x & ((1u << (h[z] & 31)) - 1u));
                            part += cw[f + 32 * z] * (in_smem ? rowv[at] : cw[s + at]);
                        }
                    }
                }
                acc += __shfl_sync(0xffffffffu, cuj, t) * part;
            }
        }
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s_acc[warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < nwarp; w++) t += s_acc[w];
            cp[u] = (float)(2.0 * t / k / (k - 1));
        }
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) tab[C[q] >> 5].x = 0u;
    }
}

// The same sum for any weights, any order of a row's columns in j's scan and
// any n whose bitmap fits: a binary search for the weight of (u, h) and the
// cube root of each product, as the reference evaluates it.  Runs only when
// `force` is set (n too large for k_onnela's table) or k_onnela_roots raised
// st->general.
__global__ void __launch_bounds__(THREADS)
k_onnela_general(const int32_t* __restrict__ R, const int32_t* __restrict__ C, const float* __restrict__ V, int32_t n,
                 float* __restrict__ cp, OnnelaState* __restrict__ st, int force)
{
    if (!force && !st->general) return;
    extern __shared__ unsigned int bm[];
    __shared__ int s_u;
    __shared__ double s_acc[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = THREADS / 32;
    const int W = (n + 31) >> 5;
    const float vm = fkey_inv(st->vmax);
    for (int w = threadIdx.x; w < W; w += THREADS) bm[w] = 0u;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_u = atomicAdd(&st->next, 1);
        __syncthreads();
        const int u = s_u;
        if (u >= n) break;
        const int32_t s = R[u], e = R[u + 1];
        const int k = e - s;
        if (k < 2) {
            if (threadIdx.x == 0) cp[u] = 0.0f;
            continue;
        }
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) atomicOr(&bm[C[q] >> 5], 1u << (C[q] & 31));
        __syncthreads();
        double acc = 0.0;
        for (int32_t q = s + warp; q < e; q += nwarp) {
            const int j = C[q];
            const double wuj = (double)__fdiv_rn(V[q], vm);
            for (int32_t f = R[j] + lane; f < R[j + 1]; f += 32) {
                const int h = C[f];
                if (h <= j || !((bm[h >> 5] >> (h & 31)) & 1u)) continue;
                const float wjh = __fdiv_rn(V[f], vm);
                if (wjh == 0.0f) continue;
                int32_t lo = s, hi = e - 1;
                while (lo < hi) {
                    int32_t mid = (lo + hi) >> 1;
                    if (C[mid] < h) lo = mid + 1; else hi = mid;
                }
                const double wuh = (double)__fdiv_rn(V[lo], vm);
                acc += pow((double)wjh * wuj * wuh, 1.0 / 3.0);
            }
        }
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s_acc[warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < nwarp; w++) t += s_acc[w];
            cp[u] = (float)(2.0 * t / k / (k - 1));
        }
        for (int32_t q = s + threadIdx.x; q < e; q += THREADS) bm[C[q] >> 5] = 0u;
    }
}
}  // namespace

pg_status onnela_prepare(pg_ctx* ctx, const pg_graph* g, int first_n, float* cp_dev, double* mean_dev, OnnelaArgs* a)
{
    if (!g->V) return pg_fail(ctx, PG_ERR_INVALID, "Onnela clustering needs a weighted graph");
    a->R = g->R;
    a->C = g->C;
    a->V = g->V;
    a->n = g->n;
    a->nnz = g->nnz;
    a->vmax_entries = first_n ? std::min((int64_t)g->n, g->nnz) : g->nnz;
    a->cp = cp_dev;
    a->mean = mean_dev;
    const size_t words = (size_t)((std::max(g->n, 1) + 31) / 32);
    a->smem_general = words * 4;
    if (a->smem_general > ctx->smem_optin - 4096)
        return pg_fail(ctx, PG_ERR_TOO_LARGE, "Onnela: n=%d too large", g->n);
    // the table of k_onnela takes twice the bitmap's shared memory, beside the
    // row's roots: graphs beyond it (about 850,000 nodes) take the general
    // kernel, and so do those whose table of roots finds no memory
    a->smem = words * 8;
    a->fast = a->smem + ONNELA_ROW * 8 + 1024 <= ctx->smem_optin;
    PG_TRY(pg_wst(ctx, "on.state", 1, &a->state));
    if (a->fast) {
        a->fast = pg_wst(ctx, "on.roots", (size_t)g->nnz, &a->roots) == PG_OK &&
                  pg_wst(ctx, "on.up", (size_t)g->n, &a->up) == PG_OK;
        if (a->smem + ONNELA_ROW * 8 > 48 * 1024 - 1024)
            PG_CUDA(ctx, cudaFuncSetAttribute(k_onnela, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a->smem));
    }
    if (a->smem_general > 48 * 1024)
        PG_CUDA(ctx, cudaFuncSetAttribute(k_onnela_general, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)a->smem_general));
    return PG_OK;
}

pg_status onnela_enqueue(pg_ctx* ctx, const OnnelaArgs* a)
{
    PG_CUDA(ctx, cudaMemsetAsync(a->state, 0, sizeof(OnnelaState), ctx->stream));
    const int wide = ctx->sm_count * 8;
    k_vmax<<<wide, 256, 0, ctx->stream>>>(a->V, a->vmax_entries, a->state);
    PG_LAUNCHED(ctx);
    if (a->fast) {
        k_onnela_roots<<<wide, THREADS, 0, ctx->stream>>>(a->R, a->C, a->V, a->n, a->roots, a->up, a->state);
        PG_LAUNCHED(ctx);
        k_onnela<<<wide, THREADS, a->smem, ctx->stream>>>(a->R, a->C, a->n, a->roots, a->up, a->cp, a->state);
        PG_LAUNCHED(ctx);
    }
    k_onnela_general<<<ctx->sm_count * 4, THREADS, a->smem_general, ctx->stream>>>(a->R, a->C, a->V, a->n, a->cp,
                                                                                  a->state, !a->fast);
    PG_LAUNCHED(ctx);
    k_mean_f32<<<1, 1024, 0, ctx->stream>>>(a->cp, a->n, a->mean);
    PG_LAUNCHED(ctx);
    return PG_OK;
}

// Binary clustering of one graph, enqueued only: per-node Cp (float), exact
// triangles (optional) and the FP64 mean over all nodes, in device memory.
pg_status binary_cp_prepare(pg_ctx* ctx, int n, BinaryCpArgs* a)
{
    PG_TRY(pg_wst(ctx, "cl.tri2", (size_t)n + 1, &a->tri2));
    PG_TRY(pg_wst(ctx, "cl.ctr", 1, &a->counter));
    a->smem = (size_t)((n + 31) / 32) * 4;
    if (a->smem > ctx->smem_optin - 4096) return pg_fail(ctx, PG_ERR_TOO_LARGE, "clustering: n=%d too large", n);
    if (a->smem > 48 * 1024)
        PG_CUDA(ctx, cudaFuncSetAttribute(k_triangles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a->smem));
    return PG_OK;
}

pg_status binary_cp_enqueue(pg_ctx* ctx, const BinaryCpArgs* a, const int32_t* R, const int32_t* C, int n, float* cp,
                            long long* tri, double* mean)
{
    PG_CUDA(ctx, cudaMemsetAsync(a->tri2, 0, sizeof(unsigned long long) * (n + 1), ctx->stream));
    PG_CUDA(ctx, cudaMemsetAsync(a->counter, 0, sizeof(int), ctx->stream));
    if (n > 0) {
        k_triangles<<<ctx->sm_count * 4, THREADS, a->smem, ctx->stream>>>(R, C, n, a->tri2, a->counter);
        PG_LAUNCHED(ctx);
        k_cp_binary<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>(R, n, a->tri2, cp, tri);
        PG_LAUNCHED(ctx);
    }
    k_mean_f32<<<1, 1024, 0, ctx->stream>>>(cp, n, mean);
    PG_LAUNCHED(ctx);
    return PG_OK;
}

extern "C" pg_status pg_clustering(pg_ctx* ctx, const pg_graph* g, int32_t kind, int32_t flags, float* cp,
                                   int64_t* triangles, double* mean)
{
    if (!ctx || !g || !cp) return pg_fail(ctx, PG_ERR_INVALID, "pg_clustering: null argument");
    PG_CUDA(ctx, cudaSetDevice(ctx->device));
    const int n = g->n;
    const WsIdleAtExit<2> idle{ctx, {"on.roots", "on.up"}};   // 8 bytes per entry, for this call
    float* dcp;
    double* dmean;
    PG_TRY(pg_wst(ctx, "cl.cp", (size_t)n + 1, &dcp));
    PG_TRY(pg_wst(ctx, "cl.mean", 1, &dmean));
    if (kind == 0) {
        long long* tri = nullptr;
        BinaryCpArgs a;
        PG_TRY(binary_cp_prepare(ctx, n, &a));
        if (triangles) PG_TRY(pg_wst(ctx, "cl.tri", (size_t)n + 1, &tri));
        PG_TRY(binary_cp_enqueue(ctx, &a, g->R, g->C, n, dcp, tri, dmean));
        if (triangles) PG_TRY(pg_d2h(ctx, triangles, tri, sizeof(long long) * n));
    } else if (kind == 1) {
        OnnelaArgs a;
        PG_TRY(onnela_prepare(ctx, g, flags & 1, dcp, dmean, &a));
        PG_TRY(onnela_enqueue(ctx, &a));
    } else {
        return pg_fail(ctx, PG_ERR_INVALID, "unknown clustering kind %d", kind);
    }
    PG_TRY(pg_d2h(ctx, cp, dcp, sizeof(float) * n));
    if (mean) PG_TRY(pg_d2h(ctx, mean, dmean, sizeof(double)));
    return PG_OK;
}

// ------------------------------------------------ allocation-free variant
// Binary clustering for callers that cannot allocate device memory: host
// processes whose device memory is owned by someone else (a framework's
// caching allocator or a plugin host that reserves the GPU up front), and
// latency-critical pipelines that forbid cudaMalloc after start-up because
// it can synchronise the device.  The per-node triangle counters live in
// this file-scope device array instead of a workspace allocation.  Every
// call shares it and it keeps the last call's contents, so it is cleared at
// the start of each call, and calls that overlap on the GPU (other streams,
// other host threads) race on it.
namespace {
constexpr int64_t NOALLOC_SCRATCH_WORDS = (16LL << 20) / 8;   // 16 MiB: n + 2 counters
static __device__ __align__(256) unsigned long long g_noalloc_scratch[NOALLOC_SCRATCH_WORDS];
constexpr int NOALLOC_MAX_DEVICES = 64;
constexpr int NOALLOC_SMEM_SLACK = 4096;   // static shared memory of k_triangles and margin

// Set-up state per device, filled by the first call with that device
// current: the array's device address (the host-side symbol is only a
// stand-in), the SM count and the opt-in shared memory per block, and the id
// of the CUDA context they belong to.  A new context on the device (after
// cudaDeviceReset) has a new id, and the next call resolves the address again.
struct NoallocDevice {
    unsigned long long* scratch;
    unsigned long long ctx_id;
    int sm_count;
    int smem_optin;
};
static NoallocDevice g_noalloc_dev[NOALLOC_MAX_DEVICES];

__global__ void k_noalloc_clear(unsigned long long* __restrict__ w, int64_t count)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x)
        w[q] = 0ULL;
}

// Largest n whose neighbour bitmap (n bits) fits the opt-in shared memory.
int64_t noalloc_smem_nodes(int smem_optin) { return (int64_t)(smem_optin - NOALLOC_SMEM_SLACK) / 4 * 32; }

// cuCtxGetCurrent / cuCtxGetId through the runtime's driver entry points
// (the library does not link the driver library directly).
bool current_ctx_id(unsigned long long* id)
{
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    if (!get_current || !get_id) {
        void *p = nullptr, *q = nullptr;
        cudaDriverEntryPointQueryResult r1, r2;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &r1) != cudaSuccess ||
            r1 != cudaDriverEntryPointSuccess ||
            cudaGetDriverEntryPoint("cuCtxGetId", &q, cudaEnableDefault, &r2) != cudaSuccess ||
            r2 != cudaDriverEntryPointSuccess)
            return false;
        get_current = (GetCurrent)p;
        get_id = (GetId)q;
    }
    CUcontext c = nullptr;
    if (get_current(&c) != CUDA_SUCCESS || !c) return false;
    return get_id(c, id) == CUDA_SUCCESS;
}

pg_status noalloc_setup(int dev, NoallocDevice** out)
{
    NoallocDevice& d = g_noalloc_dev[dev];
    unsigned long long id = 0;
    if (d.scratch && current_ctx_id(&id) && id == d.ctx_id) {
        *out = &d;
        return PG_OK;
    }
    void* p = nullptr;   // resolving the symbol also initialises the device's context
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return PG_ERR_CUDA;
    int sms = 0, optin = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return PG_ERR_CUDA;
    if (!current_ctx_id(&id)) return PG_ERR_CUDA;
    d.scratch = (unsigned long long*)p;
    d.ctx_id = id;
    d.sm_count = sms;
    d.smem_optin = optin;
    *out = &d;
    return PG_OK;
}
}  // namespace

extern "C" int64_t pg_clustering_noalloc_max_nodes(void)
{
    int64_t lim = NOALLOC_SCRATCH_WORDS - 2;
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess)
        lim = std::min(lim, noalloc_smem_nodes(optin));
    return lim;
}

extern "C" pg_status pg_clustering_noalloc(const int32_t* R, const int32_t* C, int32_t n, float* cp, int64_t* triangles,
                                           void* stream)
{
    if (!R || !cp || n < 0) return PG_ERR_INVALID;
    if ((int64_t)n > NOALLOC_SCRATCH_WORDS - 2) return PG_ERR_TOO_LARGE;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return PG_ERR_NO_DEVICE;
    NoallocDevice* d = nullptr;
    if (pg_status st = noalloc_setup(dev, &d); st != PG_OK) return st;
    if (n == 0) return PG_OK;
    if ((int64_t)n > noalloc_smem_nodes(d->smem_optin)) return PG_ERR_TOO_LARGE;
    const size_t smem = (size_t)((n + 31) / 32) * 4;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(k_triangles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return PG_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* tri2 = d->scratch;
    int* next_node = (int*)(tri2 + (n + 1));
    k_noalloc_clear<<<d->sm_count, 256, 0, st>>>(tri2, (int64_t)n + 2);
    k_triangles<<<d->sm_count * 4, THREADS, smem, st>>>(R, C, n, tri2, next_node);
    k_cp_binary<<<d->sm_count * 4, 256, 0, st>>>(R, n, tri2, cp, (long long*)triangles);
    return cudaGetLastError() == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}
