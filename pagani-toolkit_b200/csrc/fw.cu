// fw.cu -- weighted path length by blocked Floyd-Warshall in FP32 min-plus
// (CUBFW_Lp, W/Lp/CUBFW_Lp/CUBFW_Lp/CUBFW_Lp.cpp:13-162; phases of cuAPSP,
// CUBFW.cpp:19-168, CUBFW_ph1/2/3.cu, and BFW_C, BFW.cpp:40-109) and Onnela
// weighted clustering (Cp_2, W/Cp/Cp/Cp_2.cpp:23-130) for one graph or a
// batch of graphs in ONE persistent cooperative launch.
//
// Every graph's dense distance matrix (padded to a multiple of 64) stays on
// the device (the reference streams 3072^2 blocks over PCIe per phase and
// pads every graph to 3072).  The launch first computes, over the whole grid,
// the weight maxima, the cube roots of the normalised weights and the Onnela
// clustering of every node; then its CTAs work in teams (one, but for very
// large batches: fw_plan.h), each of which takes one bundle of graphs after
// another from a queue (largest first) and sweeps its graphs in step:
//   A  the rows: +inf, 0 on the diagonal, 1/w for the edges;
//   then for every 64-wide k-block round kb:
//   1  the row and column panels, closed in place against the closed diagonal
//      block (64 steps in order, eight at a time);
//   2  every other block: d_ij = min(d_ij, d_i,kb (x) d_kb,j); the diagonal
//      block of the next round comes first and is closed at once (64 steps in
//      registers), so no phase of its own waits for it;
//   C  per-row sums of 1/d (CUBFW_Lp.cpp:77-104);
// and at the end, per graph, Lp and the mean clustering.  The k-block width
// is fixed (64), every block is closed in the same order of steps and the
// per-graph sums run over the nodes in order, so no result depends on the
// teams or on the grid.
#include "pg_internal.cuh"
#include "fw_plan.h"
#include <algorithm>
#include <cmath>
#include <cooperative_groups.h>
#include <numeric>

namespace cg = cooperative_groups;

namespace {
constexpr int B = 64;           // k-block width
// One CTA per SM of four groups of 128 threads; a group works on a block (or
// a node) of its own and synchronises by itself (named barrier), so that a
// grid barrier has 148 arrivals and an SM still holds four blocks at once
// (592 CTAs of 128 threads spent 13 us per panel phase, mostly in barriers).
constexpr int GROUPS = 4, GT = 128;
constexpr int FW_THREADS = GROUPS * GT;
constexpr int TR = 8;   // a thread's tile: rows t / 16 + 8 r, columns 2 (t % 16), + 1, + 32, + 33
constexpr int MAX_TEAMS = 64;
constexpr int ONNELA_MAX_N = 4096; // largest graph of a batch for the Onnela row (n doubles in shared memory)

struct FWGraph {
    const int32_t* R;
    const int32_t* C;
    const float* V;     // null: every edge has distance 1
    int32_t n, np, nb;  // nodes, padded size, blocks per side
    int32_t index;      // the caller's graph number
    long long off;      // matrix offset (elements)
    long long edge0;    // offset of its entries in cw
    int32_t node0;      // its nodes in processing order
    int32_t out0;       // and in the caller's concatenated outputs
    // sums over the graphs before it (the table has one entry more, for the totals):
    long long row0;     // padded rows
    long long panel0;   // panel blocks of a round, 2 (nb - 1)
    long long inner0;   // other blocks of a round without a diagonal one, (nb - 1)^2 - 1 (0 for one block)
};

struct FwControl {
    int onnela_next;    // dynamic node scheduler
    int queue;          // next bundle
    int timeout;        // a team barrier gave up
    int pad;
    unsigned arrived[MAX_TEAMS];
    int bundle[MAX_TEAMS];  // the bundle a team works on
};

struct FwBatch {
    const FWGraph* gs;          // in processing order (blocks per side descending)
    int ng;
    int total_nodes;
    int teams;
    int bundles;
    const int* bundle0;         // first graph of every bundle, and ng
    FwControl* ctl;
    float* D;
    float* vmax;                // per graph
    double* cw;                 // per entry of every graph: (V / vmax)^(1/3)
    int32_t* up;                // per node: where the entries of its row with a column above it begin
    int onnela;                 // compute the clustering
    unsigned max_spins;         // reads of the counter that a team barrier waits for
    int hold;                   // failure-path test hook: a CTA of every team does not arrive
    double* rowsum;             // per node, in processing order
    float* eff;                 // per node, in the caller's order
    double* lp;                 // per graph, in the caller's order; then 1.0 after a timeout
    float* cp;                  // per node, in the caller's order
    double* cp_mean;            // per graph, in the caller's order
};

__device__ __forceinline__ float* blk(float* D, const FWGraph& g, int bi, int bj)
{
    return D + g.off + (long long)bi * B * g.np + (long long)bj * B;
}

__device__ __forceinline__ int group_thread() { return threadIdx.x & (GT - 1); }
__device__ __forceinline__ void group_sync()
{
    asm volatile("bar.sync %0, %1;" ::"r"(1 + ((int)threadIdx.x >> 7)), "n"(GT) : "memory");
}

// Onnela for node x of the batch (W/Cp/Cp/Cp_2.cpp:23-130, GPU weight maximum
// over all edges): sum over connected neighbour pairs j < h of
// (w_jh w_uj w_uh)^(1/3), w = V / vmax (float division), computed as
// cw_jh cw_uj cw_uh with the per-edge cube roots cw = w^(1/3) (FP64; the
// same value up to rounding).  u's row is spread into a dense shared-memory
// array (zero where h is not a neighbour), so the weight of (u, h) is one
// shared load.
__device__ void onnela_node(const FwBatch& p, const FWGraph& g, int u, double* row, double* red)
{
    const int lane = group_thread() & 31, warp = group_thread() >> 5, nwarp = GT / 32;
    const int32_t s = g.R[u], e = g.R[u + 1];
    const int k = e - s;
    double acc = 0.0;
    if (k >= 2) {
        const double* cw = p.cw + g.edge0;
        for (int32_t q = s + group_thread(); q < e; q += GT) row[g.C[q]] = cw[q];
        group_sync();
        // a warp takes every fourth neighbour j, the ranges of 32 of them read
        // at once; row j from its first column above j
        for (int32_t q0 = s + warp; q0 < e; q0 += 32 * nwarp) {
            const int32_t q = q0 + lane * nwarp;
            int j = 0, f0 = 0, f1 = 0;
            double cuj = 0.0;
            if (q < e) {
                j = g.C[q];
                f0 = p.up[g.node0 + j];
                f1 = g.R[j + 1];
                cuj = cw[q];
            }
            const int cnt = min(32, (e - q0 + nwarp - 1) / nwarp);
            // four chunks of 32 entries from entry f on, up to b
            auto fetch = [&](int f, int b, int (&h)[4], double (&w)[4]) {
#pragma unroll
                for (int z = 0; z < 4; z++) {
                    h[z] = f + 32 * z < b ? g.C[f + 32 * z] : -1;
                    w[z] = f + 32 * z < b ? cw[f + 32 * z] : 0.0;
                }
            };
            int h[4], hn[4];
            double w[4], wn[4];
            int a = __shfl_sync(0xffffffffu, f0, 0), b = __shfl_sync(0xffffffffu, f1, 0);
            fetch(a + lane, b, hn, wn);
            for (int t = 0; t < cnt; t++) {
#pragma unroll
                for (int z = 0; z < 4; z++) {
                    h[z] = hn[z];
                    w[z] = wn[z];
                }
                const int jt = __shfl_sync(0xffffffffu, j, t), f_next = a + lane + 128, b_here = b;
                // the next neighbour's row is on its way while this one is added
                a = __shfl_sync(0xffffffffu, f0, min(t + 1, 31));
                b = t + 1 < cnt ? __shfl_sync(0xffffffffu, f1, t + 1) : 0;
                fetch(a + lane, b, hn, wn);
                double part = 0.0;
                for (int f = f_next;; f += 128) {
#pragma unroll
                    for (int z = 0; z < 4; z++)
                        if (h[z] > jt) part += w[z] * row[h[z]];
                    if (f - lane >= b_here) break;
                    fetch(f, b_here, h, w);
                }
                acc += __shfl_sync(0xffffffffu, cuj, t) * part;
            }
        }
        group_sync();
        for (int32_t q = s + group_thread(); q < e; q += GT) row[g.C[q]] = 0.0;
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) red[warp] = acc;
    group_sync();
    if (group_thread() == 0) {
        double t = 0.0;
        for (int w = 0; w < nwarp; w++) t += red[w];
        p.cp[g.out0 + u] = k >= 2 ? (float)(2.0 * t / k / (k - 1)) : 0.0f;
    }
    group_sync();
}

// min(a, b, c) in one instruction (sm_100)
__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// two FP32 additions in one instruction (sm_100)
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    unsigned long long x, y, z;
    memcpy(&x, &a, 8);
    memcpy(&y, &b, 8);
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
    float2 r;
    memcpy(&r, &z, 8);
    return r;
}

struct __align__(16) FwSmem {
    union {
        struct {
            float a[B][B + 4];      // left operand, row-major: a[i][k]
            float2 b[B / 2][B];     // right operand, rows k and k + 1 interleaved: b[k / 2][j]
        } prod;
        struct {
            float dg[B][B + 4];     // the closed diagonal block (transposed for a column panel)
            float rows[8][B];       // the eight rows whose steps come next
            float2 b[4][B];         // the same at their own steps, two and two interleaved
            float tr[B][B + 1];     // for turning a column panel
        } panel;
        struct {
            float row[2][B];        // row k of the block being closed
            float col[2][B];        // column k
        } close;
        double row[ONNELA_MAX_N];   // Onnela: the node's row, dense
    };
    double red[GT / 32];
    int next;                       // Onnela: the node taken
};

// The thread's 8 x 4 outputs of a 64 x 64 block.
struct Tile {
    float v[TR][4];
    __device__ __forceinline__ void load(const float* src, int ld)
    {
        const int i0 = group_thread() >> 4, j = 2 * (group_thread() & 15);
#pragma unroll
        for (int r = 0; r < TR; r++) {
            const float2 x = *(const float2*)(src + (long long)(i0 + 8 * r) * ld + j);
            const float2 y = *(const float2*)(src + (long long)(i0 + 8 * r) * ld + j + 32);
            v[r][0] = x.x; v[r][1] = x.y; v[r][2] = y.x; v[r][3] = y.y;
        }
    }
    __device__ __forceinline__ void store(float* dst, int ld) const
    {
        const int i0 = group_thread() >> 4, j = 2 * (group_thread() & 15);
#pragma unroll
        for (int r = 0; r < TR; r++) {
            *(float2*)(dst + (long long)(i0 + 8 * r) * ld + j) = make_float2(v[r][0], v[r][1]);
            *(float2*)(dst + (long long)(i0 + 8 * r) * ld + j + 32) = make_float2(v[r][2], v[r][3]);
        }
    }
    // the block's transpose (no bank is hit twice by a warp, either way)
    __device__ __forceinline__ void transpose(float (*tr)[B + 1])
    {
        const int i0 = group_thread() >> 4, j = 2 * (group_thread() & 15);
#pragma unroll
        for (int r = 0; r < TR; r++)
#pragma unroll
            for (int x = 0; x < 4; x++) tr[i0 + 8 * r][j + (x & 1) + 16 * (x & 2)] = v[r][x];
        group_sync();
#pragma unroll
        for (int r = 0; r < TR; r++)
#pragma unroll
            for (int x = 0; x < 4; x++) v[r][x] = tr[j + (x & 1) + 16 * (x & 2)][i0 + 8 * r];
    }
};

// c = min(c, a (x) b) over 64 x 64 blocks, the first kn of their 64 steps
// (the others are padding).  Two k per step: the sums of rows k and k + 1 are
// one packed addition (the left operand holds consecutive k, the right one
// interleaves its rows), and one three-input minimum folds both; min is
// exact, so the order does not matter.  Per four k a thread issues 64 packed
// additions, 64 minima and 12 16-byte shared loads for 128 updates.  Bound by
// the minima: the loop alone runs at 65 updates per clock and SM whether two-
// or three-input minima are used (60 with scalar additions), four blocks at
// once in an SM at 51 with their loads and stores.
__device__ __forceinline__ void min_plus(FwSmem& sm, Tile& c, const float* a, const float* b, int ld, int kn)
{
    const int t = group_thread();
    // operands into shared memory: 64 rows x 16 float4 each
#pragma unroll
    for (int it = 0; it < B * B / 4 / GT; it++) {
        const int q = t + it * GT, i = q >> 4, j = (q & 15) << 2;
        *(float4*)&sm.prod.a[i][j] = *(const float4*)(a + (long long)i * ld + j);
    }
#pragma unroll
    for (int it = 0; it < B * B / 8 / GT; it++) {
        const int q = t + it * GT, k2 = q >> 4, j = (q & 15) << 2;
        const float4 x = *(const float4*)(b + (long long)(2 * k2) * ld + j);
        const float4 y = *(const float4*)(b + (long long)(2 * k2 + 1) * ld + j);
        *(float4*)&sm.prod.b[k2][j] = make_float4(x.x, y.x, x.y, y.y);
        *(float4*)&sm.prod.b[k2][j + 2] = make_float4(x.z, y.z, x.w, y.w);
    }
    group_sync();
    const int i0 = t >> 4, j0 = 2 * (t & 15);
#pragma unroll 2
    for (int k = 0; k < kn; k += 4) {
        float4 bl[2], bh[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            bl[h] = *(const float4*)&sm.prod.b[k / 2 + h][j0];
            bh[h] = *(const float4*)&sm.prod.b[k / 2 + h][j0 + 32];
        }
#pragma unroll
        for (int r = 0; r < TR; r++) {
            const float4 x = *(const float4*)&sm.prod.a[i0 + 8 * r][k];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 ak = h ? make_float2(x.z, x.w) : make_float2(x.x, x.y);
                const float2 s0 = add2(ak, make_float2(bl[h].x, bl[h].y)), s1 = add2(ak, make_float2(bl[h].z, bl[h].w));
                const float2 s2 = add2(ak, make_float2(bh[h].x, bh[h].y)), s3 = add2(ak, make_float2(bh[h].z, bh[h].w));
                c.v[r][0] = min3f(c.v[r][0], s0.x, s0.y);
                c.v[r][1] = min3f(c.v[r][1], s1.x, s1.y);
                c.v[r][2] = min3f(c.v[r][2], s2.x, s2.y);
                c.v[r][3] = min3f(c.v[r][3], s3.x, s3.y);
            }
        }
    }
    group_sync();   // the operands are overwritten next
}

// A panel block closed against the closed diagonal block dg, in place: step k
// is s_ij = min(s_ij, dg_ik + s_kj) in a row panel, and the same of the
// transposed blocks in a column panel.  The steps' order is part of the
// result: a product with the untouched panel is as exact, but it associates
// the FP32 sums of paths of three and more edges the other way round, which
// moves distances by their last bit.
// Eight steps at a time: their rows go to shared memory, a thread per column
// brings them to their own steps (a triangle of updates), and every thread
// folds them into its tile as min_plus does.  The minima are exact, so this
// equals the 64 steps, which took a barrier each (2,500 nodes: 2.02 ms, with
// the panels as plain products 1.85, with 64 barriers a panel 2.82; with the
// triangle in every thread and one barrier instead of two 2.06).
__device__ __forceinline__ void close_panel(FwSmem& sm, Tile& c, const float* dg, float* d, int ld, bool row, int kn)
{
    const int t = group_thread(), i0 = t >> 4, j0 = 2 * (t & 15);
    // the solvers: two warps of the group, other ones in every second group (an
    // SM's four schedulers each hold a warp of every group)
    const int j = t & (B - 1);
    const bool solver = (t >> 6) == ((threadIdx.x >> 7) & 1);
    c.load(d, ld);
#pragma unroll
    for (int it = 0; it < B * B / 4 / GT; it++) {
        const int q = t + it * GT;
        if (row) {
            const int i = q >> 4, j = (q & 15) << 2;
            *(float4*)&sm.panel.dg[i][j] = *(const float4*)(dg + (long long)i * ld + j);
        } else {   // a warp stores 32 consecutive words
            const int i = q & (B - 1), j = (q >> 6) << 2;
            const float4 x = *(const float4*)(dg + (long long)i * ld + j);
            sm.panel.dg[j][i] = x.x;
            sm.panel.dg[j + 1][i] = x.y;
            sm.panel.dg[j + 2][i] = x.z;
            sm.panel.dg[j + 3][i] = x.w;
        }
    }
    if (!row) c.transpose(sm.panel.tr);
#pragma unroll 1
    for (int k0 = 0; k0 < kn; k0 += 8) {
        float own[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            own[x] = c.v[0][x];
#pragma unroll
            for (int r = 1; r < TR; r++) own[x] = k0 == 8 * r ? c.v[r][x] : own[x];
        }
        *(float2*)&sm.panel.rows[i0][j0] = make_float2(own[0], own[1]);
        *(float2*)&sm.panel.rows[i0][j0 + 32] = make_float2(own[2], own[3]);
        group_sync();
        if (solver) {
            float2 s[4];   // rows k0 + 2 h, + 1 of column j
#pragma unroll
            for (int h = 0; h < 4; h++) s[h] = make_float2(sm.panel.rows[2 * h][j], sm.panel.rows[2 * h + 1][j]);
#pragma unroll
            for (int k = 1; k < 8; k++) {
                const float4 lo = *(const float4*)&sm.panel.dg[k0 + k][k0], hi = *(const float4*)&sm.panel.dg[k0 + k][k0 + 4];
                const float2 a[4] = {{lo.x, lo.y}, {lo.z, lo.w}, {hi.x, hi.y}, {hi.z, hi.w}};
                float& v = (k & 1) ? s[k / 2].y : s[k / 2].x;
#pragma unroll
                for (int h = 0; h < k / 2; h++) {
                    const float2 p = add2(a[h], s[h]);
                    v = min3f(v, p.x, p.y);
                }
                if (k & 1) v = fminf(v, a[k / 2].x + s[k / 2].x);
            }
#pragma unroll
            for (int h = 0; h < 4; h++) sm.panel.b[h][j] = s[h];
        }
        group_sync();   // `rows` is free; `b` is written again behind the next barrier
        float4 bl[4], bh[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            bl[h] = *(const float4*)&sm.panel.b[h][j0];
            bh[h] = *(const float4*)&sm.panel.b[h][j0 + 32];
        }
#pragma unroll
        for (int r = 0; r < TR; r++) {
            const float4 lo = *(const float4*)&sm.panel.dg[i0 + 8 * r][k0], hi = *(const float4*)&sm.panel.dg[i0 + 8 * r][k0 + 4];
            const float2 a[4] = {{lo.x, lo.y}, {lo.z, lo.w}, {hi.x, hi.y}, {hi.z, hi.w}};
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float2 s0 = add2(a[h], make_float2(bl[h].x, bl[h].y)), s1 = add2(a[h], make_float2(bl[h].z, bl[h].w));
                const float2 s2 = add2(a[h], make_float2(bh[h].x, bh[h].y)), s3 = add2(a[h], make_float2(bh[h].z, bh[h].w));
                c.v[r][0] = min3f(c.v[r][0], s0.x, s0.y);
                c.v[r][1] = min3f(c.v[r][1], s1.x, s1.y);
                c.v[r][2] = min3f(c.v[r][2], s2.x, s2.y);
                c.v[r][3] = min3f(c.v[r][3], s3.x, s3.y);
            }
        }
    }
    if (!row) c.transpose(sm.panel.tr);
    c.store(d, ld);
    group_sync();   // shared memory is overwritten next
}

// Closure of a diagonal block held in registers: row k and column k do not
// change in step k (d_kk = 0), so at every step their owners publish them to
// shared rows (double-buffered: one barrier per step).
__device__ __forceinline__ void close_block(FwSmem& sm, Tile& c)
{
    const int ti = group_thread() >> 4, tj = group_thread() & 15;
#pragma unroll
    for (int rk = 0; rk < TR; rk++) {
#pragma unroll 1
        for (int k8 = 0; k8 < 8; k8 += 2) {
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {   // step k = 8 rk + k8 + kk
                constexpr int half = 32 / 8;
                if (ti == k8 + kk) {
                    *(float2*)&sm.close.row[kk][2 * tj] = make_float2(c.v[rk][0], c.v[rk][1]);
                    *(float2*)&sm.close.row[kk][2 * tj + 32] = make_float2(c.v[rk][2], c.v[rk][3]);
                }
                if (tj == ((8 * rk) & 31) / 2 + k8 / 2) {
#pragma unroll
                    for (int r = 0; r < TR; r++) sm.close.col[kk][ti + 8 * r] = c.v[r][kk + (rk >= half ? 2 : 0)];
                }
                group_sync();
                const float2 b0 = *(const float2*)&sm.close.row[kk][2 * tj], b1 = *(const float2*)&sm.close.row[kk][2 * tj + 32];
#pragma unroll
                for (int r = 0; r < TR; r++) {
                    const float a = sm.close.col[kk][ti + 8 * r];
                    c.v[r][0] = fminf(c.v[r][0], a + b0.x);
                    c.v[r][1] = fminf(c.v[r][1], a + b0.y);
                    c.v[r][2] = fminf(c.v[r][2], a + b1.x);
                    c.v[r][3] = fminf(c.v[r][3], a + b1.y);
                }
            }
        }
    }
    group_sync();
}

// Barrier of a team's CTAs (all resident: the launch is cooperative).  The
// wait is bounded; after a timeout nobody waits any more and the host reports
// an error.
constexpr unsigned MAX_SPINS = 1u << 27;
struct Team {
    unsigned* arrived;
    int* timeout;
    unsigned size, target, max_spins;
    bool hold;          // test hook: this CTA's first arrival waits for a peer to give up
    __device__ void sync()
    {
        __syncthreads();
        target += size;
        if (threadIdx.x == 0) {
            if (hold)
                for (unsigned spins = 0; spins < MAX_SPINS && !*(volatile int*)timeout; spins++) {}
            __threadfence();
            atomicAdd(arrived, 1u);
            volatile unsigned* seen = arrived;
            for (unsigned spins = 0; *seen < target; spins++) {
                if (spins > max_spins || *(volatile int*)timeout) {
                    atomicExch(timeout, 1);
                    break;
                }
            }
            __threadfence();
        }
        hold = false;
        __syncthreads();
    }
    // The barrier, then the bundle that the team's first CTA took, or -1 after
    // a timeout.  One thread reads both for its CTA: another team may raise
    // the timeout between two reads, and a CTA whose threads saw different
    // values would leave some of them in the sweep and the others behind it.
    __device__ int sync_bundle(const int* bundle, int& shared_slot)
    {
        sync();
        if (threadIdx.x == 0) shared_slot = *(volatile int*)timeout ? -1 : *(volatile const int*)bundle;
        __syncthreads();
        return shared_slot;   // written again only behind the next barrier
    }
};

// the graph of node x (processing order), searched upwards from gi
__device__ __forceinline__ int graph_at(const FwBatch& p, int gi, long long x)
{
    while (x >= p.gs[gi].node0 + p.gs[gi].n) gi++;
    return gi;
}

// the graph among [a, b) whose share of a task list holds task x (counted over
// all graphs); SUM is the table's running sum of the list
template <long long FWGraph::*SUM>
__device__ __forceinline__ int task_graph(const FwBatch& p, int a, int b, long long x)
{
    int lo = a, hi = b - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.gs[mid].*SUM <= x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Floyd-Warshall of the graphs [a, b) by the CTAs of a team, all in step: a
// round's blocks of all graphs that have it form one task list.  This group is
// number vb of the team's nvb.
__device__ __forceinline__ void fw_bundle(const FwBatch& p, int a, int b, Team& team, FwSmem& sm, int vb, int nvb)
{
    const int lane = group_thread() & 31, gw = vb * (GT / 32) + (group_thread() >> 5), nw = nvb * (GT / 32);
    // ---- A: a warp per row (init_block, FormBlock.cpp:64)
    {
        const long long first = p.gs[a].row0, rows = p.gs[b].row0 - first;
        int gi = a;
        for (long long x = gw; x < rows; x += nw) {
            while (x >= p.gs[gi + 1].row0 - first) gi++;
            const FWGraph g = p.gs[gi];
            const int i = (int)(x - (g.row0 - first));
            float* d = p.D + g.off + (long long)i * g.np;
            for (int j = 4 * lane; j < g.np; j += 128) {
                float4 v = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
                if (i >= j && i < j + 4) ((float*)&v)[i - j] = 0.0f;
                *(float4*)(d + j) = v;
            }
            __syncwarp();   // the row is filled before its edges are written
            if (i >= g.n) continue;
            const int32_t s = g.R[i], e = g.R[i + 1];
            for (int32_t q = s + lane; q < e; q += 32) {
                const int j = g.C[q];
                if (j != i) d[j] = g.V ? __fdiv_rn(1.0f, g.V[q]) : 1.0f;
            }
        }
    }
    team.sync();
    Tile c;
    // the first diagonal blocks; the others are closed as soon as they are final
    for (int gi = a + vb; gi < b; gi += nvb) {
        const FWGraph g = p.gs[gi];
        float* d = blk(p.D, g, 0, 0);
        c.load(d, g.np);
        close_block(sm, c);
        c.store(d, g.np);
    }
    team.sync();
    // graphs [a, act) have more than kb blocks, [a, an) more than kb + 1
    const int rounds = p.gs[a].nb > 1 ? p.gs[a].nb : 0;
    int act = b, an = b;
    for (int kb = 0; kb < rounds; kb++) {
        while (act > a && p.gs[act - 1].nb <= kb) act--;
        while (an > a && p.gs[an - 1].nb <= kb + 1) an--;
        // 1: row and column panels
        const long long first = p.gs[a].panel0, panels = p.gs[act].panel0 - first;
        for (long long t = vb; t < panels; t += nvb) {
            const FWGraph g = p.gs[task_graph<&FWGraph::panel0>(p, a, act, first + t)];
            const int local = (int)(first + t - g.panel0), m = g.nb - 1;
            const bool row = local < m;
            int other = row ? local : local - m;
            if (other >= kb) other++;
            // rows and columns past n are padding
            close_panel(sm, c, blk(p.D, g, kb, kb), row ? blk(p.D, g, kb, other) : blk(p.D, g, other, kb), g.np, row,
                        min(B, g.n - kb * B));
        }
        team.sync();
        // 2: the other blocks, the next round's diagonal blocks first; then
        // the rest of their graphs' blocks, then those of graphs in their last round
        const long long inner = p.gs[a].inner0, n_inner = p.gs[an].inner0 - inner;
        const long long total = (an - a) + n_inner + (long long)(act - an) * kb * kb;
        for (long long t = vb; t < total; t += nvb) {
            int gi, local;
            const bool diagonal = t < an - a;
            long long x = t - (an - a);
            if (diagonal) {
                gi = a + (int)t;
                local = kb * p.gs[gi].nb;   // block (kb + 1, kb + 1) of the others
            } else if (x < n_inner) {
                gi = task_graph<&FWGraph::inner0>(p, a, an, inner + x);
                local = (int)(inner + x - p.gs[gi].inner0);
                local += local >= kb * p.gs[gi].nb;
            } else {
                x -= n_inner;
                gi = an + (int)(x / (kb * kb));
                local = (int)(x % (kb * kb));
            }
            const FWGraph g = p.gs[gi];
            const int m = g.nb - 1;
            int bi = local / m, bj = local % m;
            if (bi >= kb) bi++;
            if (bj >= kb) bj++;
            float* d = blk(p.D, g, bi, bj);
            c.load(d, g.np);
            min_plus(sm, c, blk(p.D, g, bi, kb), blk(p.D, g, kb, bj), g.np, min(B, g.n - kb * B));
            if (diagonal) close_block(sm, c);
            c.store(d, g.np);
        }
        team.sync();
    }
    // ---- C: row sums of 1/d over finite, non-tiny distances (CUBFW_Lp.cpp:77-83,99-104)
    const int end = p.gs[b].node0;
    int gi = a;
    for (long long x = (long long)p.gs[a].node0 + gw; x < end; x += nw) {
        gi = graph_at(p, gi, x);
        const FWGraph g = p.gs[gi];
        const int u = (int)x - g.node0;
        const float* row = p.D + g.off + (long long)u * g.np;
        double acc = 0.0;
        for (int v0 = lane; v0 < g.n; v0 += 128) {
            float d[4];
#pragma unroll
            for (int z = 0; z < 4; z++) d[z] = v0 + 32 * z < g.n ? row[v0 + 32 * z] : 0.0f;
#pragma unroll
            for (int z = 0; z < 4; z++)
                if (v0 + 32 * z != u && d[z] >= 0.1f) acc += 1.0 / (double)d[z];
        }
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            p.rowsum[x] = acc;
            float e = g.n > 1 ? (float)(acc / (double)(g.n - 1)) : 0.0f;
            if (e < 1.0f / (float)g.n) e = 0.0f;
            p.eff[g.out0 + u] = e;
        }
    }
}

__global__ void __launch_bounds__(FW_THREADS, 1) k_fw_batch(FwBatch p)
{
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) unsigned char fw_smem[];
    FwSmem& sm = ((FwSmem*)fw_smem)[threadIdx.x >> 7];
    const int grp = threadIdx.x >> 7, vb = grp * gridDim.x + blockIdx.x, nvb = GROUPS * gridDim.x;
    const int lane = group_thread() & 31;
    const long long gw = (long long)vb * (GT / 32) + (group_thread() >> 5), nw = (long long)nvb * (GT / 32);
    if (p.onnela) {
        // ---- weight maxima
        for (int gi = vb; gi < p.ng; gi += nvb) {
            const FWGraph g = p.gs[gi];
            const int32_t nnz = g.R[g.n];
            float m = -INFINITY;
#pragma unroll 4
            for (int32_t q = group_thread(); q < nnz; q += GT) m = fmaxf(m, g.V[q]);
            for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) sm.red[group_thread() >> 5] = m;
            group_sync();
            if (group_thread() == 0) {
                float t = -INFINITY;
                for (int w = 0; w < GT / 32; w++) t = fmaxf(t, (float)sm.red[w]);
                p.vmax[gi] = t;
            }
            group_sync();
        }
        grid.sync();
        // ---- per-entry cube roots of the normalised weights, a warp per node
        int gi = 0;
        for (long long x = gw; x < p.total_nodes; x += nw) {
            gi = graph_at(p, gi, x);
            const FWGraph g = p.gs[gi];
            const int i = (int)x - g.node0;
            const float vm = p.vmax[gi];
            const int32_t s = g.R[i], e = g.R[i + 1];
            int upto = 0;
            bool ascending = true;
            for (int32_t q = s + lane; q < e; q += 32) {
                const int j = g.C[q];
                upto += j <= i;
                ascending &= q == s || g.C[q - 1] < j;
                p.cw[g.edge0 + q] = cbrt((double)__fdiv_rn(g.V[q], vm));
            }
            upto = __reduce_add_sync(0xffffffffu, upto);
            if (!__all_sync(0xffffffffu, ascending)) upto = 0;   // any order: the whole row is scanned
            if (lane == 0) p.up[x] = s + upto;
        }
        grid.sync();
        // ---- Onnela, a group per node
        for (int q = group_thread(); q < ONNELA_MAX_N; q += GT) sm.row[q] = 0.0;
        gi = 0;
        for (;;) {
            group_sync();
            if (group_thread() == 0) sm.next = atomicAdd(&p.ctl->onnela_next, 1);
            group_sync();
            const int x = sm.next;
            if (x >= p.total_nodes) break;
            gi = graph_at(p, gi, x);
            const FWGraph g = p.gs[gi];
            onnela_node(p, g, x - g.node0, sm.row, sm.red);
        }
    }
    // ---- Floyd-Warshall by teams; CTAs of a team are neighbours
    {
        const int n_cta = gridDim.x, t = (int)((long long)blockIdx.x * p.teams / n_cta);
        const int first = (int)(((long long)t * n_cta + p.teams - 1) / p.teams);
        const int end = (int)(((long long)(t + 1) * n_cta + p.teams - 1) / p.teams);
        Team team{&p.ctl->arrived[t], &p.ctl->timeout, (unsigned)(end - first), 0u, p.max_spins,
                  p.hold && end - first > 1 && blockIdx.x == end - 1};
        __shared__ int s_bundle;
        for (;;) {
            if (blockIdx.x == first && threadIdx.x == 0) *(volatile int*)&p.ctl->bundle[t] = atomicAdd(&p.ctl->queue, 1);
            const int q = team.sync_bundle(&p.ctl->bundle[t], s_bundle);
            if (q < 0 || q >= p.bundles) break;
            fw_bundle(p, p.bundle0[q], p.bundle0[q + 1], team, sm, grp * (end - first) + (blockIdx.x - first),
                      GROUPS * (end - first));
        }
    }
    grid.sync();
    // ---- a warp per graph: sums over the nodes in order (reads 32 at a time)
    for (long long gi = gw; gi < p.ng; gi += nw) {
        const FWGraph g = p.gs[gi];
        double t = 0.0, m = 0.0;
        for (int u0 = 0; u0 < g.n; u0 += 32) {
            const bool in = u0 + lane < g.n;
            const double x = in ? p.rowsum[g.node0 + u0 + lane] : 0.0;
            const float y = in && p.onnela ? p.cp[g.out0 + u0 + lane] : 0.0f;
            const int cnt = min(32, g.n - u0);
            for (int k = 0; k < cnt; k++) {
                t += __shfl_sync(0xffffffffu, x, k);
                m += (double)__shfl_sync(0xffffffffu, y, k);
            }
        }
        if (lane == 0) {
            p.lp[g.index] = t > 0.0 ? 1.0 / (t / g.n / (g.n - 1)) : INFINITY;
            if (p.onnela) p.cp_mean[g.index] = g.n > 0 ? m / g.n : 0.0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) p.lp[p.ng] = p.ctl->timeout ? 1.0 : 0.0;
}

__global__ void k_fw_copy_out(const FWGraph* __restrict__ gs, const float* __restrict__ D, float* __restrict__ out)
{
    const FWGraph g = gs[0];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < (long long)g.n * g.n;
         q += (long long)gridDim.x * blockDim.x)
        out[q] = D[g.off + (q / g.n) * g.np + q % g.n];
}

}  // namespace

static pg_status fw_plan(pg_ctx* ctx, const pg_graph* const* graphs, int ng, bool onnela, FwBatch* P)
{
    std::vector<int> order(ng);
    std::iota(order.begin(), order.end(), 0);
    auto nb_of = [&](int i) { return std::max(1, (graphs[i]->n + B - 1) / B); };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return nb_of(x) > nb_of(y); });
    std::vector<FWGraph> tab((size_t)ng + 1);
    std::vector<int> out0(ng), blocks(ng);
    long long edges = 0, off = 0;
    int nodes = 0, nmax = 1;
    for (int i = 0; i < ng; i++) {
        out0[i] = nodes;
        nodes += graphs[i]->n;
    }
    nodes = 0;
    long long row0 = 0, panel0 = 0, inner0 = 0;
    for (int q = 0; q < ng; q++) {
        const pg_graph* g = graphs[order[q]];
        if (onnela && !g->V) return pg_fail(ctx, PG_ERR_INVALID, "Onnela clustering needs a weighted graph");
        const int nb = blocks[q] = nb_of(order[q]);
        tab[q] = {g->R, g->C, g->V, g->n, nb * B, nb, order[q], off, edges, nodes, out0[order[q]],
                  row0, panel0, inner0};
        row0 += nb * B;
        panel0 += 2LL * (nb - 1);
        inner0 += nb > 1 ? (long long)(nb - 1) * (nb - 1) - 1 : 0;
        off += (long long)nb * B * nb * B;
        nodes += g->n;
        edges += g->nnz;
        nmax = std::max(nmax, (int)g->n);
    }
    tab[ng].node0 = nodes;
    tab[ng].row0 = row0;
    tab[ng].panel0 = panel0;
    tab[ng].inner0 = inner0;
    if (onnela && nmax > ONNELA_MAX_N)
        return pg_fail(ctx, PG_ERR_TOO_LARGE, "Onnela in the batched launch: n=%d above %d", nmax, ONNELA_MAX_N);
    FwBatch& b = *P;
    memset(&b, 0, sizeof b);
    FWGraph* dtab;
    PG_TRY(pg_wst(ctx, "fw.D", (size_t)off, &b.D));
    // the bundles' first graphs lie behind the table: one upload
    const FwPlan plan = fw_batch_plan(blocks.data(), ng, ctx->sm_count, MAX_TEAMS);
    const size_t tab_bytes = sizeof(FWGraph) * ((size_t)ng + 1), cut_bytes = sizeof(int) * plan.bundle0.size();
    std::vector<unsigned char> blob(tab_bytes + cut_bytes);
    memcpy(blob.data(), tab.data(), tab_bytes);
    memcpy(blob.data() + tab_bytes, plan.bundle0.data(), cut_bytes);
    PG_TRY(pg_ws(ctx, "fw.tab", blob.size(), (void**)&dtab));
    PG_TRY(pg_wst(ctx, "fw.ctl", 1, &b.ctl));
    if (onnela) {
        PG_TRY(pg_wst(ctx, "fw.cw", (size_t)edges + 1, &b.cw));
        PG_TRY(pg_wst(ctx, "fw.up", (size_t)nodes + 1, &b.up));
        PG_TRY(pg_wst(ctx, "fw.vmax", (size_t)ng, &b.vmax));
        PG_TRY(pg_wst(ctx, "fw.cp", (size_t)nodes + 1, &b.cp));
        PG_TRY(pg_wst(ctx, "fw.cpm", (size_t)ng, &b.cp_mean));
    }
    PG_TRY(pg_wst(ctx, "fw.rows", (size_t)nodes + 1, &b.rowsum));
    PG_TRY(pg_wst(ctx, "fw.eff", (size_t)nodes + 1, &b.eff));
    PG_TRY(pg_wst(ctx, "fw.lp", (size_t)ng + 1, &b.lp));
    PG_TRY(pg_h2d(ctx, dtab, blob.data(), blob.size()));
    b.teams = plan.teams;
    b.bundles = (int)plan.bundle0.size() - 1;
    b.bundle0 = (const int*)((const unsigned char*)dtab + tab_bytes);
    b.gs = dtab;
    b.ng = ng;
    b.total_nodes = nodes;
    b.onnela = onnela;
    PG_CUDA(ctx, cudaFuncSetAttribute(k_fw_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(GROUPS * sizeof(FwSmem))));
    return PG_OK;
}

static pg_status fw_launch(pg_ctx* ctx, FwBatch b)
{
    // a pending failure-path test stall applies to this launch only (a read of
    // the counter takes about half a microsecond)
    b.hold = ctx->debug_team_stall_ns != 0;
    b.max_spins = b.hold ? (unsigned)std::min<unsigned long long>(ctx->debug_team_stall_ns / 500, MAX_SPINS) : MAX_SPINS;
    ctx->debug_team_stall_ns = 0;
    PG_CUDA(ctx, cudaMemsetAsync(b.ctl, 0, sizeof(FwControl), ctx->stream));
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctx->sm_count);
    cfg.blockDim = dim3(FW_THREADS);
    cfg.dynamicSmemBytes = GROUPS * sizeof(FwSmem);
    cfg.stream = ctx->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const int h = pg_prof_begin(ctx, "k_fw_batch");
    PG_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_fw_batch, b));
    PG_LAUNCHED(ctx);
    pg_prof_end(ctx, h);
    return PG_OK;
}

// The per-graph Lp (to lp, may be null) and the timeout mark behind them.
static pg_status fw_read_lp(pg_ctx* ctx, const FwBatch& b, double* lp)
{
    std::vector<double> h((size_t)b.ng + 1);
    PG_TRY(pg_d2h(ctx, h.data(), b.lp, sizeof(double) * h.size()));
    if (h[b.ng] != 0.0) return pg_fail(ctx, PG_ERR_TIMEOUT, "FW: a team barrier timed out");
    if (lp) std::copy(h.begin(), h.begin() + b.ng, lp);
    return PG_OK;
}

extern "C" pg_status pg_fw_paths(pg_ctx* ctx, const pg_graph* g, float* dist, float* eff, double* lp)
{
    if (!ctx || !g) return pg_fail(ctx, PG_ERR_INVALID, "pg_fw_paths: null argument");
    PG_CUDA(ctx, cudaSetDevice(ctx->device));
    const int n = g->n;
    const pg_graph* one[1] = {g};
    FwBatch b;
    PG_TRY(fw_plan(ctx, one, 1, false, &b));
    PG_TRY(fw_launch(ctx, b));
    PG_TRY(fw_read_lp(ctx, b, lp));
    if (dist) {
        float* tmp;
        PG_TRY(pg_wst(ctx, "fw.out", (size_t)n * n + 1, &tmp));
        k_fw_copy_out<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>(b.gs, b.D, tmp);
        PG_LAUNCHED(ctx);
        PG_TRY(pg_d2h_large(ctx, dist, tmp, sizeof(float) * (size_t)n * n));
    }
    if (eff) PG_TRY(pg_d2h(ctx, eff, b.eff, sizeof(float) * n));
    return PG_OK;
}

extern "C" pg_status pg_fw_batched(pg_ctx* ctx, const pg_graph* const* graphs, int32_t count, float* eff, double* lp,
                                   float* cp, double* cp_mean)
{
    if (!ctx || !graphs || count < 1) return pg_fail(ctx, PG_ERR_INVALID, "pg_fw_batched: bad arguments");
    PG_CUDA(ctx, cudaSetDevice(ctx->device));
    for (int i = 0; i < count; i++)
        if (!graphs[i]) return pg_fail(ctx, PG_ERR_INVALID, "graph %d is null", i);
    FwBatch b;
    PG_TRY(fw_plan(ctx, graphs, count, cp || cp_mean, &b));
    PG_TRY(fw_launch(ctx, b));
    PG_TRY(fw_read_lp(ctx, b, lp));
    if (eff) PG_TRY(pg_d2h(ctx, eff, b.eff, sizeof(float) * b.total_nodes));
    if (cp) PG_TRY(pg_d2h(ctx, cp, b.cp, sizeof(float) * b.total_nodes));
    if (cp_mean) PG_TRY(pg_d2h(ctx, cp_mean, b.cp_mean, sizeof(double) * count));
    return PG_OK;
}
