// gram_tc.cu -- split-BF16 Gram tiles on the 5th-generation tensor cores
// (tcgen05), fused with the threshold epilogue.  Replaces the reference's
// FP32 cublasSgemm tiles (U/CorMat/CUCorMat/CUCORMAT/CorMat.cu:93) and the
// host post-processing of every tile.
//
// z = hi + lo with hi = bf16(z), lo = bf16(z - hi).  Each 128x128 output tile
// accumulates, in FP32 inside TMEM,
//     D = Ahi*Bhi^T + Ahi*Blo^T + Alo*Bhi^T
// (the lo*lo term is below 2^-18 |z_i||z_j|).  Over K = T <= 256 the error
// of D against the exact dot product of the rounded z-scores stays below
// 1e-4, far inside the 2e-3 guard band that the FP64 recheck covers.
//
// Structure: one persistent CTA of 18 warps per SM over the upper-triangle
// tiles in row-major order, warp-specialised:
//   - warp 0 (one lane) streams K in 64-element chunks (128 B rows, 128B
//     swizzle) with TMA into a 3-stage shared-memory ring (A_hi, A_lo, B_hi,
//     B_lo per stage) guarded by full/empty mbarriers;
//   - warp 1 (one lane) issues 12 UMMA (M=128, N=128, K=16, bf16 x bf16 ->
//     fp32) per chunk into one of TWO TMEM accumulators (256 columns), a
//     tcgen05.commit releasing every stage and, per tile, the accumulator;
//   - warps 2-17 run the epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31
//     (rows), the four warps of a lane quarter 32 columns each, with
//     tcgen05.ld 32x32b.x32, classify every pair (histogram, decided edge,
//     FP64 band) in registers and hand the accumulator back (16 arrivals),
//     so the next tile's MMAs run while this tile's epilogue does.  The emit
//     pass only tests for candidates there and then handles the columns that
//     hold one (about ten of 32 at 1 %): branching on each of the 32 register
//     values and one list atomic per block made the pass take 5.3 ms at
//     58,000 voxels, 2.8 ms now (2.85 ms when nothing is kept, so the emission
//     costs nothing any more; the operands come from L2 at 9 TB/s, 26 GB per
//     pass, with the tensor pipe active 40 % of the time at 24,000 voxels).
// Every mbarrier wait is bounded by the global timer and gives up at once
// when another warp has given up; the kernel then records an error, waits
// (bounded) for its own MMAs and TMA copies, frees TMEM and returns.
#include "build_graph.cuh"
#include "tma.cuh"
#include <cuda.h>

namespace {
using namespace pg_tma;
constexpr int BM = 128, BN = 128, KC = 64;
constexpr int STAGES = 3;
constexpr int EPI_WARPS = 16;                   // four per TMEM lane quarter, 32 columns each
constexpr int WARPS = 2 + EPI_WARPS;
constexpr int THREADS = WARPS * 32;
constexpr uint32_t TILE_BYTES = BM * KC * 2;       // 16 KB per operand tile
constexpr uint32_t STAGE_BYTES = 4 * TILE_BYTES;   // A_hi, A_lo, B_hi, B_lo
constexpr uint32_t ACC_COLS = BN;                  // one FP32 accumulator
constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;       // double-buffered

struct Ctl {
    unsigned long long full[STAGES];
    unsigned long long empty[STAGES];
    unsigned long long tfull[2];
    unsigned long long tempty[2];
    unsigned long long drainbar;
    unsigned long long stallbar;   // test hook: nothing ever arrives on it
    long long issued, consumed;
    uint32_t tmem_base;
    int abort;
};

// A warp's part of an output list, gathered in shared memory and written out
// when it is nearly full: one atomic per flush instead of one per 32 x 32
// block on the list's counter (all atomics on one address are served one
// after the other), and coalesced stores.
constexpr int LIST_CAP = 80;   // a column adds at most 32
struct WarpList {
    int2* ij;
    float* r;
    int count;
    static constexpr size_t BYTES = LIST_CAP * (sizeof(int2) + sizeof(float));
    __device__ void init(unsigned char* base, int slot)
    {
        ij = (int2*)(base + (size_t)slot * BYTES);
        r = (float*)(ij + LIST_CAP);
        count = 0;
    }
    // all lanes: append (i, j, v) of the lanes in `who` (this lane: `mine`)
    __device__ void push(bool mine, unsigned who, int i, int j, float v, unsigned long long* counter, int2* out,
                         float* out_r, long long cap)
    {
        if (mine) {
            const int at = count + __popc(who & ((1u << (threadIdx.x & 31)) - 1u));
            ij[at] = make_int2(i, j);
            r[at] = v;
        }
        count += __popc(who);
        if (count > LIST_CAP - 32) flush(counter, out, out_r, cap);
    }
    __device__ void flush(unsigned long long* counter, int2* out, float* out_r, long long cap)
    {
        if (!count) return;
        __syncwarp();
        const int lane = threadIdx.x & 31;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)count);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int e = lane; e < count; e += 32) {
            const long long at = (long long)base + e;
            if (at < cap) {
                out[at] = ij[e];
                if (out_r) out_r[at] = r[e];
            }
        }
        __syncwarp();
        count = 0;
    }
};

constexpr size_t LIST_BYTES = 2 * EPI_WARPS * WarpList::BYTES;
static_assert(sizeof(Ctl) % 8 == 0, "the lists behind Ctl hold int2");
constexpr size_t smem_bytes(int mode)
{
    return 1024 /*align slack*/ + STAGES * STAGE_BYTES + sizeof(Ctl) + (mode == EPI_EMIT ? LIST_BYTES : 0);
}
static_assert(smem_bytes(EPI_EMIT) <= 227 * 1024 - 64, "shared memory of the emit pass");

// one column of this warp's 32 TMEM lanes
__device__ __forceinline__ uint32_t tmem_ld1(uint32_t taddr)
{
    uint32_t v;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    return v;
}

// Instruction descriptor, kind::f16: F32 accumulate, BF16 A and B, both
// K-major, N = 128, M = 128.
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void umma(uint32_t tmem_d, unsigned long long a, unsigned long long b, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(IDESC), "r"(acc));
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
k_gram_tc(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, int nb, int nk,
          EpiParams p, unsigned long long stall_ns, int* __restrict__ err)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ unsigned int sh_hist[MODE == EPI_HIST ? HIST_BINS : 1];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Ctl* ctl = (Ctl*)(smem + STAGES * STAGE_BYTES);
    volatile int* abort_flag = &ctl->abort;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;

    if (MODE == EPI_HIST)
        for (int b = t; b < HIST_BINS; b += THREADS) sh_hist[b] = 0;
    if (t == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&ctl->tfull[b], 1);
            mbar_init(&ctl->tempty[b], EPI_WARPS);
        }
        mbar_init(&ctl->drainbar, 1);
        mbar_init(&ctl->stallbar, 1);
        ctl->issued = 0;
        ctl->consumed = 0;
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;

    const long long nt = (long long)nb * (nb + 1) / 2;
    const long long first = (long long)blockIdx.x * (MODE == EPI_HIST ? p.tile_stride : 1);
    const long long stride = (MODE == EPI_HIST ? (long long)p.tile_stride : 1LL) * gridDim.x;
    unsigned int below = 0u, neg = 0u;

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            // failure-path test hook: wait on a barrier nothing arrives on,
            // before anything is issued
            if (stall_ns && !mbar_wait_abort(&ctl->stallbar, 0, abort_flag, stall_ns)) *abort_flag = 1;
            long long q = 0;
            for (long long L = first; L < nt && !*abort_flag; L += stride) {
                int bi, bj;
                tri_tile(L, nb, bi, bj);
                for (int c = 0; c < nk; c++) {
                    const int s = (int)(q % STAGES);
                    if (!mbar_wait_abort(&ctl->empty[s], (uint32_t)((q / STAGES) & 1) ^ 1u, abort_flag)) {
                        *abort_flag = 1;
                        break;
                    }
                    unsigned char* st = smem + (size_t)s * STAGE_BYTES;
                    mbar_expect_tx(&ctl->full[s], STAGE_BYTES);
                    tma_load(st, &map_hi, c * KC, bi * BM, &ctl->full[s]);
                    tma_load(st + TILE_BYTES, &map_lo, c * KC, bi * BM, &ctl->full[s]);
                    tma_load(st + 2 * TILE_BYTES, &map_hi, c * KC, bj * BN, &ctl->full[s]);
                    tma_load(st + 3 * TILE_BYTES, &map_lo, c * KC, bj * BN, &ctl->full[s]);
                    q++;
                    ctl->issued = q;
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            long long q = 0;
            int tl = 0;
            for (long long L = first; L < nt && !*abort_flag; L += stride, tl++) {
                const int buf = tl & 1;
                if (!mbar_wait_abort(&ctl->tempty[buf], (uint32_t)((tl >> 1) & 1) ^ 1u, abort_flag)) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t dst = tmem + (uint32_t)(buf * ACC_COLS);
                bool ok = true;
                for (int c = 0; c < nk; c++) {
                    const int s = (int)(q % STAGES);
                    if (!mbar_wait_abort(&ctl->full[s], (uint32_t)((q / STAGES) & 1), abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    unsigned char* st = smem + (size_t)s * STAGE_BYTES;
                    const unsigned long long ahi = sdesc(st), alo = sdesc(st + TILE_BYTES);
                    const unsigned long long bhi = sdesc(st + 2 * TILE_BYTES), blo = sdesc(st + 3 * TILE_BYTES);
#pragma unroll
                    for (int kk = 0; kk < KC / 16; kk++) {
                        const unsigned long long o = (unsigned long long)(kk * 32) >> 4;  // 32 B per K=16 step
                        umma(dst, ahi + o, bhi + o, (c | kk) != 0);
                        umma(dst, ahi + o, blo + o, 1u);
                        umma(dst, alo + o, bhi + o, 1u);
                    }
                    umma_commit(&ctl->empty[s]);
                    q++;
                    ctl->consumed = q;
                }
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                umma_commit(&ctl->tfull[buf]);
            }
        }
    } else {
        // ---- epilogue: row 32 (warp % 4) + lane of the tile; the warps of a
        // lane quarter share its 128 columns, 32 at a time
        const int quarter = warp & 3;
        const int part = (warp - 2) >> 2;               // 0 .. EPI_WARPS / 4 - 1
        constexpr int CHUNKS = (BN / 32) / (EPI_WARPS / 4);
        WarpList pair_list, band_list;
        if (MODE == EPI_EMIT) {
            unsigned char* lists = smem + STAGES * STAGE_BYTES + sizeof(Ctl);
            pair_list.init(lists, 2 * (warp - 2));
            band_list.init(lists, 2 * (warp - 2) + 1);
        }
        unsigned decided = 0u;
        int tl = 0;
        for (long long L = first; L < nt; L += stride, tl++) {
            int bi, bj;
            tri_tile(L, nb, bi, bj);
            const int buf = tl & 1;
            if (!mbar_wait_abort(&ctl->tfull[buf], (uint32_t)((tl >> 1) & 1), abort_flag)) {
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            const int i = bi * BM + quarter * 32 + lane;
            const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * ACC_COLS);
#pragma unroll 1
            for (int cb = part * CHUNKS; cb < (part + 1) * CHUNKS; cb++) {
                uint32_t r[32];
                tmem_ld32(src + (uint32_t)(cb * 32), r);
                const int j0 = bj * BN + cb * 32;
                if (MODE == EPI_HIST) {
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const int j = j0 + c;
                        if (i < j && j < p.N) epi_hist(__uint_as_float(r[c]), p, sh_hist, below, neg);
                    }
                } else {
                    // columns of this lane's row that may be kept: above the
                    // diagonal, inside the matrix, key at or above the band
                    const int below_diag = i - j0 + 1, inside = p.N - j0;
                    unsigned cand = 0u;
                    if (p.abs_mode) {
                        const float cut = fminf(p.lo_cut, p.edge_band);
#pragma unroll
                        for (int c = 0; c < 32; c++) cand |= (unsigned)(fabsf(__uint_as_float(r[c])) >= cut) << c;
                    } else {
                        const float cut = fminf(p.lo_cut, p.edge_band);
#pragma unroll
                        for (int c = 0; c < 32; c++) {
                            const float v = __uint_as_float(r[c]);
                            cand |= (unsigned)(v >= cut || v <= -p.edge_band) << c;
                        }
                    }
                    if (below_diag > 0) cand &= below_diag >= 32 ? 0u : ~0u << below_diag;
                    if (inside < 32) cand &= inside <= 0 ? 0u : (1u << inside) - 1u;
                    // column by column: a column's value is read once more from
                    // TMEM (registers cannot be indexed), its decided rows are
                    // one ballot
                    unsigned todo = __reduce_or_sync(0xffffffffu, cand), m1 = 0u, mt = 0u;
                    while (todo) {
                        const int q = __ffs(todo) - 1;
                        todo &= todo - 1u;
                        const float v = __uint_as_float(tmem_ld1(src + (uint32_t)(cb * 32 + q)));
                        const int cls = ((cand >> q) & 1u) ? epi_class(v, p) : 0;
                        const unsigned b1 = __ballot_sync(0xffffffffu, cls == 1), b2 = __ballot_sync(0xffffffffu, cls == 2);
                        if (b1) {
                            if (p.bits) {
                                m1 |= (unsigned)(cls == 1) << q;
                                if (lane == q) mt = b1;
                            } else {
                                pair_list.push(cls == 1, b1, i, j0 + q, epi_key(v, p.abs_mode), p.n_pairs, p.pairs,
                                               p.weighted ? p.pair_w : nullptr, p.cap_pairs);
                            }
                        }
                        if (b2) band_list.push(cls == 2, b2, i, j0 + q, v, p.n_band, p.band, p.band_r, p.cap_band);
                    }
                    if (p.bits) {
                        // row i, columns j0..; row j0 + lane, columns of this
                        // warp's rows: one word each (the same one on the diagonal)
                        decided += __popc(m1);
                        const int i0 = i - lane;
                        if (i0 == j0) {
                            m1 |= mt;
                            mt = 0u;
                        }
                        if (m1) p.bits[(size_t)i * p.bit_words + (j0 >> 5)] = m1;
                        if (mt) p.bits[(size_t)(j0 + lane) * p.bit_words + (i0 >> 5)] = mt;
                    }
                }
            }
            // the accumulator may be overwritten once every epilogue warp has read it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->tempty[buf]);
        }
        if (MODE == EPI_EMIT) {
            pair_list.flush(p.n_pairs, p.pairs, p.weighted ? p.pair_w : nullptr, p.cap_pairs);
            band_list.flush(p.n_band, p.band, p.band_r, p.cap_band);
            decided = __reduce_add_sync(0xffffffffu, decided);
            if (lane == 0 && decided) atomicAdd(p.n_pairs, (unsigned long long)decided);
        }
    }
    // the MMA thread waits (bounded) until its own MMAs have completed: TMEM
    // is freed below, whichever way the roles ended
    if (warp == 1 && lane == 0) {
        umma_commit(&ctl->drainbar);
        mbar_wait(&ctl->drainbar, 0);
    }
    __syncthreads();
    if (*abort_flag && t == 0) {
        atomicExch(err, 1);
        // the producer waits (bounded) for its copies still in flight
        for (long long q = ctl->consumed; q < ctl->issued; q++)
            if (!mbar_wait(&ctl->full[(int)(q % STAGES)], (uint32_t)((q / STAGES) & 1))) break;
    }
    if (MODE == EPI_HIST) {
        epi_hist_flush(below, neg, p);
        __syncthreads();
        for (int b = t; b < HIST_BINS; b += THREADS)
            if (sh_hist[b]) atomicAdd(&p.hist[b], sh_hist[b]);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

bool make_map(CUtensorMap* m, const __nv_bfloat16* base, int rows, int cols)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * sizeof(__nv_bfloat16)};
    cuuint32_t box[2] = {(cuuint32_t)KC, (cuuint32_t)BM};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

bool gram_tc_supported(pg_ctx* ctx, const ZOperands& z)
{
    (void)ctx;
    return encode_fn() != nullptr && z.Tp % KC == 0 && z.Np % BM == 0 && z.Tp >= KC;
}

pg_status launch_gram_tc(pg_ctx* ctx, const ZOperands& z, int mode, const EpiParams& p, int* err)
{
    CUtensorMap mhi, mlo;
    if (!make_map(&mhi, z.zhi, z.Np, z.Tp) || !make_map(&mlo, z.zlo, z.Np, z.Tp))
        return pg_fail(ctx, PG_ERR_CUDA, "cuTensorMapEncodeTiled failed for the split-BF16 operands");
    const int nb = z.Np / BM, nk = z.Tp / KC;
    const long long nt = (long long)nb * (nb + 1) / 2;
    long long grid = ctx->sm_count;
    if (grid > nt) grid = nt;
    // a pending failure-path test stall applies to this launch only
    const unsigned long long stall = ctx->debug_gram_stall_ns;
    ctx->debug_gram_stall_ns = 0;
    if (mode == EPI_HIST) {
        PG_CUDA(ctx, cudaFuncSetAttribute(k_gram_tc<EPI_HIST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem_bytes(EPI_HIST)));
        k_gram_tc<EPI_HIST><<<(int)grid, THREADS, smem_bytes(EPI_HIST), ctx->stream>>>(mhi, mlo, nb, nk, p, stall, err);
    } else {
        PG_CUDA(ctx, cudaFuncSetAttribute(k_gram_tc<EPI_EMIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem_bytes(EPI_EMIT)));
        k_gram_tc<EPI_EMIT><<<(int)grid, THREADS, smem_bytes(EPI_EMIT), ctx->stream>>>(mhi, mlo, nb, nk, p, stall, err);
    }
    PG_LAUNCHED(ctx);
    return PG_OK;
}
