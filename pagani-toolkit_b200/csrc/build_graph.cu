// build_graph.cu -- network construction (CUCorMat) on the device:
//   z-score (FP64) -> Gram tiles with fused threshold epilogue (a sampled
//   histogram and one full pass, or a histogram and an emit pass) -> FP64
//   recheck of the guard band -> exact k-th key selection (sparsity mode) ->
//   adjacency bits or undirected pairs -> sorted CSR.
// The dense correlation matrix is never stored.
#include "build_graph.cuh"
#include <cmath>
#include <cstring>
#include <algorithm>

// ------------------------------------------------------------------ z-score
// Restates the normalisation of CorMat_gpu (U/CorMat/CUCorMat/CUCORMAT/
// CorMat.cu:34-53) in FP64 with explicit round-to-nearest operations, so the
// result is bit-identical to the oracle (no contraction into FMA).
// A block takes 32 voxels.  Warps 1-7 read the samples, two chunks of 56 time
// points ahead in registers, and leave them in shared memory as the FP64
// terms of the sum; warp 0 adds them in order, one voxel per lane.  Where the
// voxels are few that chain of additions bounds it (8.7 cycles each), so
// nothing else is left in it; where they are many, the two reads of the
// series.  90 x 1200: 159 us when every lane loaded, converted and added its
// own samples, 26 us now; 58,000 x 240: 39 us both ways.
constexpr int ZT = 56, ZPROD = 7, ZROWS = (ZT + ZPROD - 1) / ZPROD;

__device__ __forceinline__ void z_fetch(float (&v)[ZROWS], const float* __restrict__ bold, int N, int T, int c, int i,
                                        int prod)
{
#pragma unroll
    for (int k = 0; k < ZROWS; k++) {
        const int r = prod + k * ZPROD, t = c * ZT + r;
        v[k] = (r < ZT && t < T && i < N) ? bold[(size_t)t * N + i] : 0.0f;
    }
}

template <bool SQUARES>
__device__ __forceinline__ void z_store(double (*buf)[32], const float (&v)[ZROWS], double mean, int lane, int prod)
{
#pragma unroll
    for (int k = 0; k < ZROWS; k++) {
        const int r = prod + k * ZPROD;
        if (r >= ZT) break;
        const double d = SQUARES ? __dsub_rn((double)v[k], mean) : (double)v[k];
        buf[r][lane] = SQUARES ? __dmul_rn(d, d) : d;
    }
}

// sum over t of x, or of (x - mean)^2, per lane of warp 0 (others return 0)
template <bool SQUARES>
__device__ __forceinline__ double z_sum(double (*buf)[ZT][32], const float* __restrict__ bold, int N, int T, int i,
                                        double mean)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, prod = warp - 1;
    const int nc = (T + ZT - 1) / ZT;
    float v0[ZROWS], v1[ZROWS];
    if (warp) {
        z_fetch(v0, bold, N, T, 0, i, prod);
        z_fetch(v1, bold, N, T, 1, i, prod);
        z_store<SQUARES>(buf[0], v0, mean, lane, prod);
    }
    __syncthreads();
    double s = 0.0;
    auto add = [&](int c) {
        const int cnt = min(ZT, T - c * ZT);
        if (cnt == ZT) {
#pragma unroll
            for (int r = 0; r < ZT; r++) s = __dadd_rn(s, buf[c & 1][r][lane]);
        } else {
            for (int r = 0; r < cnt; r++) s = __dadd_rn(s, buf[c & 1][r][lane]);
        }
    };
    // step c: chunk c is added while chunk c + 1 is stored and c + 2 is read
    for (int c = 0; c < nc; c += 2) {
        if (warp == 0) {
            add(c);
        } else {
            z_fetch(v0, bold, N, T, c + 2, i, prod);
            z_store<SQUARES>(buf[1], v1, mean, lane, prod);
        }
        __syncthreads();
        if (warp == 0) {
            if (c + 1 < nc) add(c + 1);
        } else {
            z_fetch(v1, bold, N, T, c + 3, i, prod);
            z_store<SQUARES>(buf[0], v0, mean, lane, prod);
        }
        __syncthreads();
    }
    return s;
}

__global__ void __launch_bounds__(32 * (1 + ZPROD), 5)
k_zstats(const float* __restrict__ bold, int N, int T, double* __restrict__ mu, double* __restrict__ sd,
         int* __restrict__ nzero)
{
    __shared__ double buf[2][ZT][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    const double s1 = __ddiv_rn(z_sum<false>(buf, bold, N, T, i, 0.0), (double)T);
    if (warp == 0) buf[1][0][lane] = s1;
    __syncthreads();
    const double mean = buf[1][0][lane];
    __syncthreads();
    const double s2 = __dsqrt_rn(z_sum<true>(buf, bold, N, T, i, mean));
    if (warp != 0) return;
    bool zero = false;
    if (i < N) {
        zero = !(s2 > 0.0) || isinf(s2) || isnan(s2);
        mu[i] = s1;
        sd[i] = zero ? 0.0 : s2;
    }
    const unsigned m = __ballot_sync(0xffffffffu, zero);
    if (lane == 0 && m) atomicAdd(nzero, __popc(m));
}

// 32x32 transposing tiles: reads bold[t][i] along i, writes z rows along t.
// Only the operands that the build needs are written (null: not needed).
__global__ void k_zwrite(const float* __restrict__ bold, int N, int T, int Ts, int Tp, const double* __restrict__ mu,
                         const double* __restrict__ sd, double* __restrict__ z64, float* __restrict__ z32,
                         __nv_bfloat16* __restrict__ zhi, __nv_bfloat16* __restrict__ zlo)
{
    __shared__ float tile[32][33];
    int t0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int t = t0 + r, i = i0 + threadIdx.x;
        tile[r][threadIdx.x] = (t < T && i < N) ? bold[(size_t)t * N + i] : 0.0f;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int i = i0 + r, t = t0 + threadIdx.x;
        if (t >= Tp) continue;
        double z = 0.0;
        if (i < N && t < T && sd[i] > 0.0) z = __ddiv_rn(__dsub_rn((double)tile[threadIdx.x][r], mu[i]), sd[i]);
        if (i < N && t < T) z64[(size_t)i * Ts + t] = z;
        float f = __double2float_rn(z);
        size_t o = (size_t)i * Tp + t;
        if (z32) z32[o] = f;
        if (zhi) {
            __nv_bfloat16 h = __float2bfloat16_rn(f);
            zhi[o] = h;
            zlo[o] = __float2bfloat16_rn(__fsub_rn(f, __bfloat162float(h)));
        }
    }
}

// --------------------------------------------------------- FP64 recheck
// r(i,j) exactly as the oracle: sequential t, one fused multiply-add per
// term; then the reference's range rule (post_block, CorMat.cpp:821 /
// W CorMat.cpp:821).  Key = r or |r|.  Rows start on 32-byte boundaries
// (stride Ts, a multiple of four), so a thread reads four samples of a row
// per load, eight such loads ahead of the sixteen additions they feed.
// KEEP: the compiler may not move the load towards its use.
template <bool KEEP>
__device__ __forceinline__ void load4(double (&x)[4], const double* p)
{
    if (KEEP)
        asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
                     : "l"(p));
    else
        asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p));
}

struct Samples16 {
    double x[4][4], y[4][4];
    template <bool KEEP>
    __device__ __forceinline__ void load(const double* a, const double* b)
    {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            load4<KEEP>(x[q], a + 4 * q);
            load4<KEEP>(y[q], b + 4 * q);
        }
    }
    __device__ __forceinline__ double add(double r) const
    {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int c = 0; c < 4; c++) r = __fma_rn(x[q][c], y[q][c], r);
        return r;
    }
};

// AHEAD: the next sixteen samples are loaded before the last sixteen are
// added (twice the registers): for lists too short to fill the GPU, where a
// pair is one chain of load latencies.
template <bool AHEAD>
__device__ __forceinline__ double dot_exact(const double* __restrict__ a, const double* __restrict__ b, int T)
{
    double r = 0.0;
    int t = 0;
    if (AHEAD && T >= 16) {
        Samples16 s0, s1;
        s0.load<true>(a, b);
        for (; t + 48 <= T; t += 32) {
            s1.load<true>(a + t + 16, b + t + 16);
            r = s0.add(r);
            s0.load<true>(a + t + 32, b + t + 32);
            r = s1.add(r);
        }
        r = s0.add(r);
        t += 16;
    }
    for (; t + 16 <= T; t += 16) {
        Samples16 s;
        s.load<false>(a + t, b + t);
        r = s.add(r);
    }
    for (; t + 4 <= T; t += 4) {
        double x[4], y[4];
        load4<false>(x, a + t);
        load4<false>(y, b + t);
#pragma unroll
        for (int c = 0; c < 4; c++) r = __fma_rn(x[c], y[c], r);
    }
    for (; t < T; t++) r = __fma_rn(a[t], b[t], r);
    return r;
}

__device__ __forceinline__ double range_rule(double r, int weighted)
{
    if (weighted) return (r > -1.0 - 1e-6 && r < 1.0 + 1e-6) ? r : 0.0;
    return (r >= -1.0 && r <= 1.0) ? r : 0.0;
}

// FP64 r of every band pair, and the error of the tile's r against it:
// err[0] = bits of max |r_tile - r| (non-negative doubles order as their
// bits), err[1] = sum of |r_tile - r| (r before the range rule).  With pair_w
// set, also the exact weight of every pair that the tiles decided (once per
// undirected pair: both directions have the same terms).  The lists are in
// tile order, so the pairs of a block share rows in L1; bound by those row
// reads.  58,000 voxels, top 1 %: 1.07 ms, 2.86 ms with one 8-byte load per
// term; the exact weights of 25,211 voxels (3.2M pairs, with
// 0.3M of the band) 1.02 ms, 3.2 ms when
// each of the 6.4M CSR entries was evaluated in row order.
template <bool AHEAD>
__global__ void __launch_bounds__(128, AHEAD ? 3 : 8)
k_pair_exact(const int2* __restrict__ band, const float* __restrict__ band_r, const int2* __restrict__ pairs,
             float* __restrict__ pair_w, const unsigned long long* __restrict__ counts, long long cap_pairs,
             long long cap_band, const double* __restrict__ z64, int T, int Ts, int weighted, int abs_mode,
             double* __restrict__ key64, unsigned long long* __restrict__ err)
{
    const long long nband = min((long long)counts[1], cap_band);
    const long long total = nband + (pair_w ? min((long long)counts[0], cap_pairs) : 0LL);
    double emax = 0.0, esum = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const bool in_band = q < nband;
        const int2 e = in_band ? band[q] : pairs[q - nband];
        double r = dot_exact<AHEAD>(z64 + (size_t)e.x * Ts, z64 + (size_t)e.y * Ts, T);
        if (in_band) {
            const double d = fabs((double)band_r[q] - r);
            emax = fmax(emax, d);
            esum += d;
        }
        r = range_rule(r, weighted);
        if (abs_mode) r = fabs(r);
        if (in_band) key64[q] = r;
        else pair_w[q - nband] = (float)r;
    }
    for (int o = 16; o; o >>= 1) {
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
        esum += __shfl_xor_sync(0xffffffffu, esum, o);
    }
    if ((threadIdx.x & 31) == 0 && esum > 0.0) {
        atomicMax(&err[0], (unsigned long long)__double_as_longlong(emax));
        atomicAdd((double*)&err[1], esum);
    }
}

// ----------------------------------------------------- radix selection
// One pass: a histogram of the next digit over the keys that match the prefix;
// the block that finishes last picks the digit of the m-th largest.  Once few
// enough keys match (`cap`), a pass also copies them to a list, and the passes
// after it read only that.  State lives on the device, so no pass needs the
// host.  129M keys: three full passes and three short ones, 0.57 ms (eight full
// ones of 8 bits, each with a launch of its own to pick, 1.8 ms); 1.9M keys 90
// us (130 us).
constexpr int SEL_BITS = 11, SEL_BINS = 1 << SEL_BITS, SEL_THREADS = 1024;

__global__ void __launch_bounds__(SEL_THREADS)
k_sel_pass(const unsigned long long* __restrict__ keys, long long n, SelState* __restrict__ st, int shift, int bits,
           unsigned long long* __restrict__ hist, unsigned long long* __restrict__ list, long long cap)
{
    __shared__ unsigned int h[SEL_BINS];
    __shared__ unsigned long long s_warp[SEL_THREADS / 32];
    __shared__ bool s_last;
    for (int b = threadIdx.x; b < SEL_BINS; b += SEL_THREADS) h[b] = 0u;
    __syncthreads();
    const unsigned long long prefix = st->prefix, mask = st->mask;
    const bool from_list = st->from_list, collect = !from_list && st->matching <= cap;
    const unsigned long long* src = from_list ? list : keys;
    const long long count = from_list ? st->listed : n;
    const unsigned digit = (1u << bits) - 1u;
    constexpr int U = 4;   // keys in flight per thread
    for (long long base = blockIdx.x * (long long)(U * SEL_THREADS); base < count;
         base += gridDim.x * (long long)(U * SEL_THREADS)) {
        unsigned long long k[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long q = base + u * SEL_THREADS + threadIdx.x;
            k[u] = q < count ? src[q] : ~prefix;   // past the end: matches no prefix once a digit is set
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool in = base + u * SEL_THREADS + threadIdx.x < count && (k[u] & mask) == prefix;
            const int bin = (int)((unsigned)(k[u] >> shift) & digit);
            const unsigned who = __ballot_sync(0xffffffffu, in);
            if (!who) continue;
            // the top digits of a warp's keys are often the same: one atomic then
            const int lead = __shfl_sync(0xffffffffu, bin, __ffs(who) - 1);
            if (__all_sync(0xffffffffu, !in || bin == lead)) {
                if ((threadIdx.x & 31) == 0) atomicAdd(&h[lead], (unsigned)__popc(who));
            } else if (in) {
                atomicAdd(&h[bin], 1u);
            }
            if (collect) {
                const long long s = warp_append((unsigned long long*)&st->listed, in);
                if (s >= 0 && s < cap) list[s] = k[u];
            }
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < SEL_BINS; b += SEL_THREADS)
        if (h[b]) atomicAdd(&hist[b], (unsigned long long)h[b]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->finished, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // thread t owns the t-th run of bins from the top
    constexpr int PER = SEL_BINS / SEL_THREADS;
    unsigned long long own[PER], sum = 0;
    const int top = SEL_BINS - 1 - (int)threadIdx.x * PER, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        own[k] = __ldcg(&hist[top - k]);
        hist[top - k] = 0ULL;
        sum += own[k];
    }
    unsigned long long x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    unsigned long long before = x - sum;
    for (int w = 0; w < warp; w++) before += s_warp[w];
    const unsigned long long m = (unsigned long long)st->m;
    __syncthreads();   // every thread has read m
    if (before < m && before + sum >= m) {
        int k = 0;
        while (before + own[k] < m) before += own[k++];
        st->prefix = prefix | (unsigned long long)(top - k) << shift;
        st->mask = mask | (unsigned long long)digit << shift;
        st->m = (long long)(m - before);
        st->matching = (long long)own[k];
    }
    if (threadIdx.x == 0) {
        st->finished = 0u;
        if (collect) st->from_list = 1;
    }
}

pg_status pg_radix_select(pg_ctx* ctx, const unsigned long long* keys, long long n, long long m, SelState* st_dev)
{
    long long cap = std::min(8LL << 20, n / 16 + 1024);
    const WsIdleAtExit<1> idle{ctx, {"sel.list"}};
    unsigned long long *hist, *list;
    PG_TRY(pg_wst(ctx, "sel.hist", SEL_BINS, &hist));
    if (pg_wst(ctx, "sel.list", (size_t)cap, &list) != PG_OK) {   // every pass reads all keys then
        cap = 0;
        list = nullptr;
    }
    SelState* init;
    PG_TRY(pg_hwst(ctx, "sel.init", 1, &init));
    *init = SelState{0ULL, 0ULL, m, n, 0LL, 0u, 0};
    PG_CUDA(ctx, cudaMemcpyAsync(st_dev, init, sizeof *init, cudaMemcpyHostToDevice, ctx->stream));
    PG_CUDA(ctx, cudaMemsetAsync(hist, 0, SEL_BINS * sizeof(unsigned long long), ctx->stream));
    // few blocks: each adds its bins to the global ones
    const int grid = std::max(1, std::min(ctx->sm_count * 2, ceil_div(n, 8 * SEL_THREADS)));
    for (int at = 64; at > 0;) {
        const int bits = std::min(at, SEL_BITS);
        at -= bits;
        k_sel_pass<<<grid, SEL_THREADS, 0, ctx->stream>>>(keys, n, st_dev, at, bits, hist, list, cap);
        PG_LAUNCHED(ctx);
    }
    return PG_OK;
}

// Band decision helpers.
__global__ void k_band_keys(const double* __restrict__ key64, long long n, unsigned long long* __restrict__ out)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x)
        out[q] = dkey(key64[q]);
}

// Lexicographic keys of the pairs tied with tau, complemented so that the
// radix selection of the "m-th largest" yields the m-th smallest (i, j).
__global__ void k_tie_keys(const int2* __restrict__ band, const unsigned long long* __restrict__ bkeys, long long n,
                           unsigned long long tau_key, int N, unsigned long long* __restrict__ out,
                           unsigned long long* __restrict__ ntie)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        if (bkeys[q] == tau_key) {
            unsigned long long s = atomicAdd(ntie, 1ULL);
            out[s] = ~((unsigned long long)band[q].x * (unsigned long long)N + (unsigned long long)band[q].y);
        }
    }
}

// Counters of one build in device memory, cleared at its start and read back
// with each host round trip.
struct BuildState {
    unsigned long long n_pairs;   // pairs decided by the Gram tiles
    unsigned long long n_band;    // pairs of the FP64 band
    unsigned long long n_wide;    // pairs listed between the sampled cuts
    unsigned long long n_added;   // band pairs that are edges (listed behind the decided ones)
    unsigned long long err_max;   // band error of the tiles: bits of the maximum, sum
    double err_sum;
    int zero;                     // zero-variance voxels
    int timeout;                  // a Gram pipeline wait ran out
};

// Adds the band pairs that are edges to the adjacency bits, or lists them
// behind the decided ones: key > tau, or key == tau and (i, j) <= tie_cut in
// lexicographic order.
__global__ void k_band_emit(const int2* __restrict__ band, const double* __restrict__ key64, long long cap_band,
                            double tau, int strict_only, unsigned long long tie_cut, int N, int weighted,
                            uint32_t* __restrict__ bits, int bit_words, int2* __restrict__ pairs,
                            float* __restrict__ w, BuildState* __restrict__ st, long long cap)
{
    const long long n = min((long long)st->n_band, cap_band), first = (long long)st->n_pairs;
    int added = 0;
    for (long long base = blockIdx.x * (long long)blockDim.x; base < n; base += (long long)gridDim.x * blockDim.x) {
        long long q = base + threadIdx.x;
        bool in = false;
        int2 e = make_int2(0, 0);
        double k = 0.0;
        if (q < n) {
            e = band[q];
            k = key64[q];
            if (k > tau) in = true;
            else if (!strict_only && k == tau)
                in = ((unsigned long long)e.x * (unsigned long long)N + (unsigned long long)e.y) <= tie_cut;
        }
        if (bits) {
            if (in) {
                atomicOr(&bits[(size_t)e.x * bit_words + (e.y >> 5)], 1u << (e.y & 31));
                atomicOr(&bits[(size_t)e.y * bit_words + (e.x >> 5)], 1u << (e.x & 31));
                added++;
            }
            continue;
        }
        long long s = warp_append(&st->n_added, in);
        if (s >= 0 && first + s < cap) {
            pairs[first + s] = e;
            if (weighted) w[first + s] = (float)k;
        }
    }
    added = __reduce_add_sync(0xffffffffu, added);
    if ((threadIdx.x & 31) == 0 && added) atomicAdd(&st->n_added, (unsigned long long)added);
}

// ------------------------------------------- adjacency bits -> CSR
// Rows of the bit matrix in column order are the sorted CSR rows: one pass
// counts them (a warp per row, 16 bytes per lane), one writes the columns.
// Bound by the two reads of the bits: 58,000 nodes / 33.6M entries 340 us for
// both, against 1.05 ms for degrees, scatter and row sort of a pair list.
__global__ void __launch_bounds__(256)
k_bits_count(const uint32_t* __restrict__ bits, int words, int n, int32_t* __restrict__ cnt)
{
    const int lane = threadIdx.x & 31, quads = words >> 2;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = gw; i < n; i += nw) {
        const uint4* row = (const uint4*)(bits + (size_t)i * words);
        int c = 0;
#pragma unroll 4
        for (int q = lane; q < quads; q += 32) {
            const uint4 m = row[q];
            c += __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) cnt[i] = c;
    }
}

__global__ void __launch_bounds__(256)
k_bits_csr(const uint32_t* __restrict__ bits, int words, int n, const int32_t* __restrict__ R, int32_t* __restrict__ C,
           long long nnz)
{
    const int lane = threadIdx.x & 31, quads = words >> 2;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = gw; i < n; i += nw) {
        const uint4* row = (const uint4*)(bits + (size_t)i * words);
        long long base = R[i];
        for (int q0 = 0; q0 < quads; q0 += 128) {
            uint4 v[4];   // four reads in flight
#pragma unroll
            for (int z = 0; z < 4; z++) {
                const int q = q0 + 32 * z + lane;
                v[z] = q < quads ? row[q] : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int z = 0; z < 4; z++) {
                const unsigned long long m[2] = {v[z].x | ((unsigned long long)v[z].y << 32),
                                                 v[z].z | ((unsigned long long)v[z].w << 32)};
                const int c = __popcll(m[0]) + __popcll(m[1]);
                int x = c;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                long long at = base + x - c;
#pragma unroll
                for (int k = 0; k < 2; k++)
                    for (unsigned long long b = m[k]; b; b &= b - 1ULL, at++)
                        if (at < nnz) C[at] = ((q0 + 32 * z + lane) << 7) + (k << 6) + __ffsll((long long)b) - 1;
                base += __shfl_sync(0xffffffffu, x, 31);
            }
        }
    }
}

static pg_status csr_from_bits(pg_ctx* ctx, int n, const uint32_t* bits, int words, long long n_edges, pg_graph** out)
{
    int32_t* cnt;
    PG_TRY(pg_wst(ctx, "csr.cnt", (size_t)n + 1, &cnt));
    const int grid = std::min(ctx->sm_count * 8, ceil_div(n, 8));
    k_bits_count<<<grid, 256, 0, ctx->stream>>>(bits, words, n, cnt);
    PG_LAUNCHED(ctx);
    pg_graph* g;
    PG_TRY(pg_graph_alloc(ctx, n, 2 * n_edges, false, &g));
    if (pg_status st = pg_row_offsets(ctx, cnt, n, g->R); st != PG_OK) {
        pg_graph_free(g);
        return st;
    }
    if (n_edges > 0) {
        k_bits_csr<<<grid, 256, 0, ctx->stream>>>(bits, words, n, g->R, g->C, g->nnz);
        if (pg_status st = [&]() -> pg_status { PG_LAUNCHED(ctx); return PG_OK; }(); st != PG_OK) {
            pg_graph_free(g);
            return st;
        }
    }
    *out = g;
    return PG_OK;
}

// ------------------------------------------------------------- driver
// Operands of one subject on the context stream (nothing is waited for).
// zero_dev counts the zero-variance voxels; the caller has cleared it.
enum : int { OPS_FP32 = 1, OPS_BF16 = 2 };   // z64 with z32, with zhi and zlo
static pg_status prepare_operands(pg_ctx* ctx, const float* bold, int N, int T, bool on_device, int ops, ZOperands& z,
                                  int* zero_dev)
{
    z.N = N;
    z.T = T;
    z.Ts = (T + 3) / 4 * 4;
    z.Np = (N + 127) / 128 * 128;
    z.Tp = (T + 63) / 64 * 64;
    z.z32 = nullptr;
    z.zhi = z.zlo = nullptr;
    const float* dbold = bold;
    if (!on_device) {
        float* tmp;
        PG_TRY(pg_wst(ctx, "bold", (size_t)N * T, &tmp));
        PG_CUDA(ctx, cudaMemcpyAsync(tmp, bold, sizeof(float) * (size_t)N * T, cudaMemcpyHostToDevice, ctx->stream));
        dbold = tmp;
    }
    double *mu, *sd;
    PG_TRY(pg_wst(ctx, "z.mu", (size_t)N, &mu));
    PG_TRY(pg_wst(ctx, "z.sd", (size_t)N, &sd));
    PG_TRY(pg_wst(ctx, "z.z64", (size_t)N * z.Ts, &z.z64));
    if (ops == OPS_FP32) PG_TRY(pg_wst(ctx, "z.z32", (size_t)z.Np * z.Tp, &z.z32));
    if (ops == OPS_BF16) {
        PG_TRY(pg_wst(ctx, "z.zhi", (size_t)z.Np * z.Tp, &z.zhi));
        PG_TRY(pg_wst(ctx, "z.zlo", (size_t)z.Np * z.Tp, &z.zlo));
    }
    k_zstats<<<ceil_div(N, 32), 32 * (1 + ZPROD), 0, ctx->stream>>>(dbold, N, T, mu, sd, zero_dev);
    PG_LAUNCHED(ctx);
    dim3 g(ceil_div(z.Tp, 32), ceil_div(z.Np, 32));
    k_zwrite<<<g, dim3(32, 8), 0, ctx->stream>>>(dbold, N, T, z.Ts, z.Tp, mu, sd, z.z64, z.z32, z.zhi, z.zlo);
    PG_LAUNCHED(ctx);
    return PG_OK;
}

pg_status pg_zstats(pg_ctx* ctx, const float* dbold, int N, int T, double* mu, double* sd, int* nz)
{
    PG_CUDA(ctx, cudaMemsetAsync(nz, 0, sizeof(int), ctx->stream));
    k_zstats<<<ceil_div(N, 32), 32 * (1 + ZPROD), 0, ctx->stream>>>(dbold, N, T, mu, sd, nz);
    PG_LAUNCHED(ctx);
    return PG_OK;
}

extern "C" void pg_build_opts_default(pg_build_opts* o)
{
    if (!o) return;
    memset(o, 0, sizeof *o);
    o->mode = PG_THRESH_R;
    o->value = 0.3;
    o->sign = PG_SIGNED;
    o->precision = PG_SPLIT_BF16;
    o->weighted = 0;
    o->guard = 2e-3;
    o->input_on_device = 0;
    o->exact_weights = 1;
}

// Histogram of the listed keys (bins of p, keys below p.kmin left out).
__global__ void __launch_bounds__(256)
k_wide_hist(const float* __restrict__ r, const unsigned long long* __restrict__ count, long long cap, EpiParams p)
{
    __shared__ unsigned int h[HIST_BINS];
    for (int b = threadIdx.x; b < HIST_BINS; b += 256) h[b] = 0u;
    __syncthreads();
    const long long n = min((long long)*count, cap);
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < n; q += gridDim.x * 256LL) {
        const float k = epi_key(r[q], p.abs_mode);
        if (!(k < p.kmin)) atomicAdd(&h[epi_bin(k, p)], 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < HIST_BINS; b += 256)
        if (h[b]) atomicAdd(&p.hist[b], h[b]);
}

// Splits the list between the sampled cuts by the final ones: decided edges
// (bits or list), band, dropped.  Eight entries per thread, one atomic per
// block and output for 2048 entries.
__global__ void __launch_bounds__(256)
k_wide_split(const int2* __restrict__ ij, const float* __restrict__ r, const unsigned long long* __restrict__ count,
             long long cap, EpiParams p)
{
    constexpr int U = 8;
    __shared__ unsigned int s_warp[8];
    __shared__ unsigned long long s_base[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n = min((long long)*count, cap);
    for (long long c0 = blockIdx.x * 256LL * U; c0 < n; c0 += gridDim.x * 256LL * U) {
        float v[U];
        int cls[U];
        unsigned int mine = 0u;   // decided in the low half, band in the high half
#pragma unroll
        for (int k = 0; k < U; k++) {
            const long long q = c0 + k * 256 + threadIdx.x;
            v[k] = q < n ? r[q] : 0.0f;
            cls[k] = q < n ? epi_class(v[k], p) : 0;
            mine += cls[k] == 1 ? 1u : cls[k] == 2 ? 0x10000u : 0u;
        }
        unsigned int x = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        unsigned int before = x - mine, total = 0u;
        for (int w = 0; w < 8; w++) {
            if (w < warp) before += s_warp[w];
            total += s_warp[w];
        }
        if (threadIdx.x < 2) {
            const unsigned int c = threadIdx.x ? total >> 16 : total & 0xffffu;
            s_base[threadIdx.x] = c ? atomicAdd(threadIdx.x ? p.n_band : p.n_pairs, (unsigned long long)c) : 0ULL;
        }
        __syncthreads();
        long long s1 = (long long)s_base[0] + (before & 0xffffu), s2 = (long long)s_base[1] + (before >> 16);
#pragma unroll
        for (int k = 0; k < U; k++) {
            if (!cls[k]) continue;
            const int2 e = ij[c0 + k * 256 + threadIdx.x];
            if (cls[k] == 2) {
                if (s2 < p.cap_band) {
                    p.band[s2] = e;
                    p.band_r[s2] = v[k];
                }
                s2++;
            } else if (p.bits) {
                atomicOr(&p.bits[(size_t)e.x * p.bit_words + (e.y >> 5)], 1u << (e.y & 31));
                atomicOr(&p.bits[(size_t)e.y * p.bit_words + (e.x >> 5)], 1u << (e.x & 31));
            } else {
                if (s1 < p.cap_pairs) {
                    p.pairs[s1] = e;
                    if (p.weighted) p.pair_w[s1] = epi_key(v[k], p.abs_mode);
                }
                s1++;
            }
        }
        __syncthreads();   // s_warp and s_base are reused
    }
}

static pg_status run_gram(pg_ctx* ctx, const ZOperands& z, int precision, int mode, const EpiParams& p, int* err_dev)
{
    if (precision == PG_SPLIT_BF16 && gram_tc_supported(ctx, z)) return launch_gram_tc(ctx, z, mode, p, err_dev);
    if (precision == PG_SPLIT_BF16)
        return pg_fail(ctx, PG_ERR_INVALID, "split-BF16 Gram unavailable for N=%d T=%d", z.N, z.T);
    return launch_gram_simt(ctx, z, mode, p);
}

// r mode: up to this many pairs the lists are simply sized for all of them
// (28 bytes each, 120 MB); above, a histogram pass of the Gram sizes them.
// At 2,896 nodes that pass and its host round trip cost 60 us of a 300 us
// build; at 58,000 nodes lists for every pair would take 47 GB.
constexpr long long LIST_ALL_PAIRS = 1LL << 22;

// lean: the route that needs least memory, lists sized by a full histogram.
static pg_status build_graph(pg_ctx* ctx, const float* bold, int N, int T, const pg_build_opts& o, bool lean,
                             pg_graph** out, pg_build_info* info)
{
    if (!(o.guard >= 0.0) || o.guard > 0.5) return pg_fail(ctx, PG_ERR_INVALID, "guard %g out of range", o.guard);
    if (o.mode != PG_THRESH_R && o.mode != PG_THRESH_SPARSITY)
        return pg_fail(ctx, PG_ERR_INVALID, "unknown threshold mode %d", o.mode);
    PG_CUDA(ctx, cudaSetDevice(ctx->device));
    *out = nullptr;
    // up to N^2 / 8 bytes of adjacency bits and the lists: for this call
    const WsIdleAtExit<8> idle{ctx, {"b.bits", "b.wide", "b.wide_r", "b.band", "b.band_r", "b.key64", "b.pairs", "b.pw"}};
    pg_build_info inf;
    memset(&inf, 0, sizeof inf);
    const long long M1 = (long long)N * (N - 1) / 2;
    cudaEvent_t* ev = ctx->ev;
    PG_CUDA(ctx, cudaEventRecord(ev[0], ctx->stream));

    BuildState *ds, *hs;
    unsigned char *hist_dev, *hist_host;   // the two "below" counters, then the bins
    constexpr size_t HIST_BYTES = 2 * sizeof(unsigned long long) + HIST_BINS * sizeof(unsigned int);
    PG_TRY(pg_wst(ctx, "b.state", 1, &ds));
    PG_TRY(pg_hwst(ctx, "b.state", 1, &hs));
    PG_TRY(pg_wst(ctx, "b.hist", HIST_BYTES, &hist_dev));
    PG_TRY(pg_hwst(ctx, "b.hist", HIST_BYTES, &hist_host));
    PG_CUDA(ctx, cudaMemsetAsync(ds, 0, sizeof *ds, ctx->stream));
    // reads the counters (and waits for everything before them)
    auto read_state = [&]() -> pg_status {
        PG_CUDA(ctx, cudaMemcpyAsync(hs, ds, sizeof *ds, cudaMemcpyDeviceToHost, ctx->stream));
        PG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (hs->timeout) return pg_fail(ctx, PG_ERR_TIMEOUT, "tcgen05 Gram: a pipeline wait timed out");
        return PG_OK;
    };

    ZOperands z;
    PG_TRY(prepare_operands(ctx, bold, N, T, o.input_on_device != 0, o.precision == PG_SPLIT_BF16 ? OPS_BF16 : OPS_FP32,
                            z, &ds->zero));
    PG_CUDA(ctx, cudaEventRecord(ev[1], ctx->stream));

    // ---- histogram pass(es): only keys >= kmin are binned, the rest counted
    EpiParams p;
    memset(&p, 0, sizeof p);
    p.N = N;
    p.abs_mode = o.sign == PG_ABS;
    const int weighted = o.weighted != 0;
    const bool exact_w = weighted && o.exact_weights;   // else the tile's r is the weight
    p.weighted = weighted && !exact_w;
    p.tile_stride = 1;
    const double g = o.guard;
    const float key_lo = p.abs_mode ? 0.0f : -1.0f;
    const float edge_band = (float)(1.0 - g);
    p.edge_band = (g == 0.0 && o.mode == PG_THRESH_R) ? INFINITY : edge_band;
    p.below = (unsigned long long*)hist_dev;
    p.hist = (unsigned int*)(hist_dev + 2 * sizeof(unsigned long long));
    const unsigned long long* hbelow = (const unsigned long long*)hist_host;
    const unsigned int* h = (const unsigned int*)(hist_host + 2 * sizeof(unsigned long long));
    auto set_bins = [&](float kmin) {
        p.kmin = kmin;
        p.scale = (float)HIST_BINS / (1.0f - kmin);
    };
    auto hist_pass = [&](float kmin, int stride) -> pg_status {
        set_bins(kmin);
        p.tile_stride = stride;
        PG_CUDA(ctx, cudaMemsetAsync(hist_dev, 0, HIST_BYTES, ctx->stream));
        if (M1 > 0) PG_TRY(run_gram(ctx, z, o.precision, EPI_HIST, p, &ds->timeout));
        PG_CUDA(ctx, cudaMemcpyAsync(hist_host, hist_dev, HIST_BYTES, cudaMemcpyDeviceToHost, ctx->stream));
        PG_TRY(read_state());
        p.tile_stride = 1;
        return PG_OK;
    };
    auto bin_of = [&](float key) {
        float x = (key - p.kmin) * p.scale;
        int b = (int)x;
        if (!(x >= 0.0f)) b = 0;
        return std::min(b, HIST_BINS - 1);
    };
    auto hist_total = [&]() {
        long long s = 0;
        for (int b = 0; b < HIST_BINS; b++) s += h[b];
        return s;
    };
    const bool list_all = !lean && o.mode == PG_THRESH_R && M1 <= LIST_ALL_PAIRS;
    const bool no_band = g == 0.0 && o.mode == PG_THRESH_R;
    const long long ntiles = (long long)(z.Np / 128) * (z.Np / 128 + 1) / 2;
    const int bit_words = z.Np / 32;
    const size_t bit_bytes = (size_t)N * bit_words * sizeof(uint32_t);
    long long k_edges = -1;  // sparsity: wanted edges
    float lo_cut, hi_cut;
    long long cap_pairs = 0, cap_band = 0, cap_total = 0;
    bool use_bits = false;
    int2 *pairs = nullptr, *band = nullptr;
    float* pw = nullptr;
    float* band_r = nullptr;
    double* key64 = nullptr;
    uint32_t* bits = nullptr;

    // Decided edges of a binary graph go into adjacency bits where about four
    // passes over N^2 bits (0.45 ms at 58,000 nodes) beat the list's degree
    // count, scatter and sort (62 us per million edges): from 1.3e-3 N^2 edges
    // on, and always where every pair would be listed (at most 1 MB of bits).
    // Weights need the list; the bits may take 8 GiB, and where they cannot be
    // had the (then smaller) list serves.
    auto bits_pay = [&](long long edges) {
        return !lean && !weighted && bit_bytes <= (8ULL << 30) &&
               (list_all || (double)edges >= 1.3e-3 * (double)N * (double)N) &&
               pg_wst(ctx, "b.bits", (size_t)N * bit_words, &bits) == PG_OK;
    };
    // room for the decided edges (cap_total with the band's)
    auto prepare_decided = [&]() -> pg_status {
        bits = nullptr;
        pairs = nullptr;
        if (use_bits) {
            PG_TRY(pg_wst(ctx, "b.bits", (size_t)N * bit_words, &bits));
            PG_CUDA(ctx, cudaMemsetAsync(bits, 0, bit_bytes, ctx->stream));
        } else {
            PG_TRY(pg_wst(ctx, "b.pairs", (size_t)std::max(1LL, cap_total), &pairs));
        }
        if (weighted) PG_TRY(pg_wst(ctx, "b.pw", (size_t)std::max(1LL, cap_total), &pw));
        p.bits = bits;
        p.bit_words = bit_words;
        p.pairs = pairs;
        p.pair_w = pw;
        p.n_pairs = &ds->n_pairs;
        p.cap_pairs = cap_pairs;
        return PG_OK;
    };
    auto prepare_band = [&]() -> pg_status {
        PG_TRY(pg_wst(ctx, "b.band", (size_t)std::max(1LL, cap_band), &band));
        PG_TRY(pg_wst(ctx, "b.band_r", (size_t)std::max(1LL, cap_band), &band_r));
        PG_TRY(pg_wst(ctx, "b.key64", (size_t)std::max(1LL, cap_band), &key64));
        p.band = band;
        p.band_r = band_r;
        p.n_band = &ds->n_band;
        p.cap_band = cap_band;
        return PG_OK;
    };
    // the sparsity cuts that follow from the histogram bin of the k-th key
    auto cuts_of_bin = [&](int bk) {
        const double lo_b = p.kmin + (double)bk / p.scale, hi_b = p.kmin + (double)(bk + 1) / p.scale;
        lo_cut = (float)(lo_b - g - 1.0 / p.scale);
        hi_cut = (float)(hi_b + g + 1.0 / p.scale);
    };

    if (o.mode == PG_THRESH_SPARSITY) {
        if (!(o.value >= 0.0) || o.value > 100.0)
            return pg_fail(ctx, PG_ERR_INVALID, "sparsity %g%% out of range", o.value);
        k_edges = pg_sparsity_edges(N, (float)o.value);
        if (k_edges > M1) k_edges = M1;
    } else {
        lo_cut = (float)(o.value - g);
        hi_cut = (float)(o.value + g);
        if (g == 0.0) lo_cut = hi_cut = nextafterf((float)o.value, INFINITY);  // tile decides alone: key > value
    }
    const float r_floor = std::max(key_lo, std::min(o.mode == PG_THRESH_R ? lo_cut : 0.0f, edge_band) - 1e-3f);

    // ---- Large problems: a histogram of every 8th tile, then ONE full Gram
    // pass.  r mode takes the sizes of its lists from the sample.  Sparsity
    // mode takes two cuts from it that enclose the final band with 5 % of the
    // wanted edges (and four standard deviations) to spare: pairs above are
    // decided, pairs between go to a list, and the list's histogram places the
    // k-th key in the same bin that a full histogram pass would.  Where the
    // sample misled (a list overflows, or the k-th key or its band lies
    // outside the cuts) the full histogram below decides, as for small
    // problems.  58,000 voxels: the second full pass cost 2.3 of 7.9 ms; below
    // two sampled tiles per SM it costs no more than the sample.
    float floor_key = key_lo;
    bool one_pass = false;
    const bool sampled = !list_all && (o.mode == PG_THRESH_R ? !lean : k_edges > 0) && ntiles >= 16LL * ctx->sm_count;
    if (sampled) {
        PG_TRY(hist_pass(o.mode == PG_THRESH_R ? r_floor : key_lo, 8));
        const double f = (double)(hist_total() + (o.mode == PG_THRESH_R ? (long long)hbelow[0] : 0)) / (double)M1;
        const int be = bin_of(edge_band);
        auto room = [&](double n) { return std::min(M1, (long long)(1.3 * n / f) + 65536); };
        double n_above = 0.0, n_list = (double)hbelow[1];   // sampled pairs above the cuts and between them
        bool fits = f > 0.0;
        if (o.mode == PG_THRESH_R) {
            const int bh = bin_of(hi_cut), bl = bin_of(lo_cut);
            for (int b = 0; b < HIST_BINS; b++) {
                if (b >= bh) n_above += h[b];
                if ((b >= bl && b <= bh) || b >= be) n_list += h[b];
            }
            fits = fits && lo_cut >= p.kmin;
        } else {
            const double ks = (double)k_edges * f, slack = 0.05 * ks + 4.0 * std::sqrt(ks) + 16.0;
            const double want = 2.0 * ks + 1024.0;
            long long acc = 0;
            int b_hi = -1, b_lo = -1, bf = 0;
            for (int b = HIST_BINS - 1; b >= 0; b--) {
                acc += h[b];
                if (b_hi < 0 && (double)acc >= ks - slack) b_hi = b;
                if (b_lo < 0 && (double)acc >= ks + slack) b_lo = b;
                if ((double)acc >= want) { bf = b; break; }
            }
            const double s_min = p.kmin, s_scale = p.scale;
            // floor of the binned range, with room for twice the wanted edges
            if (ntiles >= 64LL * ctx->sm_count)
                floor_key = (float)std::max((double)key_lo, s_min + (double)bf / s_scale - g - 4.0 / s_scale);
            set_bins(floor_key);
            hi_cut = (float)(s_min + (b_hi + 1) / s_scale + g + 3.0 / p.scale);
            lo_cut = (float)(s_min + b_lo / s_scale - g - 3.0 / p.scale);
            fits = fits && ks > slack && b_lo >= 0 && lo_cut > p.kmin && lo_cut > key_lo && hi_cut < edge_band;
            for (int b = b_lo < 0 ? 0 : b_lo; b < HIST_BINS; b++) {
                const double key = s_min + (b + 1) / s_scale;   // upper edge of the sampled bin
                if (key > hi_cut) n_above += h[b];
                else n_list += h[b];
                if (b >= be) n_list += h[b];
            }
            n_list *= 1.25;   // the bins that the cuts divide
        }
        cap_pairs = room(n_above);
        cap_band = no_band ? 0 : room(n_list);
        cap_total = cap_pairs + cap_band;
        if (fits && !lean && cap_pairs <= (long long)INT32_MAX) {   // lean: the sample places the floor only
            use_bits = bits_pay(k_edges >= 0 ? k_edges : cap_pairs);
            if (use_bits) cap_pairs = cap_total = M1;
            PG_CUDA(ctx, cudaEventRecord(ev[2], ctx->stream));
            PG_TRY(prepare_decided());
            PG_TRY(prepare_band());
            p.lo_cut = lo_cut;
            p.hi_cut = hi_cut;
            if (o.mode == PG_THRESH_R) {
                PG_TRY(run_gram(ctx, z, o.precision, EPI_EMIT, p, &ds->timeout));
                PG_TRY(read_state());
                one_pass = (long long)hs->n_pairs <= cap_pairs && (long long)hs->n_band <= cap_band;
            } else {
                int2* wide;
                float* wide_r;
                PG_TRY(pg_wst(ctx, "b.wide", (size_t)cap_band, &wide));
                PG_TRY(pg_wst(ctx, "b.wide_r", (size_t)cap_band, &wide_r));
                p.band = wide;
                p.band_r = wide_r;
                p.n_band = &ds->n_wide;
                PG_TRY(run_gram(ctx, z, o.precision, EPI_EMIT, p, &ds->timeout));
                PG_CUDA(ctx, cudaMemsetAsync(hist_dev, 0, HIST_BYTES, ctx->stream));
                k_wide_hist<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>(wide_r, &ds->n_wide, cap_band, p);
                PG_LAUNCHED(ctx);
                PG_CUDA(ctx, cudaMemcpyAsync(hist_host, hist_dev, HIST_BYTES, cudaMemcpyDeviceToHost, ctx->stream));
                PG_TRY(read_state());
                // every key at or above a bin below bin(hi_cut) and above
                // bin(lo_cut) has been decided or listed
                const float w_lo = lo_cut, w_hi = hi_cut;
                const int top = bin_of(w_hi), bottom = bin_of(w_lo);
                long long acc = (long long)hs->n_pairs;
                for (int b = HIST_BINS - 1; b >= top; b--) acc += h[b];
                one_pass = (long long)hs->n_pairs <= cap_pairs && (long long)hs->n_wide <= cap_band && acc < k_edges;
                if (one_pass) {
                    int bk = top - 1;
                    for (; bk > bottom; bk--)
                        if ((acc += h[bk]) >= k_edges) break;
                    cuts_of_bin(bk);
                    one_pass = bk > bottom && lo_cut >= w_lo && hi_cut <= w_hi;
                }
                if (one_pass) {
                    cap_pairs = p.cap_pairs = cap_total;   // the list's decided pairs join the others
                    p.lo_cut = lo_cut;
                    p.hi_cut = hi_cut;
                    p.band = band;
                    p.band_r = band_r;
                    p.n_band = &ds->n_band;
                    k_wide_split<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>(wide, wide_r, &ds->n_wide, cap_band, p);
                    PG_LAUNCHED(ctx);
                }
            }
            if (!one_pass) {
                PG_CUDA(ctx, cudaMemsetAsync(&ds->n_pairs, 0, sizeof ds->n_pairs, ctx->stream));
                PG_CUDA(ctx, cudaMemsetAsync(&ds->n_band, 0, sizeof ds->n_band, ctx->stream));
            }
        }
        if (o.mode == PG_THRESH_R) {   // the cuts are the caller's
            p.lo_cut = lo_cut;
            p.hi_cut = hi_cut;
        }
    }

    // ---- Otherwise: a full histogram pass, then the emit pass
    if (!one_pass) {
        if (o.mode == PG_THRESH_SPARSITY) {
            PG_TRY(hist_pass(floor_key, 1));
            if (floor_key > key_lo && hist_total() < k_edges) PG_TRY(hist_pass(key_lo, 1));  // sample misled us
            if (k_edges <= 0) {
                lo_cut = hi_cut = INFINITY;
            } else {
                long long acc = 0;
                int bk = 0;
                for (int b = HIST_BINS - 1; b >= 0; b--) {
                    acc += h[b];
                    if (acc >= k_edges) { bk = b; break; }
                }
                cuts_of_bin(bk);
            }
        } else if (!list_all) {
            PG_TRY(hist_pass(r_floor, 1));
        }
        PG_CUDA(ctx, cudaEventRecord(ev[2], ctx->stream));
        if (!list_all && hist_total() + (long long)hbelow[0] != M1)
            return pg_fail(ctx, PG_ERR_INTERNAL, "histogram holds %lld pairs, expected %lld",
                           hist_total() + (long long)hbelow[0], M1);
        if (lo_cut < key_lo) lo_cut = key_lo;
        // capacities: every pair, or from the histogram (upper bounds: the bin
        // mapping is monotone)
        cap_pairs = cap_band = 0;
        if (list_all) {
            cap_pairs = cap_total = M1;
            cap_band = no_band ? 0 : M1;
        } else {
            int bh = std::isfinite(hi_cut) ? bin_of(hi_cut) : HIST_BINS;
            int bl = std::isfinite(lo_cut) ? bin_of(lo_cut) : HIST_BINS;
            int be = bin_of(edge_band);
            for (int b = 0; b < HIST_BINS; b++) {
                if (b >= bh) cap_pairs += h[b];
                if (b >= bl || b >= be) cap_band += h[b];
            }
            if (lo_cut < p.kmin) cap_band += (long long)hbelow[0];   // band reaches below the binned range
            if (hi_cut < p.kmin) cap_pairs += (long long)hbelow[0];
            cap_band += (long long)hbelow[1];                         // r <= -(1 - guard), signed keys
            if (no_band) cap_band = 0;
            cap_total = cap_pairs + cap_band;
        }
        if (cap_pairs > (long long)INT32_MAX) return pg_fail(ctx, PG_ERR_TOO_LARGE, "too many edges");
        use_bits = bits_pay(k_edges >= 0 ? k_edges : cap_pairs);
        PG_TRY(prepare_decided());
        PG_TRY(prepare_band());
        p.lo_cut = lo_cut;
        p.hi_cut = hi_cut;
        if (M1 > 0 && cap_total > 0) PG_TRY(run_gram(ctx, z, o.precision, EPI_EMIT, p, &ds->timeout));
    }
    PG_CUDA(ctx, cudaEventRecord(ev[3], ctx->stream));

    // ---- FP64 recheck (and exact weights of the decided pairs)
    double tau = o.value;
    const long long n_exact = cap_band + (exact_w ? cap_pairs : 0);
    if (n_exact > 0) {
        const int grid = (int)std::max(1LL, std::min(ctx->sm_count * 16LL, (n_exact + 127) / 128));
        // the deeper pipeline where even a list of every pair leaves the SMs
        // with a few warps each (N = 90 x 1200: 120 -> 47 us); above,
        // the registers are better spent on more warps
        auto kern = list_all && n_exact <= 1024LL * ctx->sm_count ? k_pair_exact<true> : k_pair_exact<false>;
        kern<<<grid, 128, 0, ctx->stream>>>(band, band_r, pairs, exact_w ? pw : nullptr, &ds->n_pairs, cap_pairs, cap_band,
                                            z.z64, T, z.Ts, weighted, p.abs_mode, key64, &ds->err_max);
        PG_LAUNCHED(ctx);
    }
    auto check_caps = [&]() -> pg_status {
        if ((long long)hs->n_pairs > cap_pairs || (long long)hs->n_band > cap_band)
            return pg_fail(ctx, PG_ERR_INTERNAL, "emit overflow: %llu/%lld decided, %llu/%lld band", hs->n_pairs,
                           cap_pairs, hs->n_band, cap_band);
        return PG_OK;
    };
    int strict_only = 1;
    unsigned long long tie_cut = 0;
    if (o.mode == PG_THRESH_SPARSITY && k_edges > 0) {
        PG_TRY(read_state());
        PG_TRY(check_caps());
        const long long n_above = (long long)hs->n_pairs, n_band = (long long)hs->n_band;
        long long m = k_edges - n_above;  // rank inside the band
        if (m <= 0 || m > n_band)
            return pg_fail(ctx, PG_ERR_INTERNAL, "band does not contain the k-th key (k=%lld above=%lld band=%lld)",
                           k_edges, n_above, n_band);
        unsigned long long *bkeys, *tkeys;
        SelState *st, *sh;
        PG_TRY(pg_wst(ctx, "b.bkeys", (size_t)n_band, &bkeys));
        PG_TRY(pg_wst(ctx, "b.sel", 1, &st));
        PG_TRY(pg_hwst(ctx, "b.sel", 1, &sh));
        int grid = std::max(1, std::min(ctx->sm_count * 8, ceil_div(n_band, 256)));
        k_band_keys<<<grid, 256, 0, ctx->stream>>>(key64, n_band, bkeys);
        PG_LAUNCHED(ctx);
        PG_TRY(pg_radix_select(ctx, bkeys, n_band, m, st));
        PG_TRY(pg_d2h(ctx, sh, st, sizeof *sh));
        const unsigned long long tau_key = sh->prefix;
        tau = dkey_inv(tau_key);
        const long long need = sh->m, ties = sh->matching;   // ties at tau still to take (>= 1), and all of them
        strict_only = 0;
        if (ties <= need) {
            tie_cut = ~0ULL;
        } else {
            // pick the lexicographically first ones
            unsigned long long* ntie;
            PG_TRY(pg_wst(ctx, "b.tkeys", (size_t)ties + 1, &tkeys));
            PG_TRY(pg_wst(ctx, "b.ntie", 1, &ntie));
            PG_CUDA(ctx, cudaMemsetAsync(ntie, 0, sizeof(unsigned long long), ctx->stream));
            k_tie_keys<<<grid, 256, 0, ctx->stream>>>(band, bkeys, n_band, tau_key, N, tkeys, ntie);
            PG_LAUNCHED(ctx);
            PG_TRY(pg_radix_select(ctx, tkeys, ties, need, st));
            PG_TRY(pg_d2h(ctx, sh, st, sizeof *sh));
            tie_cut = ~sh->prefix;
        }
    } else if (o.mode == PG_THRESH_SPARSITY) {
        tau = INFINITY;
    }
    if (cap_band > 0) {
        const int grid = (int)std::max(1LL, std::min(ctx->sm_count * 8LL, (cap_band + 255) / 256));
        k_band_emit<<<grid, 256, 0, ctx->stream>>>(band, key64, cap_band, tau, strict_only, tie_cut, N, weighted, bits, bit_words,
                                                   pairs, pw, ds, cap_total);
        PG_LAUNCHED(ctx);
    }
    PG_TRY(read_state());
    PG_TRY(check_caps());
    PG_CUDA(ctx, cudaEventRecord(ev[4], ctx->stream));
    const long long n_band = (long long)hs->n_band;
    const long long n_edges = (long long)(hs->n_pairs + hs->n_added);
    inf.above_pairs = (long long)hs->n_pairs;
    inf.band_pairs = n_band;
    inf.zero_variance = hs->zero;
    if (n_edges > cap_total) return pg_fail(ctx, PG_ERR_INTERNAL, "edge list overflow");
    if (k_edges >= 0 && k_edges > 0 && n_edges != k_edges)
        return pg_fail(ctx, PG_ERR_INTERNAL, "sparsity graph has %lld edges, expected %lld", n_edges, k_edges);

    // ---- CSR
    pg_graph* gph;
    if (2 * n_edges > INT32_MAX)
        return pg_fail(ctx, PG_ERR_TOO_LARGE, "%lld directed entries exceed the int32 CSR", 2LL * n_edges);
    if (use_bits) PG_TRY(csr_from_bits(ctx, N, bits, bit_words, n_edges, &gph));
    else PG_TRY(pg_csr_from_pairs(ctx, N, pairs, pw, n_edges, &gph));
    cudaError_t e = cudaEventRecord(ev[5], ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        pg_graph_free(gph);
        return pg_fail(ctx, PG_ERR_CUDA, "pg_build_graph: %s", cudaGetErrorString(e));
    }
    float ms;
    cudaEventElapsedTime(&ms, ev[0], ev[1]); inf.ms_zscore = ms;
    cudaEventElapsedTime(&ms, ev[1], ev[2]); inf.ms_hist = ms;
    cudaEventElapsedTime(&ms, ev[2], ev[3]); inf.ms_emit = ms;
    cudaEventElapsedTime(&ms, ev[3], ev[4]); inf.ms_select = ms;
    cudaEventElapsedTime(&ms, ev[4], ev[5]); inf.ms_csr = ms;
    if (n_band > 0) {
        memcpy(&inf.band_err_max, &hs->err_max, 8);
        inf.band_err_mean = hs->err_sum / (double)n_band;
    }
    inf.tau = tau;
    inf.edges = n_edges;
    inf.sparsity_percent = M1 > 0 ? 100.0 * (double)n_edges / (double)M1 : 0.0;
    if (info) *info = inf;
    *out = gph;
    return PG_OK;
}

extern "C" pg_status pg_build_graph(pg_ctx* ctx, const float* bold, int32_t N, int32_t T,
                                    const pg_build_opts* opts_in, pg_graph** out, pg_build_info* info)
{
    if (!ctx || !bold || !out || N < 1 || T < 1)
        return pg_fail(ctx, PG_ERR_INVALID, "pg_build_graph: bad arguments (N=%d T=%d)", N, T);
    pg_build_opts o;
    if (opts_in) o = *opts_in; else pg_build_opts_default(&o);
    pg_status st = build_graph(ctx, bold, N, T, o, false, out, info);
    if (st == PG_ERR_NOMEM) {
        // sampled list sizes, lists of every pair and adjacency bits want room
        // to spare: where that is missing, the route that sizes its lists
        // exactly, in memory that holds nothing else of the first attempt
        pg_ws_reclaim(ctx);
        st = build_graph(ctx, bold, N, T, o, true, out, info);
    }
    return st;
}
