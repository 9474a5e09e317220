// dense_pair.cu -- the dense matmul of long portions on pairs of SMs: Y[m][n] = sum_k X[m][k] * W[n][k], both bfloat16 rows, fp32 accumulation (tcgen05, cta_group::2).
//
// Two CTAs on two SMs share one product of 256 weight rows x NB tokens: each brings its own 128 weight rows and HALF of the tokens, the tensor cores of both read both halves.
//   warp 0       streams the operands by TMA, DP_BK wide k-steps through a ring; both CTAs' copies complete on the first CTA's barrier.  The weights of the first stages are
//                asked for before the launch wait
//   warp 1       of the first CTA issues the MMAs of both and hands the stages back to both producers (commits to both CTAs' barriers)
//   warps 2..9   accumulators to memory, two warps per 32 weight rows, a half of the columns each
// The pairs walk the tiles; two accumulators in tensor memory take turns, so that a tile's way out overlaps the next one's products.  Where the tiles leave most pairs idle, 2 or 4
// pairs of one cluster take a share of K each and add their sums up through distributed shared memory, in share order.
// NB and the shares are launch arguments (pib_dense_pair_plan).
// What bounds it: a k-step of few tokens takes 0.22 - 0.33 us of one SM, whose tensor core reads its 128 weight rows from shared memory once per MMA whatever the tokens (57 clocks an MMA
// at 32 tokens): hence the shares.  Wide tiles over many rounds run at the tensor cores' rate under the operands' way into shared memory: a 128 x 128 tile per CTA (dense_mma.cu)
// asks for 128 bytes per clock and SM, a pair's 256 x 256 for 64.  us a launch, the one-CTA tiles / this (outputs x K, tokens, bfloat16 rows given): 8000 x 2048 at 1512 71 / 43
// (1.17 PFLOP/s), 5632 x 2048 at 4096 123 / 72 (1.31), 2048 x 5632 at 1512 42 / 30, at 282 32 / 15, at 20 25 / 10.
// Every wait is bounded (tc_common.cuh).
#include <cuda_bf16.h>

#include "tc_common.cuh"

#define DP_STAGES  6                         // at most; as many as DP_RING holds
#define DP_THREADS 320
#define DP_BK      128                       // two 64-wide tiles of each operand
#define DP_A_TILE  (128 * 64 * 2)
#define DP_RING    (192 * 1024)
#define DP_BARS    (2 * DP_STAGES + 4)
#define DP_SMEM    ((size_t) DP_RING + DP_BARS * 8 + 32 + 1024)

__device__ __forceinline__ uint32_t dp_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t dp_mapa(uint32_t a, uint32_t rank) { uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank)); return r; }
__device__ __forceinline__ void dp_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// What follows is called by a converged warp; one elected lane issues.  A k-step's instructions sit in one block behind one election: with an election each the producer and
// the issuing warp took 0.29 us a step instead of 0.24, which is what a step of few tokens costs.
// a stage of one operand: its two 64-wide tiles
__device__ __forceinline__ void dp_load2(uint32_t dst, uint32_t tile, const CUtensorMap * map, uint32_t bar, int k, int row) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%4, %6, %7}], [%3];\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%5, %6, %7}], [%3];\n\t}"
                 ::"r"(dst), "r"(dst + tile), "l"(map), "r"(bar), "r"(k), "r"(k + 64), "r"(row), "r"(0) : "memory");
}
// both operands; the first CTA (expect) announces the bytes of both CTAs' copies
__device__ __forceinline__ void dp_load4(uint32_t dst, uint32_t b_tile, const CUtensorMap * wmap, const CUtensorMap * xmap, uint32_t bar, int k, int n, int m, uint32_t expect, uint32_t own_bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.and.b32 e, %11, 0, q;\n\t"
                 "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%12], %13;\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%4, {%7, %9, %14}], [%6];\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%4, {%8, %9, %14}], [%6];\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%2], [%5, {%7, %10, %14}], [%6];\n\t"
                 "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%5, {%8, %10, %14}], [%6];\n\t}"
                 ::"r"(dst), "r"(dst + DP_A_TILE), "r"(dst + 2 * DP_A_TILE), "r"(dst + 2 * DP_A_TILE + b_tile), "l"(wmap), "l"(xmap), "r"(bar), "r"(k), "r"(k + 64), "r"(n), "r"(m),
                   "r"(expect), "r"(own_bar), "r"(bytes), "r"(0) : "memory");
}
__device__ __forceinline__ void dp_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
// a k-step: eight MMAs of K 16, 32 bytes further along both operands each, and the commit to the barrier at this place in both CTAs of the pair
#define DP_MMA(A, B, ACC) "@q tcgen05.mma.cta_group::2.kind::f16 [%0], " A ", " B ", %5, {%7, %7, %7, %7, %7, %7, %7, %7}, " ACC ";\n\t"
#define DP_NEXT(A, B, D)  "add.s64 a, " A ", " D ";\n\tadd.s64 b, " B ", " D ";\n\t"
__device__ __forceinline__ void dp_step(uint32_t tmem_d, uint64_t a0, uint64_t b0, uint64_t a1, uint64_t b1, uint32_t idesc, uint32_t accumulate, uint32_t bar, uint16_t mask) {
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 DP_MMA("%1", "%2", "p") DP_NEXT("%1", "%2", "2") DP_MMA("a", "b", "1") DP_NEXT("%1", "%2", "4") DP_MMA("a", "b", "1") DP_NEXT("%1", "%2", "6") DP_MMA("a", "b", "1")
                 DP_MMA("%3", "%4", "1") DP_NEXT("%3", "%4", "2") DP_MMA("a", "b", "1") DP_NEXT("%3", "%4", "4") DP_MMA("a", "b", "1") DP_NEXT("%3", "%4", "6") DP_MMA("a", "b", "1")
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%8], %9;\n\t}"
                 ::"r"(tmem_d), "l"(a0), "l"(b0), "l"(a1), "l"(b1), "r"(idesc), "r"(accumulate), "r"(0u), "r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void dp_commit(uint32_t bar, uint16_t mask) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"(mask) : "memory");
}

struct dp_args {
    int M, N, K, NB, tiles_m, tiles, shares, w_made;
    float * Y; int64_t ldy; int y_bf16;                          // y_bf16: Y holds bfloat16 rows
    float e0, e1;
    float * Y2; int64_t ld2; int n2; const int32_t * rows2;      // outputs n >= n2 go to Y2[rows2[m] * ld2 + n - n2]
    int * err;
};

// COLS columns of the lane's weight row, tokens m0 .., to memory; w0 the warp's first row
template <int EPI, int COLS> __device__ __forceinline__ void dp_out(const dp_args & A, const uint32_t (&v)[COLS], int orow, int w0, int m0) {
    const int left = A.M - m0;
    if (pib_epi_pairs(EPI)) {                        // a pair's two weight rows sit in neighbouring lanes: the even lane writes the pair's output
#pragma unroll
        for (int j = 0; j < COLS; j++) {
            const float mine = __uint_as_float(v[j]), other = __shfl_xor_sync(0xffffffffu, mine, 1);
            if (!(orow & 1) && orow + 1 < A.N && j < left) {
                const size_t at = (size_t) (m0 + j) * A.ldy + (orow >> 1);
                const float  o  = pib_glu_pair<EPI, true>(mine, other, A.e0);
                if (A.y_bf16) reinterpret_cast<__nv_bfloat16 *>(A.Y)[at] = __float2bfloat16_rn(o);
                else          A.Y[at] = o;
            }
        }
    } else if (orow < A.N) {
        if (A.y_bf16) {
            __nv_bfloat16 * p = reinterpret_cast<__nv_bfloat16 *>(A.Y) + (size_t) m0 * A.ldy + orow;
#pragma unroll
            for (int j = 0; j < COLS; j++, p += A.ldy) if (j < left) *p = __float2bfloat16_rn(pib_epilogue<EPI, true>(__uint_as_float(v[j]), A.e0, A.e1));
        } else if (w0 + 31 < A.n2) {                 // none of the warp's rows goes to Y2
            float * p = A.Y + (size_t) m0 * A.ldy + orow;
#pragma unroll
            for (int j = 0; j < COLS; j++, p += A.ldy) if (j < left) *p = pib_epilogue<EPI, true>(__uint_as_float(v[j]), A.e0, A.e1);
        } else {
            const bool second = orow >= A.n2;
            float *    base   = second ? A.Y2 + (orow - A.n2) : A.Y + orow;
#pragma unroll
            for (int j = 0; j < COLS; j++) if (j < left) base[second ? (size_t) A.rows2[m0 + j] * A.ld2 : (size_t) (m0 + j) * A.ldy] = pib_epilogue<EPI, true>(__uint_as_float(v[j]), A.e0, A.e1);
        }
    }
}

template <int EPI>
__global__ void __launch_bounds__(DP_THREADS, 1)
dense_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ dp_args A) {
    extern __shared__ __align__(1024) uint8_t dp_dsm[];
    uint8_t *  sm  = dp_dsm + ((1024u - (dt_smem(dp_dsm) & 1023u)) & 1023u);
    uint64_t * bar = reinterpret_cast<uint64_t *>(sm + DP_RING);          // full[S], free[S], accumulator ready[2], accumulator read[2]
    uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(bar + DP_BARS);
    volatile int * abort_s = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t bar_f = dt_smem(bar), bar_e = bar_f + DP_STAGES * 8, bar_t = bar_e + DP_STAGES * 8, bar_r = bar_t + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, crank = (int) dp_rank(), rank = crank & 1, S = A.shares, share = crank >> 1;
    const int unit = blockIdx.x / (2 * S), units = gridDim.x / (2 * S);                // a pair, or the cluster that shares a tile's K
    const uint32_t first = (uint32_t) (crank & ~1);                                    // the pair's first CTA
    const uint16_t both = (uint16_t) (3u << first);
    const int half = A.NB >> 1, b_tile = half * 128, stage = 2 * (DP_A_TILE + b_tile), stages = min(DP_STAGES, DP_RING / stage);
    const int all_steps = (A.K + DP_BK - 1) / DP_BK, k0 = all_steps * share / S, n_ksteps = all_steps * (share + 1) / S - k0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < DP_STAGES; s++) { dt_mbar_init(bar_f + s * 8, 1); dt_mbar_init(bar_e + s * 8, 1); }
        for (int a = 0; a < 2; a++) { dt_mbar_init(bar_t + a * 8, 1); dt_mbar_init(bar_r + a * 8, 16); }
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    dp_cluster_sync();                                           // the other CTA's barriers exist
    const uint32_t lead_f = dp_mapa(bar_f, first), sm0 = dt_smem(sm), bytes = 2 * (uint32_t) stage;
    // the weights of the first stages do not wait for the launch before this one, unless that made them
    const int early = A.w_made ? 0 : min(stages, n_ksteps);
    if (warp == 0)
        for (int s = 0; s < early; s++) {
            if (rank == 0) dp_expect(bar_f + s * 8, bytes);
            dp_load2(sm0 + s * stage, DP_A_TILE, &wmap, lead_f + s * 8, (k0 + s) * DP_BK, unit / A.tiles_m * 256 + rank * 128);
        }
    pib_pdl_wait();
    pib_pdl_trigger();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dt_smem(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (warp == 0)
        for (int s = 0; s < early; s++)
            dp_load2(sm0 + s * stage + 2 * DP_A_TILE, b_tile, &xmap, lead_f + s * 8, (k0 + s) * DP_BK, unit % A.tiles_m * A.NB + rank * half);
    dt_fence_before();
    __syncthreads();
    dp_cluster_sync();                                           // the other CTA's tensor memory is there
    dt_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        int  s = early == stages ? 0 : early, skip = early;
        uint32_t ph = early == stages ? 0 : 1;                   // the first round finds its stages free
        for (int tile = unit; tile < A.tiles && ok; tile += units) {
            const int n0 = tile / A.tiles_m * 256 + rank * 128, m0 = tile % A.tiles_m * A.NB + rank * half;
            for (int kt = skip; kt < n_ksteps; kt++) {
                ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_e + s * 8, ph, abort_s));
                if (!ok) break;
                dp_load4(sm0 + s * stage, b_tile, &wmap, &xmap, lead_f + s * 8, (k0 + kt) * DP_BK, n0, m0, rank == 0, bar_f + s * 8, bytes);
                if (++s == stages) { s = 0; ph ^= 1; }
            }
            skip = 0;
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = dt_idesc(256, A.NB);
            const uint64_t d0 = dt_desc(sm0);
            int  s = 0, n = 0;
            uint32_t ph = 0;
            for (int tile = unit; tile < A.tiles && ok; tile += units, n++) {
                const int acc = n & 1;
                if (n >= 2) ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_r + acc * 8, ((n >> 1) - 1) & 1, abort_s));
                if (!ok) break;
                for (int kt = 0; kt < n_ksteps; kt++) {
                    ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_f + s * 8, ph, abort_s));
                    if (!ok) break;
                    dt_fence_after();
                    const uint64_t ad = d0 + (uint64_t) (s * stage >> 4), bd = ad + (2 * DP_A_TILE >> 4);
                    dp_step(tmem + acc * 256, ad, bd, ad + (DP_A_TILE >> 4), bd + (b_tile >> 4), idesc, kt != 0, bar_e + s * 8, both);
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
                if (ok) dp_commit(bar_t + acc * 8, both);
            }
        }
    } else {
        const int q4 = warp & 3, hf = (warp - 2) >> 2;
        const uint32_t lead_r = dp_mapa(bar_r, first);
        float * part = reinterpret_cast<float *>(sm);            // a share's sums, [token][row]: every MMA has completed, the ring is free
        int n = 0;
        for (int tile = unit; tile < A.tiles; tile += units, n++) {
            const int acc = n & 1, w0 = tile / A.tiles_m * 256 + rank * 128 + q4 * 32, m0 = tile % A.tiles_m * A.NB;
            ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_t + acc * 8, (n >> 1) & 1, abort_s));
            if (!ok) break;
            dt_fence_after();
#pragma unroll 1
            for (int c0 = hf * 32; c0 < A.NB; c0 += 64) {
                if (m0 + c0 >= A.M) break;
                uint32_t v[32];
                dt_ld32(tmem + ((uint32_t) (q4 * 32) << 16) + acc * 256 + c0, v);
                dt_wait_ld();
                if (S == 1) dp_out<EPI>(A, v, w0 + lane, w0, m0 + c0);
                else
#pragma unroll
                    for (int j = 0; j < 32; j++) part[(c0 + j) * 128 + q4 * 32 + lane] = __uint_as_float(v[j]);
            }
            dt_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(lead_r + acc * 8) : "memory");
        }
    }
    __syncwarp();
    if (S > 1) {                                                 // one tile per cluster
        dp_cluster_sync();
        if (warp >= 2 && !*abort_s) {
            const int q4 = warp & 3, hf = (warp - 2) >> 2, w0 = unit / A.tiles_m * 256 + rank * 128 + q4 * 32, m0 = unit % A.tiles_m * A.NB;
            for (int c0 = (share * 2 + hf) * 8; c0 < A.NB && m0 + c0 < A.M; c0 += S * 16) {
                float t[8];
                for (int sh = 0; sh < S; sh++) {                 // in share order
                    const uint32_t src = dp_mapa(sm0 + (uint32_t) (c0 * 128 + q4 * 32 + lane) * 4, (uint32_t) (sh * 2 + rank));
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        float o;
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(o) : "r"(src + j * 512) : "memory");
                        t[j] = sh ? t[j] + o : o;
                    }
                }
                uint32_t v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = __float_as_uint(t[j]);
                dp_out<EPI>(A, v, w0 + lane, w0, m0 + c0);
            }
        }
    }
    dt_fence_before();
    __syncthreads();
    if (*abort_s) {
        // a wait ran out: say so, give copies and MMAs still in flight time to land (bounded), then free the tensor memory
        if (threadIdx.x == 0) atomicExch(A.err, 1 + (int) blockIdx.x);
        for (int i = 0; i < 2000; i++) __nanosleep(1000);
        __syncthreads();
    }
    dp_cluster_sync();                                           // both CTAs have read their accumulators (and the shares' sums), nothing arrives at a barrier any more
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ---- host side --------------------------------------------------------------------------------------------------------------------
// Tile width and shares of K: the least of what a launch takes by this model of its time in us, made from 700 points (N x K of 3072 x 2048, 2048 x 5632, 5632 x 2048, 8000 x 2048
// and 1024 x 2816, 20 to 2500 tokens): a k-step costs more the wider the tile and the more pairs read at once, from 160 tokens on the ring holds three steps instead of
// four or more; a round is as long as its tiles; shares cost the meeting of their sums.  Shares of S take clusters of 2 S CTAs, of which the machine holds fewer than its SMs allow
// (33 of 4 CTAs, 15 of 8).  The choice was at most 1.5 us behind the best of those points.  Beyond them it holds as far as the one-CTA tiles are no faster, which was looked at for
// 48 matrices up to 128256 x 4096 and 8192 x 28672 and is left to dt_one_cta (dense_mma.cu) where they are.
void pib_dense_pair_plan(int M, int N, int K, int * nb, int * shares) {
    const int pairs = pib_num_sms() / 2, tn = (N + 255) / 256, steps = (K + DP_BK - 1) / DP_BK;
    double best = 0;
    for (int NB = 256; NB >= 32; NB -= 32) {
        const int tiles = tn * ((M + NB - 1) / NB);
        for (int S = 1; S <= 4; S *= 2) {
            if (S > 1 && (steps < 2 * S || tiles > (S == 2 ? pairs * 4 / 9 : pairs / 5))) continue;
            const int    rounds = (tiles * S + pairs - 1) / pairs;
            const double used = (double) tiles * S / ((double) rounds * pairs), step = 0.19 + NB * 0.0011 * (1 + used) + (NB >= 160 ? 0.06 : 0.0);
            const double c = (S > 1 ? 1 : rounds) * ((steps + S - 1) / S) * step + (S > 1 ? 1.0 + 0.012 * NB : 0.0);
            if (best == 0 || c < best) { best = c; *nb = NB; *shares = S; }
        }
    }
}

int pib_dense_pair(const pib_mm & a, const CUtensorMap & wmap, const CUtensorMap & xmap, int NB, int shares, int * err, cudaStream_t st) {
    const int tiles_m = (a.M + NB - 1) / NB, tiles = tiles_m * ((a.N + 255) / 256), pairs = pib_num_sms() / 2;
    const dp_args A = { a.M, a.N, a.K, NB, tiles_m, tiles, shares, a.w_made, a.Y, a.ldy, a.y_bf16, a.e0, a.e1, a.Y2, a.ld2, a.Y2 ? a.n2 : 0x7fffffff, a.rows2, err };
    const dim3 grid((unsigned) (2 * shares * (shares > 1 || tiles < pairs ? tiles : pairs)));
#define DP_GO(EPI) do {                                                                                                                            \
        static pib_per_device attrs;                                                                                                                \
        PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(dense_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) DP_SMEM); })); \
        pib_launch_cluster(dense_pair_kernel<EPI>, grid, dim3(DP_THREADS), dim3((unsigned) (2 * shares), 1, 1), DP_SMEM, st, wmap, xmap, A);         \
    } while (0)
    switch (a.epi) {
        case PIB_EPI_RELU2:       DP_GO(PIB_EPI_RELU2); break;
        case PIB_EPI_XIELU:       DP_GO(PIB_EPI_XIELU); break;
        case PIB_EPI_GLU_PAIR:    DP_GO(PIB_EPI_GLU_PAIR); break;
        case PIB_EPI_GEGLU_PAIR:  DP_GO(PIB_EPI_GEGLU_PAIR); break;
        case PIB_EPI_SWIGLU_PAIR: DP_GO(PIB_EPI_SWIGLU_PAIR); break;
        default:                  DP_GO(PIB_EPI_NONE); break;
    }
#undef DP_GO
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}
