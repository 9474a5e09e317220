// gemm_q4k_tc.cu -- the quantised matmul (K1) for WIDE batches (prompt ingestion, up to PIB_PROMPT_MAX tokens at once): Q4_K weights are dequantised to fp16
// straight into tensor memory and multiplied there on the 5th-generation tensor cores (tcgen05.mma with A in tensor memory, fp32 accumulators), the
// activation tile arriving by TMA.  Replaces, for these batch sizes, the reference's ggml_compute_forward_mul_mat at large ne11 (ggml.c:9388) /
// ggml_cuda_op_mul_mat_cublas (ggml-cuda.cu:6562: dequantise + cuBLAS).
//
// Arithmetic: y[t][r] = sum_k w(r, k) * x^(t, k) with w = d * sc * q - dmin * m (the reference's dequantize_row_q4_K formula,
// ggml-quants.c:1917) rounded to fp16, and x^ = the token's Q8_K quantised activation q8 * d (what the reference's integer dot
// product multiplies with) rounded to fp16; fp32 accumulation over K in tensor memory.  This is NOT the reference's summation
// order and not bit-exact; it is checked against the oracle to a tolerance (tests/test_gpu_gemm.py) and used for prompt chunks only
// -- verification batches (<= 16 tokens) keep the GEMV kernels.
//
// A CTA owns 128 output rows and a tile of up to 256 tokens, and one share of K when a cluster splits it:
//   warp 0          TMA: the activation tile [NB tokens x 128 k] fp16 of every k-step (cp.async.bulk.tensor.2d, 128-byte swizzle)
//   warp 1          allocates tensor memory, issues the MMAs (8 x K=16 per k-step) and commits them to the mbarriers
//   warp 2          weight records: one bulk copy per 16-row tile and super-block into a ring, started before the launch wait
//   warps 3..       G groups of 8: a warp owns one 16-row tile, turns its 16-byte fragment pieces into fp16 pairs in registers and stores them with
//                   tcgen05.st.16x256b: the record layout (lane g, t holds rows g and g + 8, gemv_mma.cu) IS that instruction's register layout, only
//                   the order of k inside a 64-wide chunk differs, and x^ is written in the same order (tg_kpos).  Afterwards the epilogue.
// Weights run four k-steps ahead in tensor memory; the activations' places are a ring of their own where they come in pieces (256 tokens: with two weight steps the groups waited for
// the MMAs of the step before last; with four, and the producer and the issuing warp counting their places along, 12288 x 4096 32.7 -> 27.6 us, 4096 x 4096 18.8 -> 16.4,
// 57344 x 8192 204 -> 192).
// What bounds it: up to about 100 tokens the dequantisation, 109 warp instructions per 16 rows x 64 k issued at 0.6 per clock and scheduler (57344 x 8192
// at 40 tokens 96 us, where the weights' bytes take 40; with the operand written to and read from shared memory, the form this replaced, 173 us); with
// 256 tokens the tensor cores and the activation tiles' way into shared memory (192 us; 151 at the dense peak).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "q8k_quant.cuh"
#include "tc_common.cuh"

#define TG_BM      128                 // output rows per accumulator (UMMA M)
#define TG_BK      128                 // k elements per step (two 128-byte swizzle rows of fp16): half a super-block
#define TG_TILE_BYTES 2304             // Q4_K record of (16 rows, 256 k), see gemv_mma.cu

// G groups of 8 warps feed the accumulator (G = 2: the groups take the k-steps in turn); with G = 1 two CTAs share an SM
template <int NB, int G> struct tg_cfg {
    static constexpr int CTAS    = 3 - G;                                // per SM
    static constexpr int STAGES  = G == 2 ? 4 : NB > 64 ? 2 : 3;   // k-steps of weights in tensor memory
    static constexpr int PIECES  = NB > 128 ? 2 : 1;                     // activations arrive in pieces of a k-step where shared memory holds two whole steps only, which are
    static constexpr int BSTAGES = NB > 128 ? 4 : STAGES;                // late then (256 tokens: 246 -> 193 us); elsewhere a second barrier per step costs more (24 tokens: 31 -> 44)
    static constexpr int WSTAGES = NB == 128 && G == 1 ? 2 : 3;          // super-blocks of weight records in shared memory
    static constexpr int WARPS   = 8 * G, THREADS = 96 + 32 * WARPS;
    static constexpr int W_BYTES = 8 * TG_TILE_BYTES, B_BYTES = NB * 256 / PIECES;
    static constexpr int TM_COLS = 512 / CTAS;                           // tensor memory: NB accumulator columns, then STAGES x 64 columns of weights
    static constexpr int RED     = TG_BM * NB * 4;                       // the partial sums of a K split reuse the rings
    static constexpr int SCL_OFF = BSTAGES * B_BYTES + WSTAGES * W_BYTES; // the warps' expanded scales
    static constexpr int RING    = SCL_OFF + WARPS * 1024;
    static constexpr int N_BAR   = 2 * (STAGES + BSTAGES + WSTAGES) + 1;
    static constexpr int BAR_OFF = RED > RING ? RED : RING;
    static constexpr size_t SMEM = (size_t) BAR_OFF + N_BAR * 8 + 32 + 1024;
    static_assert(NB + STAGES * 64 <= TM_COLS && G <= STAGES, "tensor memory");
};

// ---- x^: quantised activations back to fp16, [b][K], k order inside a chunk as above -----------------------------------------------------------
__global__ void __launch_bounds__(256) tg_xhat_kernel(const int8_t * __restrict__ qs, const float * __restrict__ d, int64_t n16, int K16, __half * __restrict__ xh) {
    pib_pdl_wait();
    pib_pdl_trigger();
    const int64_t i = (int64_t) blockIdx.x * 256 + threadIdx.x;              // sixteen consecutive elements of one row
    if (i >= n16) return;
    const float dx = d[(i / K16) * (K16 / 16) + (i % K16) / 16];
    const int4  q  = reinterpret_cast<const int4 *>(qs)[i];
    __half *    o  = xh + (i >> 2) * 64;
    const int   e0 = (int) (i & 3) * 16;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int w = u == 0 ? q.x : u == 1 ? q.y : u == 2 ? q.z : q.w;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = __fmul_rn((float) (int8_t) (w >> (8 * j)), dx);
        const __half2 p[2] = { __floats2half2_rn(v[0], v[2]), __floats2half2_rn(v[1], v[3]) };
        *reinterpret_cast<uint2 *>(o + tg_kpos(e0 + 4 * u)) = *reinterpret_cast<const uint2 *>(p);
    }
}

__device__ __forceinline__ void tg_bulk(uint32_t dst, const void * src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// N (1 or 2) boxes of 64 k and the announcement of their bytes; by a converged warp, one elected lane issues (a lane's own loop with its places formed by division took 600 clocks a round)
template <int N> __device__ __forceinline__ void tg_load(uint32_t dst, uint32_t box, const CUtensorMap * map, uint32_t bar, uint32_t bytes, int k, int row) {
    if (N == 2) asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %4;\n\t"
                             "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%5, %7}], [%3];\n\t"
                             "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%6, %7}], [%3];\n\t}"
                             ::"r"(dst), "r"(dst + box), "l"(map), "r"(bar), "r"(bytes), "r"(k), "r"(k + 64), "r"(row) : "memory");
    else asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], %3;\n\t"
                      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%4, %5}], [%2];\n\t}"
                      ::"r"(dst), "l"(map), "r"(bar), "r"(bytes), "r"(k), "r"(row) : "memory");
}
// four MMAs of 16 k, A in tensor memory, B in shared memory; by a converged warp
__device__ __forceinline__ void tg_mma4(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b32 a;\n\t.reg .b64 b;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t"
                 "add.s32 a, %1, 8;\n\tadd.s64 b, %2, 2;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, {%5, %5, %5, %5}, 1;\n\t"
                 "add.s32 a, %1, 16;\n\tadd.s64 b, %2, 4;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, {%5, %5, %5, %5}, 1;\n\t"
                 "add.s32 a, %1, 24;\n\tadd.s64 b, %2, 6;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, {%5, %5, %5, %5}, 1;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// 16 lanes x 64 columns: register 4a + j of lane (g, t) is column 8a + 2t + (j & 1) of lane g + 8 (j >> 1)
__device__ __forceinline__ void tg_st_frag(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
                 "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
// Waits are bounded: TG_TRIES tries, then the block's abort flag is raised and every role gives up.  The weight producer, which is a whole
// super-block or two ahead, sleeps in the barrier unit (up to NAP ns a try) and leaves its issue slots to the others; those poll, because a sleeper wakes late.
#define TG_TRIES (1 << 20)
template <uint32_t NAP> __device__ __forceinline__ uint32_t tg_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (NAP) asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(NAP) : "memory");
    else     asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// by a whole warp, which leaves together: what follows are .sync.aligned instructions, and lanes that left one by one would run them in parts
template <uint32_t NAP = 0> __device__ __forceinline__ bool tg_wait(uint32_t bar, uint32_t parity, volatile int * abort_s) {
    for (int it = 0; it < TG_TRIES; it++) {
        if (__all_sync(0xffffffffu, tg_try<NAP>(bar, parity))) return true;
        if ((it & 15) == 15 && __any_sync(0xffffffffu, *abort_s)) return false;
    }
    *abort_s = 1;
    return false;
}
__device__ __forceinline__ __half2 tg_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t tg_u(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// {d * sc, -dmin * m} of sub-blocks 2c, 2c + 1 of one row, each twice in a word (get_scale_min_k4, ggml-quants.c:1446): d * sc has 17 bits, so the fp16
// product is its value rounded once
__device__ __forceinline__ uint4 tg_scales(uint4 h, int c) {
    const uint32_t sc = c < 2 ? h.y & 0x3f3f3f3fu : (h.w & 0x0f0f0f0fu) | (((h.y >> 6) & 0x03030303u) << 4);
    const uint32_t mn = c < 2 ? h.z & 0x3f3f3f3fu : ((h.w >> 4) & 0x0f0f0f0fu) | (((h.z >> 6) & 0x03030303u) << 4);
    const __half2  d = __low2half2(tg_h2(h.x)), nm = __hneg2(__high2half2(tg_h2(h.x))), k1024 = __float2half2_rn(1024.f);
    const uint32_t s0 = c & 1 ? 0x4242 : 0x4040, s1 = s0 + 0x0101;
    return make_uint4(tg_u(__hmul2(__hsub2(tg_h2(__byte_perm(sc, 0x64646464u, s0)), k1024), d)), tg_u(__hmul2(__hsub2(tg_h2(__byte_perm(mn, 0x64646464u, s0)), k1024), nm)),
                      tg_u(__hmul2(__hsub2(tg_h2(__byte_perm(sc, 0x64646464u, s1)), k1024), d)), tg_u(__hmul2(__hsub2(tg_h2(__byte_perm(mn, 0x64646464u, s1)), k1024), nm)));
}
// (v & m) | 0x6400 in both halves, in one instruction (both constants in registers): nibbles enter fp16 as 1024 + q (low) and 1024 + 16 q (high)
__device__ __forceinline__ __half2 tg_pick(uint32_t v, uint32_t m) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(m), "r"(0x64006400u));
    return tg_h2(r);
}
// a word of eight nibbles -> low pairs (e0, e2), (e1, e3) and high pairs, each d1 * q + o with one rounding (q comes back exactly first)
__device__ __forceinline__ void tg_word(uint32_t v, __half2 d_lo, __half2 o_lo, __half2 d_hi, __half2 o_hi, uint32_t & l0, uint32_t & l1, uint32_t & h0, uint32_t & h1) {
    const __half2 k1024 = __float2half2_rn(1024.f), sixteenth = __float2half2_rn(0.0625f), k64 = __float2half2_rn(-64.f);
    const uint32_t s = v >> 8;
    l0 = tg_u(__hfma2(__hsub2(tg_pick(v, 0x000F000Fu), k1024), d_lo, o_lo));
    l1 = tg_u(__hfma2(__hsub2(tg_pick(s, 0x000F000Fu), k1024), d_lo, o_lo));
    h0 = tg_u(__hfma2(__hfma2(tg_pick(v, 0x00F000F0u), sixteenth, k64), d_hi, o_hi));
    h1 = tg_u(__hfma2(__hfma2(tg_pick(s, 0x00F000F0u), sixteenth, k64), d_hi, o_hi));
}
// a chunk's two pieces of one row: registers 4a + J0 + {0, 1} of the fragment
template <int C, int J0> __device__ __forceinline__ void tg_chunk_row(uint32_t w0, uint32_t w1, uint4 f, uint32_t (&o)[32]) {
    const __half2 dl = tg_h2(f.x), ol = tg_h2(f.y), dh = tg_h2(f.z), oh = tg_h2(f.w);
    tg_word(w0, dl, ol, dh, oh, o[16 * C + J0], o[16 * C + J0 + 1], o[16 * C + J0 + 8], o[16 * C + J0 + 9]);
    tg_word(w1, dl, ol, dh, oh, o[16 * C + J0 + 4], o[16 * C + J0 + 5], o[16 * C + J0 + 12], o[16 * C + J0 + 13]);
}

// ---- the GEMM ------------------------------------------------------------------------------------------------------------------
// grid (blocks, 1, K shares); the K shares of a block are one cluster
template <int NB, int G>
__global__ void __launch_bounds__(tg_cfg<NB, G>::THREADS, tg_cfg<NB, G>::CTAS)
gemm_q4k_tc_kernel(const uint8_t * __restrict__ tiles, int nsb, int N, int x0, int ny, const __grid_constant__ CUtensorMap xmap, int b_all, float * __restrict__ y_all, int * __restrict__ err) {
    using C = tg_cfg<NB, G>;
    extern __shared__ __align__(1024) uint8_t tg_dsm[];
    uint8_t *  sB  = tg_dsm + ((1024u - (dt_smem(tg_dsm) & 1023u)) & 1023u);      // [BSTAGES][64 k][NB rows][128 B], 1024-byte aligned (swizzle atom)
    uint8_t *  sW  = sB + C::BSTAGES * C::B_BYTES;                                // [WSTAGES][8 tiles][2304 B]
    uint64_t * bar = reinterpret_cast<uint64_t *>(sB + C::BAR_OFF);
    uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(bar + C::N_BAR);
    volatile int * abort_s = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // weights: step full / free; activations: piece full / free; records: full / free; accumulators complete
    const uint32_t bar_a = dt_smem(bar), bar_e = bar_a + C::STAGES * 8, bar_b = bar_e + C::STAGES * 8, bar_be = bar_b + C::BSTAGES * 8, bar_w = bar_be + C::BSTAGES * 8, bar_we = bar_w + C::WSTAGES * 8,
                   bar_t = bar_we + C::WSTAGES * 8, bar_bf = C::PIECES == 1 ? bar_e : bar_be;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = gridDim.z, sb_lo = (int) ((long long) nsb * blockIdx.z / S), sb_hi = (int) ((long long) nsb * (blockIdx.z + 1) / S);
    const int n_sb = sb_hi - sb_lo, n_ksteps = n_sb * 2;
    // block x0 + blockIdx.x: row block and token tile, the ny tiles of a row block next to each other
    const int row0 = (x0 + (int) blockIdx.x) / ny * TG_BM, tok0 = (x0 + (int) blockIdx.x) % ny * NB, b = min(NB, b_all - tok0);
    float *   y = y_all + (size_t) tok0 * N;
    const int n_tiles = min(8, (N + 15) / 16 - row0 / 16);                   // 16-row tiles this block has

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) { dt_mbar_init(bar_a + s * 8, 8); dt_mbar_init(bar_e + s * 8, 1); }
        for (int s = 0; s < C::BSTAGES; s++) { dt_mbar_init(bar_b + s * 8, 1); dt_mbar_init(bar_be + s * 8, 1); }
        for (int s = 0; s < C::WSTAGES; s++) { dt_mbar_init(bar_w + s * 8, 1); dt_mbar_init(bar_we + s * 8, C::WARPS); }
        dt_mbar_init(bar_t, 1);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dt_smem(tmem_slot)), "r"((uint32_t) C::TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    dt_fence_before();
    __syncthreads();
    dt_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        pib_pdl_wait();
        pib_pdl_trigger();
        int  s = 0, k = sb_lo * 256;
        uint32_t ph = 1;                                           // the first round finds its places free
        for (int kp = 0; kp < C::PIECES * n_ksteps; kp++, k += 128 / C::PIECES) {
            if (!tg_wait(bar_bf + s * 8, ph, abort_s)) break;
            tg_load<2 / C::PIECES>(dt_smem(sB) + s * C::B_BYTES, NB * 128, &xmap, bar_b + s * 8, C::B_BYTES, k, tok0);
            if (++s == C::BSTAGES) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        // instruction descriptor: fp32 accumulate, fp16 x fp16, both K-major, N = NB, M = 128
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t) (NB >> 3) << 17) | ((uint32_t) (TG_BM >> 4) << 24);
        const uint64_t bd0 = dt_desc(dt_smem(sB));
        int  s = 0, sp = 0;
        uint32_t ph = 0, php = 0;
        for (int kt = 0; kt < n_ksteps && ok; kt++) {
            ok = tg_wait(bar_a + s * 8, ph, abort_s);
            for (int j = 0; j < C::PIECES && ok; j++) {
                ok = tg_wait(bar_b + sp * 8, php, abort_s);
                if (!ok) break;
                dt_fence_after();
                const uint64_t bd = bd0 + (uint64_t) (sp * C::B_BYTES >> 4);
                const uint32_t ta = tmem + NB + s * 64 + j * 32;
                tg_mma4(tmem, ta, bd, idesc, (kt | j) != 0);      // 8 columns of weights and 32 bytes of activations further along K each
                if (C::PIECES == 1) tg_mma4(tmem, ta + 32, bd + (NB * 128 >> 4), idesc, 1);
                else dt_commit(bar_be + sp * 8);                  // the piece is free when these MMAs have read it
                if (++sp == C::BSTAGES) { sp = 0; php ^= 1; }
            }
            if (ok) dt_commit(bar_e + s * 8);
            if (++s == C::STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) dt_commit(bar_t);
    } else if (warp == 2) {
        // weights are immutable: their copies do not wait for the launch before this one
        const uint8_t * src = tiles + ((size_t) (row0 / 16 + lane) * nsb + sb_lo) * TG_TILE_BYTES;
        for (int i = 0; i < n_sb; i++) {
            const int s = i % C::WSTAGES;
            if (i >= C::WSTAGES && !tg_wait<1000>(bar_we + s * 8, ((i / C::WSTAGES) - 1) & 1, abort_s)) break;
            if (lane == 0) dt_mbar_expect_tx(bar_w + s * 8, (uint32_t) n_tiles * TG_TILE_BYTES);
            __syncwarp();
            if (lane < n_tiles) tg_bulk(dt_smem(sW + s * C::W_BYTES + lane * TG_TILE_BYTES), src + (size_t) i * TG_TILE_BYTES, TG_TILE_BYTES, bar_w + s * 8);
        }
    } else {
        // ---- warps 3..: tensor-memory lanes 32 q .. 32 q + 31 belong to warp number q mod 4; rows q * 32 + hf * 16 ----
        const int p = warp - 3, gs = p >> 3, q = warp & 3, hf = (p >> 2) & 1, g = lane >> 2;
        uint4 *         scl  = reinterpret_cast<uint4 *>(sB + C::SCL_OFF) + p * 64;       // [chunks][16 rows] factors of this warp's record
        const uint8_t * rec0 = sW + (q * 2 + hf) * TG_TILE_BYTES;
        const uint32_t  ta0  = tmem + ((uint32_t) (q * 32 + hf * 16) << 16) + NB;
        int      ws = 0, sl = gs, s_prev = 0;                      // ring places, counted along instead of divided
        uint32_t wph = 0, eph = 1;                                 // phases: records full, step free (the first round passes at once)
        constexpr int NH = 2 / G;                                  // k-steps of a record that this warp takes
        for (int i = 0; i < n_sb && ok; i++) {
            if (!tg_wait(bar_w + ws * 8, wph, abort_s)) { ok = false; break; }
            const uint8_t * rec = rec0 + ws * C::W_BYTES;
            __syncwarp();                                          // the factors of the record before have been read
            // every lane forms the factors of one row and one (G = 2) or two chunks; the lanes of a row pair read them back per chunk
#pragma unroll
            for (int h = 0; h < NH; h++) {
                const int r = lane & 15, c = (gs + h) * 2 + (lane >> 4);
                scl[h * 32 + lane] = tg_scales(*reinterpret_cast<const uint4 *>(rec + 2048 + r * 16), c);
            }
            uint4 v[2 * NH];
#pragma unroll
            for (int c = 0; c < 2 * NH; c++) v[c] = *reinterpret_cast<const uint4 *>(rec + (gs * 2 + c) * 512 + lane * 16);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < NH; h++) {                         // 128 k: chunks 2 (gs + h), + 1
                uint32_t o[32];
                tg_chunk_row<0, 0>(v[2 * h].x, v[2 * h].y, scl[h * 32 + g], o);
                tg_chunk_row<0, 2>(v[2 * h].z, v[2 * h].w, scl[h * 32 + g + 8], o);
                tg_chunk_row<1, 0>(v[2 * h + 1].x, v[2 * h + 1].y, scl[h * 32 + 16 + g], o);
                tg_chunk_row<1, 2>(v[2 * h + 1].z, v[2 * h + 1].w, scl[h * 32 + 16 + g + 8], o);
                if (h == NH - 1) {
                    // The ring place is given back to a bulk copy, a write of the async proxy, which nothing orders behind this lane's generic reads of the record but a
                    // proxy fence: every lane's reads, its fence, the warp's meeting, one arrival.  (Without the fence and with the arrival right behind the loads
                    // quads of rows came out wrong where calls follow one another closely, 69 of 200 calls.)
                    dt_fence_async();
                    __syncwarp();
                    if (lane == 0) dt_arrive(bar_we + ws * 8);
                    if (++ws == C::WSTAGES) { ws = 0; wph ^= 1; }
                }
                if (i | h) {                                       // the step before: its stores had this step's arithmetic to land in
                    dt_wait_st();
                    dt_fence_before();
                    if (lane == 0) dt_arrive(bar_a + s_prev * 8);
                    __syncwarp();
                }
                ok = tg_wait(bar_e + sl * 8, eph, abort_s);
                if (!ok) break;
                dt_fence_after();
                tg_st_frag(ta0 + sl * 64, o);
                s_prev = sl;
                sl += G;
                if (sl >= C::STAGES) { sl -= C::STAGES; eph ^= 1; }
            }
        }
        dt_wait_st();
        dt_fence_before();
        if (lane == 0) dt_arrive(bar_a + s_prev * 8);
        __syncwarp();
        // ---- accumulators: a lane is a row; two (four) warps per 32 rows share the columns ----
        pib_pdl_wait();
        pib_pdl_trigger();
        ok = ok && tg_wait(bar_t, 0, abort_s);
        if (ok) {
            dt_fence_after();
            const int r = q * 32 + lane, orow = row0 + r;
            float * part = reinterpret_cast<float *>(sB);
#pragma unroll 1
            for (int c0 = (gs * 2 + hf) * 32; c0 < NB; c0 += 64 * G) {
                if (S == 1 && c0 >= b) break;
                uint32_t u[32];
                dt_ld32(tmem + ((uint32_t) (q * 32) << 16) + c0, u);
                dt_wait_ld();
                if (S > 1) {                                    // this share's sums, [token][row]: the rings are free, every MMA has completed
#pragma unroll
                    for (int j = 0; j < 32; j++) part[(c0 + j) * TG_BM + r] = __uint_as_float(u[j]);
                } else if (orow < N) {
#pragma unroll
                    for (int j = 0; j < 32; j++) if (c0 + j < b) y[(size_t) (c0 + j) * N + orow] = __uint_as_float(u[j]);
                }
            }
        }
    }
    __syncwarp();
    if (S > 1) {
        // K shares meet through distributed shared memory: every CTA of the cluster adds its part of the tokens, in share order
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (warp >= 3 && !*abort_s) {
            const int r = (threadIdx.x - 96) & 127, orow = row0 + r;
            const uint32_t base = dt_smem(sB);
            for (int j = blockIdx.z * 2 * G + ((threadIdx.x - 96) >> 7); j < b; j += 2 * G * S) {
                float v = 0.f;
                for (int s = 0; s < S; s++) {
                    uint32_t a;
                    float    o;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(base + (uint32_t) (j * TG_BM + r) * 4), "r"(s));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(o) : "r"(a) : "memory");
                    v = s ? v + o : o;
                }
                if (orow < N) y[(size_t) j * N + orow] = v;
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");      // nobody leaves while its sums are read
    }
    dt_fence_before();
    __syncthreads();
    if (*abort_s) {
        // a wait ran out: say so, give copies and MMAs still in flight time to land (bounded), then free the tensor memory
        if (threadIdx.x == 0) atomicExch(err, 1 + (int) blockIdx.x);
        for (int i = 0; i < 2000; i++) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t) C::TM_COLS) : "memory");
}

// ---- host side --------------------------------------------------------------------------------------------------------------------
typedef CUresult (*tg_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static tg_encode_fn tg_encode() {
    static tg_encode_fn fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult st;
        void * p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &st) == cudaSuccess && st == cudaDriverEntryPointSuccess) fn = (tg_encode_fn) p;
    }
    return fn;
}

// token tiles and tokens per CTA
static int tg_tiles_of(int b) { return (b + 255) / 256; }
static int tg_nb_of(int b_all) { const int ny = tg_tiles_of(b_all), b = (b_all + ny - 1) / ny; return b <= 32 ? 32 : b <= 64 ? 64 : b <= 96 ? 96 : b <= 128 ? 128 : b <= 192 ? 192 : 256; }
size_t pib_gemm_xhat_bytes(int64_t K, int b) { return (size_t) (b <= 32 ? 32 : b <= 64 ? 64 : b <= 128 ? 128 : b <= 256 ? 256 : b) * K * sizeof(__half); }

// Clusters of S CTAs, one CTA per SM, that the machine holds at once: not every GPC's SMs divide by S, so it is fewer than the SMs do (148 SMs: 148, 74, 33, 15 of
// 1, 2, 4, 8 CTAs, which the launches bear out: 34 clusters of 4 take two rounds).
template <int NB>
static int tg_fit(int S) {
    using C = tg_cfg<NB, 2>;
    static std::atomic<int> known[5];                                            // of 1, 2, 3, 4, 8; + 1
    std::atomic<int> & k = known[S < 5 ? S - 1 : 4];
    if (const int v = k.load()) return v - 1;
    int n = 0;
    if (cudaFuncSetAttribute(gemm_q4k_tc_kernel<NB, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) C::SMEM) == cudaSuccess) {
        cudaLaunchAttribute at;
        memset(&at, 0, sizeof(at));
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = (unsigned) S;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, (unsigned) S); cfg.blockDim = dim3(C::THREADS); cfg.dynamicSmemBytes = C::SMEM; cfg.attrs = &at; cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_q4k_tc_kernel<NB, 2>, &cfg) != cudaSuccess) n = 0;
    }
    cudaGetLastError();
    k.store(n + 1);
    return n;
}
static int tg_fit_nb(int NB, int S) {
    switch (NB) {
        case 32:  return tg_fit<32>(S);
        case 64:  return tg_fit<64>(S);
        case 96:  return tg_fit<96>(S);
        case 128: return tg_fit<128>(S);
        case 192: return tg_fit<192>(S);
        default:  return tg_fit<256>(S);
    }
}

// blocks [x0, x0 + nx), K in S shares
template <int NB, int G>
static int tg_launch(const pib_weight * w, const __half * xh, int b, int x0, int nx, int S, float * y, cudaStream_t st) {
    using C = tg_cfg<NB, G>;
    tg_encode_fn enc = tg_encode();
    if (!enc) { pib_set_error("pib_gemm: cuTensorMapEncodeTiled not available"); return PIB_ERR_UNSUPP; }
    CUtensorMap map;
    const cuuint64_t gdim[2] = { (cuuint64_t) w->K, (cuuint64_t) b };            // rows behind b are zero-filled
    const cuuint64_t gstr[1] = { (cuuint64_t) w->K * sizeof(__half) };
    const cuuint32_t box[2]  = { 64, (cuuint32_t) NB };
    const cuuint32_t estr[2] = { 1, 1 };
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void *) xh, gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { pib_set_error("pib_gemm: cuTensorMapEncodeTiled failed (%d)", (int) r); return PIB_ERR_CUDA; }
    // Two CTAs of one group share an SM where there are more of them than SMs.  Where there are not, and all clusters find room at one per SM, they ask for so much shared memory
    // that they do not: launched while the quantiser in front still runs they would double up (us a call: 4096 x 14336 at 56 / 64 tokens 28.8 29.1 / 21.9 22.3, 4096 x 12288
    // at 64 26.2 / 20.3)
    const size_t smem = G == 1 && nx * S <= pib_num_sms() && nx <= tg_fit_nb(NB, S) ? std::max(C::SMEM, (size_t) PIB_GEMV_SPREAD) : C::SMEM;
    static pib_per_device attrs;
    PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(gemm_q4k_tc_kernel<NB, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) std::max(C::SMEM, (size_t) PIB_GEMV_SPREAD)); }));
    const dim3 grid((unsigned) nx, 1, (unsigned) S);
    int * err = pib_tc_error_word(st);
    if (!err) { pib_set_error("pib_gemm: no memory for the stream's error word"); return PIB_ERR_NOMEM; }
    if (S > 1) pib_launch_cluster(gemm_q4k_tc_kernel<NB, G>, grid, dim3(C::THREADS), dim3(1, 1, (unsigned) S), smem, st, w->tiles, (int) (w->K / 256), (int) w->N, x0, tg_tiles_of(b), map, b, y, err);
    else       pib_launch(gemm_q4k_tc_kernel<NB, G>, grid, dim3(C::THREADS), smem, st, w->tiles, (int) (w->K / 256), (int) w->N, x0, tg_tiles_of(b), map, b, y, err);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

// The launches of a matmul of N x K and b tokens: blocks [0, full) and behind them `rest`, each with its K shares; G groups of dequantising warps per CTA (1: two CTAs per SM).
struct tg_plan { int G, full, s_full, rest, s_rest; };
static tg_plan tg_plan_of(int64_t N, int64_t K, int b) {
    const int NB = tg_nb_of(b), nsb = (int) (K / 256), nx = (int) ((N + TG_BM - 1) / TG_BM) * tg_tiles_of(b), sms = pib_num_sms();
    // K shares of n blocks, with G groups, whose clusters all find room at once; every share keeps at least two super-blocks.  With two CTAs per SM, S of them need
    // the room of S / 2, less a sixteenth that packing loses (occupancy queries count one CTA of this kernel per SM; of 4 CTAs 70 clusters ran at once, 72 did not).
    // us at 34 and 37 blocks of K = 4096 / 100 tokens and 17 of 8192 / 256, shares by room / by SMs alone: 16.9 / 22.5, 16.8 / 22.8, 22.6 / 31.6.
    auto shares = [&](int n, int G) {
        int S = 1;
        while (S < 8 && nsb / (S * 2) >= 2 && n <= (G == 2 ? tg_fit_nb(NB, S * 2) : tg_fit_nb(NB, S) * 15 / 16)) S *= 2;
        // three where four do not fit (two / three, 34 .. 42 blocks: K = 4096 at 100 / 256 tokens 23.6 33.8 / 21.5 29.7 .. 31.7, K = 14336 44.0 62.2 / 35.8 50.2)
        if (G == 2 && S == 2 && nsb >= 6 && n <= tg_fit_nb(NB, 3)) S = 3;
        return S;
    };
    // More blocks than clusters of two find room for, and no more than three shares of each find at two CTAs per SM (of 90 blocks; of 92 they take two rounds): without them the
    // blocks are fewer than the SMs.  From the K on where a share is worth its meeting (one / three shares, us, 40 64 100 128 tokens: 80 blocks of 8192 38.0 40.0 43.0 44.9 / 31.8 33.8
    // 39.9 42.0, of 14336 59.1 60.7 66.1 67.7 / 44.0 46.1 54.2 56.9; of 6144 31.7 32.7 35.8 35.7 / 27.6 29.6 35.4 36.7; of 4096 25.5 25.6 27.7 27.9 / 24.9 25.6 30.2 31.7;
    // 90 blocks of 8192 39.5 39.9 43.4 44.4 / 33.7 35.8 42.0 46.4: above 64 tokens 81 blocks at most).
    const bool three = NB <= 128 && nx > tg_fit_nb(NB, 2) && (NB <= 64 ? 18 * nx <= 11 * sms && nsb >= 18 : 20 * nx <= 11 * sms && nsb >= 32);
    // One CTA with two groups, or two CTAs with one, per SM (us, one / two, 40 and 128 tokens): 12288 x 4096 (96 row blocks) 18.7 / 20.8 and 20.9 / 29.6,
    // 10240 x 8192 (80) 31.4 / 33.4 and 33.8 / 42.7, 22016 x 4096 (172) 35.5 / 29.4 and 39.5 / 34.7, 8192 x 28672 (64, in 2 / 4 shares) 54.2 / 49.1 and 68.5 / 67.7.
    // Above 128 tokens the accumulator takes half of the tensor memory: one.
    const bool two = NB <= 128 && (nx > sms || (NB <= 64 && shares(nx, 2) > 1));
    if (two || three) return { 1, nx, three ? 3 : shares(nx, 1), 0, 1 };
    // whole rounds of one CTA per SM, then what is left over in K shares (448 row blocks are three rounds and four blocks)
    int full = nx / sms * sms, rest = nx - full;
    if (full > 0 && shares(rest, 2) == 1) { full = nx; rest = 0; }
    return { 2, full, full > 0 ? shares(full, 2) : 1, rest, rest > 0 ? shares(rest, 2) : 1 };
}
extern "C" int pib_gemm_shares(int64_t N, int64_t K, int b, int * groups) {
    if (N <= 0 || K <= 0 || K % 256 || b < 1 || b > PIB_PROMPT_MAX) return -1;
    const tg_plan p = tg_plan_of(N, K, b);
    if (groups) *groups = p.G;
    return p.rest ? p.s_rest : p.s_full;
}

// y[b][N] = W x^; act_dev = the Q8_K activation planes of `b` tokens (act_quant.cu), xhat_dev = scratch of pib_gemm_xhat_bytes; or act_dev = null and xhat_dev already
// written by the quantiser (51 launches of 4 us in a 700-token prompt through four layers)
int pib_gemm_q4k_tc(const pib_weight * w, const void * act_dev, int b, float * y_dev, void * xhat_dev, cudaStream_t st) {
    if (!w || w->type != PIB_TYPE_Q4_K || !w->tiles || b < 1 || b > PIB_PROMPT_MAX) { pib_set_error("pib_gemm: needs Q4_K tiles and 1 <= b <= %d", PIB_PROMPT_MAX); return PIB_ERR_ARG; }
    const pib_act_layout L = pib_act_layout_of(PIB_TYPE_Q4_K, w->K, b);
    const uint8_t * act = (const uint8_t *) act_dev;
    __half * xh = (__half *) xhat_dev;
    const int64_t n16 = (int64_t) b * (w->K / 16);
    if (act && b > PIB_MAX_BATCH) { xh = (__half *) (const_cast<uint8_t *>(act) + L.qsl_off); act = nullptr; }      // the quantiser has written the operand
    if (act) pib_launch(tg_xhat_kernel, dim3((unsigned) ((n16 + 255) / 256)), dim3(256), 0, st, (const int8_t *) (act + L.qs_off), (const float *) (act + L.d_off), n16, (int) (w->K / 16), xh);
    PIB_CHECK(cudaGetLastError());
    const tg_plan p = tg_plan_of(w->N, w->K, b);
    const int NB = tg_nb_of(b);
    auto go = [&](int x0, int n, int S) {
        if (p.G == 1)
            switch (NB) {
                case 32: return tg_launch<32, 1>(w, xh, b, x0, n, S, y_dev, st);
                case 64: return tg_launch<64, 1>(w, xh, b, x0, n, S, y_dev, st);
                case 96: return tg_launch<96, 1>(w, xh, b, x0, n, S, y_dev, st);
                default: return tg_launch<128, 1>(w, xh, b, x0, n, S, y_dev, st);
            }
        switch (NB) {
            case 32:  return tg_launch<32, 2>(w, xh, b, x0, n, S, y_dev, st);
            case 64:  return tg_launch<64, 2>(w, xh, b, x0, n, S, y_dev, st);
            case 96:  return tg_launch<96, 2>(w, xh, b, x0, n, S, y_dev, st);
            case 128: return tg_launch<128, 2>(w, xh, b, x0, n, S, y_dev, st);
            case 192: return tg_launch<192, 2>(w, xh, b, x0, n, S, y_dev, st);
            default:  return tg_launch<256, 2>(w, xh, b, x0, n, S, y_dev, st);
        }
    };
    int rc = PIB_OK;
    if (p.full > 0) rc = go(0, p.full, p.s_full);
    if (rc == PIB_OK && p.rest > 0) rc = go(p.full, p.rest, p.s_rest);
    return rc;
}

extern "C" size_t pib_gemm_scratch_bytes(int64_t K, int b) { return pib_gemm_xhat_bytes(K, b); }
extern "C" int pib_gemm(const pib_weight * w, const void * act_dev, int b, float * y_dev, void * scratch_dev, pib_stream s) {
    if (!act_dev || !y_dev || !scratch_dev || b > 256) { pib_set_error("pib_gemm: bad arguments"); return PIB_ERR_ARG; }
    return pib_gemm_q4k_tc(w, act_dev, b, y_dev, scratch_dev, (cudaStream_t) s);
}
extern "C" int pib_gemm_check(pib_stream s) { return pib_tc_check((cudaStream_t) s); }
// activation quantiser for any number of rows (pib_quantize_act is limited to verification batches)
extern "C" int pib_quantize_act_rows(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, pib_stream s);

int pib_quantize_act_c(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, const int * cancel, cudaStream_t st, void * xhat = nullptr, bool lean = false);

// host-buffer convenience for the parity tests (like pib_mul_mat_host): x_host [b][K] fp32 -> y_host [b][N]
extern "C" int pib_gemm_host(const pib_weight * w, const float * x_host, int b, float * y_host) {
    if (!w || b < 1 || b > 256) { pib_set_error("pib_gemm_host: bad arguments"); return PIB_ERR_ARG; }
    const size_t xb = (size_t) b * w->K * 4, yb = (size_t) b * w->N * 4, ab = pib_act_bytes(PIB_TYPE_Q4_K, w->K, b), hb = pib_gemm_xhat_bytes(w->K, b);
    uint8_t * buf = nullptr;
    PIB_CHECK(cudaMalloc(&buf, xb + yb + ab + hb + 4096));
    auto al = [](size_t v) { return (v + 1023) & ~(size_t) 1023; };
    float * x = (float *) buf;
    float * y = (float *) (buf + al(xb));
    void *  act = buf + al(xb) + al(yb);
    void *  xh = buf + al(xb) + al(yb) + al(ab);
    int rc = PIB_OK;
    if (cudaMemcpy(x, x_host, xb, cudaMemcpyHostToDevice) != cudaSuccess) rc = PIB_ERR_CUDA;
    // the activation quantiser takes at most PIB_MAX_BATCH rows per launch; its planes are per launch, so quantise in one go
    // through the engine-internal entry point (any b)
    if (rc == PIB_OK) rc = pib_quantize_act_c(PIB_TYPE_Q4_K, x, b, w->K, act, nullptr, nullptr);
    if (rc == PIB_OK && (rc = pib_gemm_q4k_tc(w, act, b, y, xh, nullptr)) != PIB_OK) { cudaFree(buf); return rc; }
    if (rc == PIB_OK && (rc = pib_tc_check(nullptr)) != PIB_OK) { cudaFree(buf); return rc; }
    if (rc == PIB_OK && cudaMemcpy(y_host, y, yb, cudaMemcpyDeviceToHost) != cudaSuccess) rc = PIB_ERR_CUDA;
    if (rc == PIB_ERR_CUDA) pib_set_error("pib_gemm_host: %s", cudaGetErrorString(cudaGetLastError()));
    cudaFree(buf);
    return rc;
}

extern "C" int pib_quantize_act_rows(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, pib_stream s) {
    if (b < 1 || b > 256) { pib_set_error("pib_quantize_act_rows: 1 <= b <= 256"); return PIB_ERR_ARG; }
    return pib_quantize_act_c(wtype, x_dev, b, K, act_dev, nullptr, (cudaStream_t) s);
}
