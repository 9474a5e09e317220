// dense_mm.cu -- matmuls with dense (unquantised) weights: Y[m][n] = sum_k X[m][k] * W[n][k], weights bfloat16 or float32 rows.
//
// Two arithmetic modes, chosen per call:
//   * served mode: X is rounded to bfloat16 when it is staged (the operand precision of the tensor cores), W is bfloat16, every
//     product is accumulated in fp32;
//   * exact mode: W float32, X float32, fmaf chains in k order -- true 32-bit, no reduced-precision matrix mode.
// One launch covers Z independent problems (heads of an attention layer, experts of a mixture) that differ by constant
// strides; with `zrange` problem z owns a run of rows of a sorted list (tokens grouped by expert) and rows may be gathered
// through an index list.
//
// Kernels: mm_tile_kernel (any shape; 64 x 64 x 16 tiles, 4 x 4 outputs per thread), for up to MV_MAXB rows mv_mma_kernel (bfloat16 weights: 16 weight rows
// per block against all tokens on the tensor cores) or mv_rows_kernel (float32 weights, shapes the former does not take: one warp per weight row), and for up
// to 128 float32 outputs
// over many rows mm_few_cols_kernel (a warp per four rows: a router's logits, where 64-wide output tiles would leave most of the machine idle).
#include "hybrid.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#define MM_BM 64
#define MM_BN 64
#define MM_BK 16
#define MV_MAXB 16

__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float ld_w(const float * p) { return *p; }
__device__ __forceinline__ float ld_w(const __nv_bfloat16 * p) { return __bfloat162float(*p); }

struct mm_dev {
    const void * W; int64_t ldw, wz;
    const float * X; int64_t ldx, xz; const int32_t * xrows; int xdiv;
    float * Y; int64_t ldy, yz;
    int M, N, K;
    const int32_t * zrange;
    float e0, e1;
    const int32_t * zlist;
    float * Y2; int64_t ld2; int n2; const int32_t * rows2;      // outputs n >= n2: Y2[rows2[m] * ld2 + n - n2]
    int w_made;                                                  // W comes from an earlier launch (pib_mm)
};
__device__ __forceinline__ float * mm_out(const mm_dev & a, float * Y, int m, int n) { return n >= a.n2 ? a.Y2 + (size_t) a.rows2[m] * a.ld2 + (n - a.n2) : Y + (size_t) m * a.ldy + n; }

template <typename WT, bool ROUND, int EPI>
__global__ void __launch_bounds__(256) mm_tile_kernel(mm_dev a) {
    pib_pdl_wait();
    pib_pdl_trigger();
    const int z = blockIdx.z;
    int row0 = 0, row1 = a.M;
    if (a.zrange) { row0 = a.zrange[z]; row1 = a.zrange[z + 1]; }
    const int m0 = row0 + blockIdx.x * MM_BM;
    if (m0 >= row1) return;
    const int n0 = blockIdx.y * MM_BN;
    const WT *    W = reinterpret_cast<const WT *>(a.W) + (size_t) z * a.wz;
    const float * X = a.X + (size_t) z * a.xz;
    float *       Y = a.Y + (size_t) z * a.yz;
    __shared__ float Xs[MM_BK][MM_BM + 4];
    __shared__ float Ws[MM_BK][MM_BN + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    // rows this thread stages: element (r, kk) with kk = tid % 16, r = tid / 16 + 16 * l
    int64_t xoff[4];
    bool    xok[4], wok[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const int r = (tid >> 4) + 16 * l;
        const int m = m0 + r;
        xok[l] = m < row1;
        const int src = xok[l] ? (a.xrows ? a.xrows[m] / a.xdiv : m) : 0;
        xoff[l] = (int64_t) src * a.ldx;
        wok[l] = n0 + r < a.N;
    }
    const int kk = tid & 15;
    for (int k0 = 0; k0 < a.K; k0 += MM_BK) {
        const bool kok = k0 + kk < a.K;
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const int r = (tid >> 4) + 16 * l;
            float xv = (xok[l] && kok) ? X[xoff[l] + k0 + kk] : 0.f;
            if (ROUND) xv = round_bf16(xv);
            Xs[kk][r] = xv;
            Ws[kk][r] = (wok[l] && kok) ? ld_w(W + (size_t) (n0 + r) * a.ldw + k0 + kk) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MM_BK; k++) {
            float xa[4], wb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) xa[i] = Xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) wb[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(xa[i], wb[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty * 4 + i;
        if (m >= row1) continue;
        if (pib_epi_pairs(EPI)) {
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int n = n0 + tx * 4 + j;
                if (n + 1 < a.N) Y[(size_t) m * a.ldy + (n >> 1)] = pib_glu_pair<EPI, ROUND>(acc[i][j], acc[i][j + 1], a.e0);
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n >= a.N) continue;
            *mm_out(a, Y, m, n) = pib_epilogue<EPI, ROUND>(acc[i][j], a.e0, a.e1);
        }
    }
}

// ---- few rows (decoding): one warp per weight row n, lanes stride over k in 16-byte pieces, B <= MV_MAXB rows of X at once ----
template <typename WT> struct wvec;
template <> struct wvec<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static void load(const __nv_bfloat16 * p, float * o) {
        const int4 r = ld_stream_v4(p);
        const uint32_t u[4] = { (uint32_t) r.x, (uint32_t) r.y, (uint32_t) r.z, (uint32_t) r.w };
#pragma unroll
        for (int i = 0; i < 4; i++) { o[2 * i] = __uint_as_float(u[i] << 16); o[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
    }
};
template <> struct wvec<float> {
    static constexpr int N = 4;
    __device__ static void load(const float * p, float * o) {
        const int4 r = ld_stream_v4(p);
        o[0] = __int_as_float(r.x); o[1] = __int_as_float(r.y); o[2] = __int_as_float(r.z); o[3] = __int_as_float(r.w);
    }
};

// the rows [row0, row1) of problem z (at most B of them) against weight row n
template <typename WT, bool ROUND, int EPI, int B>
__device__ __forceinline__ void mv_rows_body(const mm_dev & a, bool xvec, int z, int n, int lane, int row0, int row1) {
    constexpr int NR = pib_epi_pairs(EPI) ? 2 : 1;        // paired outputs: the warp walks the pair's two weight rows one after the other
    const float * X = a.X + (size_t) z * a.xz;
    float *       Y = a.Y + (size_t) z * a.yz;
    constexpr int V = wvec<WT>::N;
    const float * xr[B];
#pragma unroll
    for (int b = 0; b < B; b++) {
        const int m = row0 + b < row1 ? row0 + b : row0;
        xr[b] = X + (int64_t) (a.xrows ? a.xrows[m] / a.xdiv : m) * a.ldx;
    }
    float res[NR][B];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const WT * W = reinterpret_cast<const WT *>(a.W) + (size_t) z * a.wz + (size_t) (n * NR + r) * a.ldw;
        float acc[B];
#pragma unroll
        for (int b = 0; b < B; b++) acc[b] = 0.f;
        const int Kv = a.K - a.K % V;
        // few rows: the loop is bound by the weight bytes a warp has in flight, so more trips are opened at once
#pragma unroll (B <= 2 ? 4 : 2)
        for (int k = lane * V; k < Kv; k += 32 * V) {
            float w[V];
            wvec<WT>::load(W + k, w);
#pragma unroll
            for (int b = 0; b < B; b++) {
                float xv[V];
                if (xvec) {             // rows of X start on 16-byte boundaries (checked on the host): 128-bit loads
#pragma unroll
                    for (int i = 0; i < V; i += 4) *reinterpret_cast<float4 *>(xv + i) = *reinterpret_cast<const float4 *>(xr[b] + k + i);
                } else {
#pragma unroll
                    for (int i = 0; i < V; i++) xv[i] = xr[b][k + i];
                }
#pragma unroll
                for (int i = 0; i < V; i++) acc[b] = fmaf(ROUND ? round_bf16(xv[i]) : xv[i], w[i], acc[b]);
            }
        }
        for (int k = Kv + lane; k < a.K; k += 32) {
            const float w = ld_w(W + k);
#pragma unroll
            for (int b = 0; b < B; b++) { float xv = xr[b][k]; if (ROUND) xv = round_bf16(xv); acc[b] = fmaf(xv, w, acc[b]); }
        }
#pragma unroll
        for (int b = 0; b < B; b++) res[r][b] = warp_sum(acc[b]);
    }
#pragma unroll
    for (int b = 0; b < B; b++) {
        if (lane == 0 && row0 + b < row1)
            *mm_out(a, Y, row0 + b, n) = pib_epi_pairs(EPI) ? pib_glu_pair<EPI, ROUND>(res[0][b], res[NR - 1][b], a.e0) : pib_epilogue<EPI, ROUND>(res[0][b], a.e0, a.e1);
    }
}

// B = the most rows any problem can own (the batch's total).  A grouped problem (zrange) usually owns fewer -- an expert of a decode
// step has one or two of the batch's pairs -- and takes the instance that fits its own count, so that it stays bound by its weights' bytes
// and not by B times the arithmetic.  Every row's sum is formed in the same order whichever instance runs.
template <typename WT, bool ROUND, int EPI, int B>
__device__ __forceinline__ void mv_rows_fit(const mm_dev & a, bool xvec, int z, int n, int lane, int row0, int row1) {
    const int cnt = row1 - row0;
    if (B > 1 && cnt == 1)               mv_rows_body<WT, ROUND, EPI, 1>(a, xvec, z, n, lane, row0, row1);
    else if (B > 2 && cnt <= 2)          mv_rows_body<WT, ROUND, EPI, 2>(a, xvec, z, n, lane, row0, row1);
    else if (B > 4 && cnt <= 4)          mv_rows_body<WT, ROUND, EPI, (B > 4 ? 4 : B)>(a, xvec, z, n, lane, row0, row1);
    else if (B > 8 && cnt <= 8)          mv_rows_body<WT, ROUND, EPI, (B > 8 ? 8 : B)>(a, xvec, z, n, lane, row0, row1);
    else                                 mv_rows_body<WT, ROUND, EPI, B>(a, xvec, z, n, lane, row0, row1);
}
// the problem of grid place iz: the iz-th one that has rows (zlist), or iz itself; false when there is nothing to do
__device__ __forceinline__ bool mv_problem(const mm_dev & a, int iz, int B, int & z, int & row0, int & row1) {
    z = iz; row0 = 0; row1 = a.M;
    if (a.zlist) { if (iz >= a.zlist[0]) return false; z = a.zlist[1 + iz]; }
    if (a.zrange) { row0 = a.zrange[z]; row1 = a.zrange[z + 1]; }
    if (row1 - row0 > B) row1 = row0 + B;            // the host only picks these kernels when every z has at most B rows
    return row0 < row1;
}
template <typename WT, bool ROUND, int EPI, int B>
__global__ void __launch_bounds__(256) mv_rows_kernel(mm_dev a, bool xvec) {
    pib_pdl_wait();
    pib_pdl_trigger();
    int z, row0, row1;
    if (!mv_problem(a, blockIdx.z, B, z, row0, row1)) return;
    const int lane = threadIdx.x & 31, n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (n >= (pib_epi_pairs(EPI) ? a.N / 2 : a.N)) return;
    if (a.zrange) mv_rows_fit<WT, ROUND, EPI, B>(a, xvec, z, n, lane, row0, row1);
    else          mv_rows_body<WT, ROUND, EPI, B>(a, xvec, z, n, lane, row0, row1);
}
// a grouped problem and a plain one in one launch: blocks [0, za * blocks_a) walk the weight rows of a's problems with rows, the others b's
template <typename WT, bool ROUND, int EPI, int B>
__global__ void __launch_bounds__(256) mv_experts_kernel(mm_dev a, mm_dev b, bool xva, bool xvb, int blocks_a, int za) {
    pib_pdl_wait();
    pib_pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = blockDim.x >> 5, blk = blockIdx.x - blocks_a * za;
    int z, row0, row1;
    if (blk < 0) {
        const int n = ((int) blockIdx.x % blocks_a) * per + warp;
        if (!mv_problem(a, blockIdx.x / blocks_a, B, z, row0, row1) || n >= (pib_epi_pairs(EPI) ? a.N / 2 : a.N)) return;
        mv_rows_fit<WT, ROUND, EPI, B>(a, xva, z, n, lane, row0, row1);
    } else {
        const int n = blk * per + warp;
        if (n < (pib_epi_pairs(EPI) ? b.N / 2 : b.N)) mv_rows_fit<WT, ROUND, EPI, B>(b, xvb, 0, n, lane, 0, b.M);
    }
}

// two independent few-row matmuls in one launch (decode steps: a launch costs as much as a small matrix): blocks [0, blocks_a) walk a's weight rows,
// the others b's
template <typename WT, bool ROUND, int EPI_B, int B>
__global__ void __launch_bounds__(256) mv_pair_kernel(mm_dev a, mm_dev b, bool xva, bool xvb, int blocks_a) {
    pib_pdl_wait();
    pib_pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = blockDim.x >> 5;
    if ((int) blockIdx.x < blocks_a) {
        const int n = blockIdx.x * per + warp;
        if (n < a.N) mv_rows_body<WT, ROUND, PIB_EPI_NONE, B>(a, xva, 0, n, lane, 0, a.M);
    } else {
        const int n = (blockIdx.x - blocks_a) * per + warp;
        if (n < (pib_epi_pairs(EPI_B) ? b.N / 2 : b.N)) mv_rows_body<WT, ROUND, EPI_B, B>(b, xvb, 0, n, lane, 0, b.M);
    }
}

// ---- few rows, bfloat16 weights: 16 weight rows x up to 16 tokens per block on the tensor cores (mma.sync, fp32 accumulators) ----
// The eight warps of a block share K; a lane's 16-byte piece of a weight row (k = 32 c + 8 t .. + 7, t = lane % 4) is the A operand of two products as it
// is: k slots 2t, 2t + 1 and 2t + 8, 2t + 9 of product j stand for elements 8t + 4j .. + 3, and the lane reads the same eight elements of "its" token for B.
// So no value passes through shared memory, an activation is rounded once per block, and a warp's weight bytes are all in flight together -- the first ones
// before the launch wait where W is a weight, which nothing writes (not for the key and value rows that an attention gathers and passes as W: pib_mm.w_made).
// The tensor core cuts what falls off its accumulator, always towards zero, so every product of 16 k starts from none and is added up here, rounded to nearest: one
// accumulator for all of a warp's k drifted (error against 64 bits 2.4e-7 at K = 2048, 2.1e-6 at 16384; now 8.5e-8 and 1.7e-7, fused multiply-adds 8.0e-8 and 1.7e-7).
// What bounds it: the weights' way from memory.  The form it replaced (a warp per weight row, mv_rows_kernel) rounded every activation for every weight row: at
// four tokens 32 conversions per 16 bytes of weights (5632 x 2048, 1 / 4 / 16 tokens: 5.8 / 6.1 / 9.1 us, at four 21.7 before).
// Weights wait in shared memory: a warp asks for MVM_U chunks of 32 k at a time and DEPTH such groups at once (a lane copies what it reads back itself).  In registers one group was in
// flight, and each trip paid memory's latency and then the activations'.  How deep: as many bytes as an SM's CTAs can hold (launch_mm).
#define MVM_U 4                      // 32-k chunks of a group
#define MVM_GROUP (MVM_U * 1024)     // bytes of a group and warp: 16 rows x 64 bytes a chunk
__device__ __forceinline__ void mvm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t mvm_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
// weight rows 16 tile .. + 15 of problem z against its rows [row0, row1) (at most 8 NT).  WAIT: the launch wait comes here, behind the first loads of immutable weights
template <int EPI, int NT, int DEPTH, bool WAIT>
__device__ __forceinline__ void mvm_body(const mm_dev & a, int z, int tile, int row0, int row1) {
    __shared__ float red[8][8 * NT][16];
    extern __shared__ __align__(16) uint8_t mvm_ring[];
    constexpr int D = DEPTH ? DEPTH : 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nch = (a.K + 31) / 32, c0 = nch * warp / 8, c1 = nch * (warp + 1) / 8, n0 = tile * 16, groups = (c1 - c0 + MVM_U - 1) / MVM_U;
    const __nv_bfloat16 * W = reinterpret_cast<const __nv_bfloat16 *>(a.W) + (size_t) z * a.wz + 8 * t;
    const __nv_bfloat16 * wa = W + (size_t) min(n0 + g, a.N - 1) * a.ldw, * wb = W + (size_t) min(n0 + g + 8, a.N - 1) * a.ldw;
    const uint8_t * own  = mvm_ring + warp * (D * MVM_GROUP) + lane * 16;
    const uint32_t  ring = (uint32_t) __cvta_generic_to_shared(own);
    auto issue = [&](int q) {                                               // group q of this warp into place q mod DEPTH; pieces past the end become zeros and are not read
        if (q < groups) {
#pragma unroll
            for (int u = 0; u < MVM_U; u++) {
                const int  c  = c0 + q * MVM_U + u;
                const bool in = c < c1 && c * 32 + 8 * t < a.K;
                const uint32_t dst = ring + (uint32_t) (q % D) * MVM_GROUP + u * 1024, bytes = in ? 16u : 0u;
                const __nv_bfloat16 * pa = in ? wa + c * 32 : reinterpret_cast<const __nv_bfloat16 *>(a.W), * pb = in ? wb + c * 32 : pa;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(pa), "r"(bytes) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 512), "l"(pb), "r"(bytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int4 ra[MVM_U], rb[MVM_U];                                              // DEPTH 0: one group, in registers
    auto load = [&](int q) {
#pragma unroll
        for (int u = 0; u < MVM_U; u++) {
            const int  c  = c0 + q * MVM_U + u;
            const bool in = c < c1 && c * 32 + 8 * t < a.K;
            ra[u] = in ? ld_stream_v4(wa + c * 32) : make_int4(0, 0, 0, 0);
            rb[u] = in ? ld_stream_v4(wb + c * 32) : make_int4(0, 0, 0, 0);
        }
    };
    if (WAIT && a.w_made) pib_pdl_wait();
    if (DEPTH == 0) load(0);
#pragma unroll
    for (int q = 0; q < DEPTH; q++) issue(q);
    if (WAIT) { pib_pdl_wait(); pib_pdl_trigger(); }      // a second wait returns at once
    const float * x[NT];
    bool          has[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int m = row0 + g + 8 * j;
        has[j] = m < row1;
        x[j]   = a.X + (size_t) z * a.xz + (int64_t) (has[j] ? (a.xrows ? a.xrows[m] / a.xdiv : m) : 0) * a.ldx + 8 * t;
    }
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    for (int q = 0; q < groups; q++) {
        const int c = c0 + q * MVM_U;
        constexpr int XU = DEPTH ? MVM_U : 1;                               // DEPTH: the group's activations in flight together, in front of the wait for its weights
        float4 xa[NT][XU], xb[NT][XU];
        auto load_x = [&](int u, int k) {
            const bool in = c + u < c1 && (c + u) * 32 + 8 * t < a.K;
#pragma unroll
            for (int j = 0; j < NT; j++) {
                xa[j][k] = xb[j][k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in && has[j]) { xa[j][k] = *reinterpret_cast<const float4 *>(x[j] + (c + u) * 32); xb[j][k] = *reinterpret_cast<const float4 *>(x[j] + (c + u) * 32 + 4); }
            }
        };
        if (DEPTH) {
#pragma unroll
            for (int u = 0; u < MVM_U; u++) load_x(u, u % XU);
        }
        if (DEPTH == 0) { if (q) load(q); }
        else asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        const uint8_t * place = own + (q % D) * MVM_GROUP;
#pragma unroll
        for (int u = 0; u < MVM_U; u++) {
            if (DEPTH == 0) load_x(u, 0);
            if (DEPTH) { ra[u] = *reinterpret_cast<const int4 *>(place + u * 1024); rb[u] = *reinterpret_cast<const int4 *>(place + u * 1024 + 512); }
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const float4 p = xa[j][u % XU], r = xb[j][u % XU];
                float c4[4] = { 0.f, 0.f, 0.f, 0.f }, d4[4] = { 0.f, 0.f, 0.f, 0.f };
                mvm_mma(c4, (uint32_t) ra[u].x, (uint32_t) rb[u].x, (uint32_t) ra[u].y, (uint32_t) rb[u].y, mvm_pack(p.x, p.y), mvm_pack(p.z, p.w));
                mvm_mma(d4, (uint32_t) ra[u].z, (uint32_t) rb[u].z, (uint32_t) ra[u].w, (uint32_t) rb[u].w, mvm_pack(r.x, r.y), mvm_pack(r.z, r.w));
#pragma unroll
                for (int e = 0; e < 4; e++) acc[j][e] += c4[e] + d4[e];
            }
        }
        if (DEPTH) {
            __syncwarp();                                                   // the place has been read (by the lanes that fill it)
            issue(q + DEPTH);
        }
    }
    if (DEPTH) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int j = 0; j < NT; j++) {
        red[warp][8 * j + 2 * t][g]     = acc[j][0]; red[warp][8 * j + 2 * t + 1][g]     = acc[j][1];
        red[warp][8 * j + 2 * t][g + 8] = acc[j][2]; red[warp][8 * j + 2 * t + 1][g + 8] = acc[j][3];
    }
    __syncthreads();
    const int m = threadIdx.x >> 4, r = threadIdx.x & 15, n = n0 + r;
    if (m >= 8 * NT) return;                                                // whole warps: a warp holds two tokens
    float v = red[0][m][r];
#pragma unroll
    for (int w = 1; w < 8; w++) v += red[w][m][r];
    const float o = pib_epi_pairs(EPI) ? __shfl_down_sync(0xffffffffu, v, 1) : 0.f;      // paired outputs: rows 2i, 2i + 1 sit in neighbouring lanes
    if (row0 + m >= row1) return;
    float * Y = a.Y + (size_t) z * a.yz;
    if (pib_epi_pairs(EPI)) { if (!(r & 1) && n + 1 < a.N) *mm_out(a, Y, row0 + m, n >> 1) = pib_glu_pair<EPI, true>(v, o, a.e0); }
    else if (n < a.N) *mm_out(a, Y, row0 + m, n) = pib_epilogue<EPI, true>(v, a.e0, a.e1);
}
template <int EPI, int NT, int DEPTH>
__global__ void __launch_bounds__(256, DEPTH >= 5 ? 1 : (NT == 2 && DEPTH) || DEPTH >= 3 ? 2 : 3) mv_mma_kernel(mm_dev a) {
    if (!a.zrange && !a.zlist) { mvm_body<EPI, NT, DEPTH, true>(a, blockIdx.z, blockIdx.x, 0, a.M); return; }
    pib_pdl_wait();
    pib_pdl_trigger();
    int z, row0, row1;
    if (mv_problem(a, blockIdx.z, 8 * NT, z, row0, row1)) mvm_body<EPI, NT, DEPTH, false>(a, z, blockIdx.x, row0, row1);
}
// mv_experts_kernel's and mv_pair_kernel's work in this form
template <int EPI, int NT>
__global__ void __launch_bounds__(256, NT == 2 ? 2 : 3) mv_mma_experts_kernel(mm_dev a, mm_dev b, int tiles_a, int za) {
    const int blk = blockIdx.x - tiles_a * za;
    if (blk >= 0) { mvm_body<EPI, NT, 2, true>(b, 0, blk, 0, b.M); return; }
    pib_pdl_wait();
    pib_pdl_trigger();
    int z, row0, row1;
    if (mv_problem(a, blockIdx.x / tiles_a, 8 * NT, z, row0, row1)) mvm_body<EPI, NT, 2, false>(a, z, (int) blockIdx.x % tiles_a, row0, row1);
}
template <int EPI_B, int NT, int DEPTH>
__global__ void __launch_bounds__(256, NT == 2 && DEPTH ? 2 : 3) mv_mma_pair_kernel(mm_dev a, mm_dev b, int tiles_a) {
    if ((int) blockIdx.x < tiles_a) mvm_body<PIB_EPI_NONE, NT, DEPTH, true>(a, 0, blockIdx.x, 0, a.M);
    else                            mvm_body<EPI_B, NT, DEPTH, true>(b, 0, blockIdx.x - tiles_a, 0, b.M);
}
// whether one group of weights in registers is the better form of a launch (the figures: launch_mm); a warp has `need` groups at most
static int  mvm_groups(int K) { return ((K + 31) / 32 + 8 * MVM_U - 1) / (8 * MVM_U); }
static bool mvm_registers(long long ctas, int need, int M) { const long long sms = pib_num_sms(); return ctas > 2 * sms && (need == 1 || (M > 8 && ctas <= 3 * sms)); }
// bfloat16 weights whose 16-byte pieces and the activations' lie on 16-byte boundaries (the caller has looked at the weights)
template <typename WT, bool ROUND> static bool mvm_fits(const mm_dev & a, bool xvec) { return std::is_same<WT, __nv_bfloat16>::value && ROUND && xvec && a.K % 8 == 0; }

// ---- few outputs, many rows (a router's logits over a prompt): a warp takes FC_ROWS rows of X and NB outputs, lanes stride over k in 16-byte pieces ----
// float32 weights and activations, no rounding.  A weight piece is used for FC_ROWS rows, so the matrix crosses L1 once per that many rows; grid.y walks the
// outputs in runs of NB.
#define FC_ROWS 4
template <int NB, bool VEC>
__global__ void __launch_bounds__(128) mm_few_cols_kernel(mm_dev a) {
    pib_pdl_wait();
    pib_pdl_trigger();
    const int lane = threadIdx.x & 31, m0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * FC_ROWS, n0 = blockIdx.y * NB;
    if (m0 >= a.M) return;
    const float * W = reinterpret_cast<const float *>(a.W) + (size_t) n0 * a.ldw;
    const int nn = min(NB, a.N - n0);
    const float * x[FC_ROWS];
#pragma unroll
    for (int r = 0; r < FC_ROWS; r++) x[r] = a.X + (size_t) min(m0 + r, a.M - 1) * a.ldx;
    float acc[FC_ROWS][NB];
#pragma unroll
    for (int r = 0; r < FC_ROWS; r++)
#pragma unroll
        for (int n = 0; n < NB; n++) acc[r][n] = 0.f;
    if (VEC) {
        for (int k = lane * 4; k < a.K; k += 128) {
            float4 xv[FC_ROWS];
#pragma unroll
            for (int r = 0; r < FC_ROWS; r++) xv[r] = *reinterpret_cast<const float4 *>(x[r] + k);
#pragma unroll
            for (int n = 0; n < NB; n++) {
                const float4 w = *reinterpret_cast<const float4 *>(W + (size_t) min(n, nn - 1) * a.ldw + k);      // no branch: the loads of a trip are in flight together
#pragma unroll
                for (int r = 0; r < FC_ROWS; r++) acc[r][n] = fmaf(xv[r].w, w.w, fmaf(xv[r].z, w.z, fmaf(xv[r].y, w.y, fmaf(xv[r].x, w.x, acc[r][n]))));
            }
        }
    } else {
        for (int k = lane; k < a.K; k += 32) {
            float xv[FC_ROWS];
#pragma unroll
            for (int r = 0; r < FC_ROWS; r++) xv[r] = x[r][k];
#pragma unroll
            for (int n = 0; n < NB; n++) {
                const float w = W[(size_t) min(n, nn - 1) * a.ldw + k];
#pragma unroll
                for (int r = 0; r < FC_ROWS; r++) acc[r][n] = fmaf(xv[r], w, acc[r][n]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < FC_ROWS; r++)
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const float v = warp_sum(acc[r][n]);
            if (lane == 0 && n < nn && m0 + r < a.M) a.Y[(size_t) (m0 + r) * a.ldy + n0 + n] = v;
        }
}

template <typename K> static cudaError_t mvm_smem(pib_per_device & attrs, K kernel, size_t smem) {
    return attrs.once([&] {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int) cudaSharedmemCarveoutMaxShared);
    });
}
#define MVM_SMEM(DEPTH) ((size_t) 8 * (DEPTH) * MVM_GROUP)          // none: the group sits in registers
template <int EPI, int NT, int DEPTH> static int mvm_launch(dim3 grid, cudaStream_t st, const mm_dev & d) {
    static pib_per_device attrs;
    if (DEPTH) PIB_CHECK(mvm_smem(attrs, mv_mma_kernel<EPI, NT, DEPTH>, MVM_SMEM(DEPTH)));
    pib_launch(mv_mma_kernel<EPI, NT, DEPTH>, grid, dim3(256), MVM_SMEM(DEPTH), st, d);
    return PIB_OK;
}

template <typename WT, bool ROUND, int EPI>
static int launch_mm(const pib_mm & a, const mm_dev & d, cudaStream_t st) {
    const int  V = wvec<WT>::N;
    // the row kernel wants aligned 16-byte weight loads: row stride, z stride and base all multiples of the vector
    const bool vec_ok = a.ldw % V == 0 && a.wz % V == 0 && ((uintptr_t) a.W & 15) == 0;
    // few rows in all (with zrange: no problem z can own more than the total): a warp per weight row; problems without rows leave at once
    if (a.M <= MV_MAXB && vec_ok) {
        dim3 grid((unsigned) (((pib_epi_pairs(EPI) ? a.N / 2 : a.N) + 7) / 8), 1, (unsigned) (a.zlist && a.M < a.Z ? a.M : a.Z));
        const bool xvec = a.ldx % 4 == 0 && a.xz % 4 == 0 && ((uintptr_t) a.X & 15) == 0;
        if (mvm_fits<WT, ROUND>(d, xvec)) {
            grid.x = (unsigned) ((a.N + 15) / 16);
            // groups that a warp has at most, as far as the shared memory of one, two or more CTAs per SM holds them: what is not needed keeps the next launch's CTAs out
            // (us a launch, one group in registers / this: 2048 x 5632 at 1 / 4 / 16 tokens 10.0 10.5 19.9 / 6.2 6.4 8.8, 2048 x 2048 4.2 4.3 7.3 / 3.0 3.0 4.2, 8000 x 2048 9.8 10.4 17.6 /
            // 8.3 9.3 11.7; one group alone, at 4 / 9 / 16: 2048 x 1024 2.5 3.6 3.8 / 1.9 2.3 2.5, 3072 x 1024 3.0 4.2 4.5 / 2.4 2.9 3.6).  Registers where a group is all and two CTAs per
            // SM do not take all rows at once (32000 x 1024 at 8 tokens 15.8 / 18.2), and for 9 to 16 tokens where a round of three CTAs per SM, the registers' number, is enough and one
            // of two is not (5120 x 2048 at 16 9.0 / 9.9)
            const long long ctas = (long long) grid.x * grid.z, sms = pib_num_sms();
            const int need = mvm_groups(a.K), depth = std::min(need, ctas <= sms ? 5 : ctas <= 2 * sms ? 3 : 2);
#define MVM_GO(DEPTH) rc = a.M <= 8 ? mvm_launch<EPI, 1, DEPTH>(grid, st, d) : mvm_launch<EPI, 2, DEPTH>(grid, st, d)
            int rc;
            if (mvm_registers(ctas, need, a.M)) MVM_GO(0);
            else if (depth <= 1) MVM_GO(1); else if (depth == 2) MVM_GO(2); else if (depth == 3) MVM_GO(3); else MVM_GO(5);
#undef MVM_GO
            if (rc != PIB_OK) return rc;
        } else
        if (a.M == 1)      pib_launch(mv_rows_kernel<WT, ROUND, EPI, 1>, dim3(grid), dim3(256), (size_t) (0), st, d, xvec);
        else if (a.M == 2) pib_launch(mv_rows_kernel<WT, ROUND, EPI, 2>, dim3(grid), dim3(256), (size_t) (0), st, d, xvec);
        else if (a.M <= 4) pib_launch(mv_rows_kernel<WT, ROUND, EPI, 4>, dim3(grid), dim3(256), (size_t) (0), st, d, xvec);
        else if (a.M <= 8) pib_launch(mv_rows_kernel<WT, ROUND, EPI, 8>, dim3(grid), dim3(256), (size_t) (0), st, d, xvec);
        else               pib_launch(mv_rows_kernel<WT, ROUND, EPI, MV_MAXB>, dim3(grid), dim3(256), (size_t) (0), st, d, xvec);
    } else {
        dim3 grid((unsigned) ((a.M + MM_BM - 1) / MM_BM), (unsigned) ((a.N + MM_BN - 1) / MM_BN), (unsigned) a.Z);
        pib_launch(mm_tile_kernel<WT, ROUND, EPI>, dim3(grid), dim3(256), (size_t) (0), st, d);
    }
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

int pib_dense_mm_tc(const pib_mm & a, cudaStream_t st);     // dense_mma.cu: bfloat16 tensor-core tiles; PIB_ERR_UNSUPP when the shape does not fit

int pib_dense_mm(const pib_mm & a, cudaStream_t st) {
    if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.Z <= 0) return PIB_OK;
    if (a.exact && a.wtype != PIB_TYPE_F32) { pib_set_error("dense matmul: exact mode needs float32 weights"); return PIB_ERR_ARG; }
    if (a.Y2 && (a.Z != 1 || a.zrange || pib_epi_pairs(a.epi) || !a.rows2)) { pib_set_error("dense matmul: a second destination takes one plain problem and a row list"); return PIB_ERR_ARG; }
    if (a.wtype == PIB_TYPE_BF16 && !a.exact) {
        const int rc = pib_dense_mm_tc(a, st);
        if (rc != PIB_ERR_UNSUPP) return rc;
    }
    if (a.x_bf16 || a.y_bf16) { pib_set_error("dense matmul: bfloat16 activations need the tensor-core path (more than 16 rows, strides multiples of 8)"); return PIB_ERR_UNSUPP; }
    mm_dev d = { a.W, a.ldw, a.wz, a.X, a.ldx, a.xz, a.xrows, a.xdiv < 1 ? 1 : a.xdiv, a.Y, a.ldy, a.yz, a.M, a.N, a.K, a.zrange, a.e0, a.e1, a.zlist, a.Y2, a.ld2, a.Y2 ? a.n2 : 0x7fffffff, a.rows2, a.w_made };
    if (a.wtype == PIB_TYPE_F32 && a.exact && !a.Y2 && a.N <= 128 && a.M > MV_MAXB && a.Z == 1 && !a.xrows && !a.zrange && a.epi == PIB_EPI_NONE) {
        const int  NB = a.N <= 8 ? 8 : a.N <= 16 ? 16 : 24;
        const bool vec = a.K % 4 == 0 && a.ldw % 4 == 0 && a.ldx % 4 == 0 && (((uintptr_t) a.W | (uintptr_t) a.X) & 15) == 0;
        dim3 grid((unsigned) ((a.M + 4 * FC_ROWS - 1) / (4 * FC_ROWS)), (unsigned) ((a.N + NB - 1) / NB));
#define FC_GO(NB) do { if (vec) pib_launch(mm_few_cols_kernel<NB, true>, grid, dim3(128), (size_t) 0, st, d); else pib_launch(mm_few_cols_kernel<NB, false>, grid, dim3(128), (size_t) 0, st, d); } while (0)
        if (NB == 8) FC_GO(8); else if (NB == 16) FC_GO(16); else FC_GO(24);
#undef FC_GO
        PIB_CHECK(cudaGetLastError());
        return PIB_OK;
    }
    if (pib_epi_pairs(a.epi) && (a.N & 1)) { pib_set_error("dense matmul: paired outputs need an even number of weight rows"); return PIB_ERR_ARG; }
#define MM_GO(WT, ROUND) (a.epi == PIB_EPI_RELU2 ? launch_mm<WT, ROUND, PIB_EPI_RELU2>(a, d, st) : a.epi == PIB_EPI_XIELU ? launch_mm<WT, ROUND, PIB_EPI_XIELU>(a, d, st) : \
                          a.epi == PIB_EPI_GLU_PAIR ? launch_mm<WT, ROUND, PIB_EPI_GLU_PAIR>(a, d, st) : \
                          a.epi == PIB_EPI_GEGLU_PAIR ? launch_mm<WT, ROUND, PIB_EPI_GEGLU_PAIR>(a, d, st) : \
                          a.epi == PIB_EPI_SWIGLU_PAIR ? launch_mm<WT, ROUND, PIB_EPI_SWIGLU_PAIR>(a, d, st) : \
                                                    launch_mm<WT, ROUND, PIB_EPI_NONE>(a, d, st))
    if (a.wtype == PIB_TYPE_BF16) return MM_GO(__nv_bfloat16, true);
    if (a.wtype == PIB_TYPE_F32) return a.exact ? MM_GO(float, false) : MM_GO(float, true);
#undef MM_GO
    pib_set_error("dense matmul: weight type %d", a.wtype);
    return PIB_ERR_UNSUPP;
}

// a (no epilogue) and b (none or PIB_EPI_GEGLU_PAIR) do not depend on each other; up to MV_MAXB rows they share a launch, else they follow one another
template <typename WT, bool ROUND, int EPI_B>
static int launch_pair(const mm_dev & a, const mm_dev & b, bool xva, bool xvb, cudaStream_t st) {
    const int ba = (a.N + 7) / 8, bb = ((pib_epi_pairs(EPI_B) ? b.N / 2 : b.N) + 7) / 8;
    const dim3 grid((unsigned) (ba + bb));
    if (mvm_fits<WT, ROUND>(a, xva) && mvm_fits<WT, ROUND>(b, xvb)) {
        const int ta = (a.N + 15) / 16, tb = (b.N + 15) / 16;
        static pib_per_device one, two;
        // (one group, 1024 + 5632 rows x 1024 at 8 / 9 / 16 tokens: registers 4.0 5.2 5.4 us, shared memory 4.3 6.3 7.3)
        if (mvm_registers(ta + tb, mvm_groups(std::max(a.K, b.K)), a.M)) {
            if (a.M <= 8) pib_launch(mv_mma_pair_kernel<EPI_B, 1, 0>, dim3((unsigned) (ta + tb)), dim3(256), MVM_SMEM(0), st, a, b, ta);
            else          pib_launch(mv_mma_pair_kernel<EPI_B, 2, 0>, dim3((unsigned) (ta + tb)), dim3(256), MVM_SMEM(0), st, a, b, ta);
        } else {
            PIB_CHECK(a.M <= 8 ? mvm_smem(one, mv_mma_pair_kernel<EPI_B, 1, 2>, MVM_SMEM(2)) : mvm_smem(two, mv_mma_pair_kernel<EPI_B, 2, 2>, MVM_SMEM(2)));
            if (a.M <= 8) pib_launch(mv_mma_pair_kernel<EPI_B, 1, 2>, dim3((unsigned) (ta + tb)), dim3(256), MVM_SMEM(2), st, a, b, ta);
            else          pib_launch(mv_mma_pair_kernel<EPI_B, 2, 2>, dim3((unsigned) (ta + tb)), dim3(256), MVM_SMEM(2), st, a, b, ta);
        }
    } else
    if (a.M == 1)      pib_launch(mv_pair_kernel<WT, ROUND, EPI_B, 1>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba);
    else if (a.M == 2) pib_launch(mv_pair_kernel<WT, ROUND, EPI_B, 2>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba);
    else if (a.M <= 4) pib_launch(mv_pair_kernel<WT, ROUND, EPI_B, 4>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba);
    else if (a.M <= 8) pib_launch(mv_pair_kernel<WT, ROUND, EPI_B, 8>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba);
    else               pib_launch(mv_pair_kernel<WT, ROUND, EPI_B, MV_MAXB>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}
int pib_dense_mm_pair(const pib_mm & a, const pib_mm & b, cudaStream_t st) {
    const int V = a.wtype == PIB_TYPE_BF16 ? 8 : 4;
    auto plain = [&](const pib_mm & m) { return m.Z == 1 && !m.xrows && !m.zrange && !m.x_bf16 && !m.Y2 && m.ldw % V == 0 && ((uintptr_t) m.W & 15) == 0; };
    if (a.M < 1 || a.M > MV_MAXB || a.M != b.M || a.wtype != b.wtype || a.exact != b.exact || !plain(a) || !plain(b) || a.epi != PIB_EPI_NONE ||
        (b.epi != PIB_EPI_NONE && b.epi != PIB_EPI_GEGLU_PAIR) || (pib_epi_pairs(b.epi) && (b.N & 1)) || (a.exact && a.wtype != PIB_TYPE_F32)) {
        const int rc = pib_dense_mm(a, st);
        return rc != PIB_OK ? rc : pib_dense_mm(b, st);
    }
    auto dev = [](const pib_mm & m) { return mm_dev{ m.W, m.ldw, m.wz, m.X, m.ldx, m.xz, nullptr, 1, m.Y, m.ldy, m.yz, m.M, m.N, m.K, nullptr, m.e0, m.e1, nullptr, nullptr, 0, 0x7fffffff, nullptr, m.w_made }; };
    auto xvec = [](const pib_mm & m) { return m.ldx % 4 == 0 && ((uintptr_t) m.X & 15) == 0; };
#define PAIR_GO(WT, ROUND) (b.epi == PIB_EPI_NONE ? launch_pair<WT, ROUND, PIB_EPI_NONE>(dev(a), dev(b), xvec(a), xvec(b), st) \
                                                  : launch_pair<WT, ROUND, PIB_EPI_GEGLU_PAIR>(dev(a), dev(b), xvec(a), xvec(b), st))
    if (a.wtype == PIB_TYPE_BF16) return PAIR_GO(__nv_bfloat16, true);
    return a.exact ? PAIR_GO(float, false) : PAIR_GO(float, true);
#undef PAIR_GO
}

template <typename WT, bool ROUND, int EPI>
static int launch_experts(const mm_dev & a, const mm_dev & b, bool xva, bool xvb, int za, cudaStream_t st) {
    const int ba = ((pib_epi_pairs(EPI) ? a.N / 2 : a.N) + 7) / 8, bb = ((pib_epi_pairs(EPI) ? b.N / 2 : b.N) + 7) / 8, rows = a.M > b.M ? a.M : b.M;
    const dim3 grid((unsigned) (ba * za + bb));
    if (mvm_fits<WT, ROUND>(a, xva && a.xz % 4 == 0) && mvm_fits<WT, ROUND>(b, xvb)) {
        const int ta = (a.N + 15) / 16, tb = (b.N + 15) / 16;
        static pib_per_device one, two;
        PIB_CHECK(rows <= 8 ? mvm_smem(one, mv_mma_experts_kernel<EPI, 1>, MVM_SMEM(2)) : mvm_smem(two, mv_mma_experts_kernel<EPI, 2>, MVM_SMEM(2)));
        if (rows <= 8) pib_launch(mv_mma_experts_kernel<EPI, 1>, dim3((unsigned) (ta * za + tb)), dim3(256), MVM_SMEM(2), st, a, b, ta, za);
        else           pib_launch(mv_mma_experts_kernel<EPI, 2>, dim3((unsigned) (ta * za + tb)), dim3(256), MVM_SMEM(2), st, a, b, ta, za);
    } else
    if (rows == 1)      pib_launch(mv_experts_kernel<WT, ROUND, EPI, 1>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba, za);
    else if (rows == 2) pib_launch(mv_experts_kernel<WT, ROUND, EPI, 2>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba, za);
    else if (rows <= 4) pib_launch(mv_experts_kernel<WT, ROUND, EPI, 4>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba, za);
    else if (rows <= 8) pib_launch(mv_experts_kernel<WT, ROUND, EPI, 8>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba, za);
    else                pib_launch(mv_experts_kernel<WT, ROUND, EPI, MV_MAXB>, grid, dim3(256), (size_t) 0, st, a, b, xva, xvb, ba, za);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}
int pib_dense_mm_experts(const pib_mm & a, const pib_mm & b, cudaStream_t st) {
    const int V = a.wtype == PIB_TYPE_BF16 ? 8 : 4;
    auto fits = [&](const pib_mm & m) { return m.M >= 1 && m.M <= MV_MAXB && !m.x_bf16 && !m.Y2 && m.ldw % V == 0 && m.wz % V == 0 && ((uintptr_t) m.W & 15) == 0; };
    const bool epi_ok = a.epi == PIB_EPI_NONE || (a.epi == PIB_EPI_SWIGLU_PAIR && a.N % 2 == 0 && b.N % 2 == 0);
    if (!fits(a) || !fits(b) || !a.zrange || b.Z != 1 || b.zrange || b.xrows || a.wtype != b.wtype || a.exact != b.exact || a.epi != b.epi || !epi_ok || (a.exact && a.wtype != PIB_TYPE_F32)) {
        const int rc = pib_dense_mm(a, st);
        return rc != PIB_OK ? rc : pib_dense_mm(b, st);
    }
    auto dev = [](const pib_mm & m) {
        return mm_dev{ m.W, m.ldw, m.wz, m.X, m.ldx, m.xz, m.xrows, m.xdiv < 1 ? 1 : m.xdiv, m.Y, m.ldy, m.yz, m.M, m.N, m.K, m.zrange, m.e0, m.e1, m.zlist, nullptr, 0, 0x7fffffff, nullptr, m.w_made };
    };
    auto xvec = [](const pib_mm & m) { return m.ldx % 4 == 0 && ((uintptr_t) m.X & 15) == 0; };
    const int za = a.zlist && a.M < a.Z ? a.M : a.Z;
#define EXPERTS_GO(WT, ROUND) (a.epi == PIB_EPI_NONE ? launch_experts<WT, ROUND, PIB_EPI_NONE>(dev(a), dev(b), xvec(a), xvec(b), za, st) \
                                                     : launch_experts<WT, ROUND, PIB_EPI_SWIGLU_PAIR>(dev(a), dev(b), xvec(a), xvec(b), za, st))
    if (a.wtype == PIB_TYPE_BF16) return EXPERTS_GO(__nv_bfloat16, true);
    return a.exact ? EXPERTS_GO(float, false) : EXPERTS_GO(float, true);
#undef EXPERTS_GO
}

pib_weight * pib_dense_upload(int type, const void * host, int64_t N, int64_t K) {
    if ((type != PIB_TYPE_BF16 && type != PIB_TYPE_F32) || N <= 0 || K <= 0) { pib_set_error("dense weight: type %d, %lld x %lld", type, (long long) N, (long long) K); return nullptr; }
    pib_weight * w = (pib_weight *) calloc(1, sizeof(pib_weight));
    w->type = type; w->N = N; w->K = K;
    w->bytes = (size_t) N * K * (type == PIB_TYPE_BF16 ? 2 : 4);
    if (cudaMalloc(&w->base, w->bytes + 256) != cudaSuccess) {
        pib_set_error("dense weight: cudaMalloc of %zu bytes failed", w->bytes);
        cudaGetLastError(); free(w);
        return nullptr;
    }
    w->owns = 1;
    if (host && cudaMemcpy(w->base, host, w->bytes, cudaMemcpyHostToDevice) != cudaSuccess) {
        pib_set_error("dense weight: upload failed: %s", cudaGetErrorString(cudaGetLastError()));
        pib_weight_free(w);
        return nullptr;
    }
    return w;
}

// a producer of W that lets the launch behind it start at once and is late itself
__global__ void mm_late_copy_kernel(const uint4 * __restrict__ src, uint4 * __restrict__ dst, int n16) {
    pib_pdl_wait();
    pib_pdl_trigger();
    for (int i = 0; i < 200; i++) __nanosleep(1000);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += gridDim.x * blockDim.x) dst[i] = src[i];
}
// for the tests: Y[M][N] = X[M][K] W^T with W [N][K] (bfloat16 bits) written by the launch right in front of the matmul; K a multiple of 8
extern "C" int pib_dense_mm_made_host(const void * W, const float * X, float * Y, int M, int N, int K) {
    if (M < 1 || N < 1 || K < 8 || K % 8) { pib_set_error("dense matmul: bad arguments"); return PIB_ERR_ARG; }
    const size_t wb = (size_t) N * K * 2, xb = (size_t) M * K * 4, yb = (size_t) M * N * 4;
    uint8_t * src = nullptr, * dst = nullptr; float * dX = nullptr, * dY = nullptr;
    int rc = PIB_OK;
    if (cudaMalloc(&src, wb) != cudaSuccess || cudaMalloc(&dst, wb) != cudaSuccess || cudaMalloc(&dX, xb) != cudaSuccess || cudaMalloc(&dY, yb) != cudaSuccess) rc = PIB_ERR_NOMEM;
    if (rc == PIB_OK) {
        cudaMemcpy(src, W, wb, cudaMemcpyHostToDevice);
        cudaMemcpy(dX, X, xb, cudaMemcpyHostToDevice);
        cudaMemset(dst, 0, wb);
        pib_mm a;
        a.W = dst; a.ldw = K; a.X = dX; a.ldx = K; a.Y = dY; a.ldy = N; a.M = M; a.N = N; a.K = K; a.w_made = 1;
        // one block: the matmul's blocks find room beside it
        pib_launch(mm_late_copy_kernel, dim3(1), dim3(256), (size_t) 0, (cudaStream_t) nullptr, (const uint4 *) src, (uint4 *) dst, (int) (wb / 16));
        rc = pib_dense_mm(a, nullptr);
        if (rc == PIB_OK && cudaMemcpy(Y, dY, yb, cudaMemcpyDeviceToHost) != cudaSuccess) rc = PIB_ERR_CUDA;
    }
    for (void * p : { (void *) src, (void *) dst, (void *) dX, (void *) dY }) if (p) cudaFree(p);
    if (rc != PIB_OK) pib_set_error("dense matmul: %s", cudaGetErrorString(cudaGetLastError()));
    return rc;
}

// host-buffer convenience for the parity tests: every operand in host memory, shapes and strides as in pib_mm (elements).
// W: bfloat16 bits (wtype PIB_TYPE_BF16) or float32; zrange / xrows may be null; e0, e1: the epilogue's constants.
extern "C" int pib_dense_mm_host(int wtype, const void * W, int64_t w_elems, int64_t ldw, int64_t wz, const float * X, int64_t x_elems, int64_t ldx, int64_t xz,
                                 const int32_t * xrows, int xdiv, float * Y, int64_t y_elems, int64_t ldy, int64_t yz, int M, int N, int K, int Z,
                                 const int32_t * zrange, int epi, int exact, float e0, float e1) {
    const size_t wb = (size_t) w_elems * (wtype == PIB_TYPE_BF16 ? 2 : 4);
    void * dW = nullptr; float * dX = nullptr, * dY = nullptr; int32_t * dR = nullptr, * dZ = nullptr;
    int rc = PIB_OK;
    if (cudaMalloc(&dW, wb + 256) != cudaSuccess || cudaMalloc(&dX, (size_t) x_elems * 4 + 256) != cudaSuccess || cudaMalloc(&dY, (size_t) y_elems * 4 + 256) != cudaSuccess ||
        cudaMalloc(&dR, (size_t) M * 4 + 256) != cudaSuccess || cudaMalloc(&dZ, (size_t) (Z + 1) * 4 + 256) != cudaSuccess) rc = PIB_ERR_NOMEM;
    if (rc == PIB_OK) {
        cudaMemcpy(dW, W, wb, cudaMemcpyHostToDevice);
        cudaMemcpy(dX, X, (size_t) x_elems * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(dY, Y, (size_t) y_elems * 4, cudaMemcpyHostToDevice);
        if (xrows) cudaMemcpy(dR, xrows, (size_t) M * 4, cudaMemcpyHostToDevice);
        if (zrange) cudaMemcpy(dZ, zrange, (size_t) (Z + 1) * 4, cudaMemcpyHostToDevice);
        pib_mm a;
        a.W = dW; a.wtype = wtype; a.ldw = ldw; a.wz = wz; a.X = dX; a.ldx = ldx; a.xz = xz; a.xrows = xrows ? dR : nullptr; a.xdiv = xdiv;
        a.Y = dY; a.ldy = ldy; a.yz = yz; a.M = M; a.N = N; a.K = K; a.Z = Z; a.zrange = zrange ? dZ : nullptr; a.epi = epi; a.exact = exact; a.e0 = e0; a.e1 = e1;
        rc = pib_dense_mm(a, nullptr);
        if (rc == PIB_OK && cudaDeviceSynchronize() != cudaSuccess) { pib_set_error("dense matmul: %s", cudaGetErrorString(cudaGetLastError())); rc = PIB_ERR_CUDA; }
        if (rc == PIB_OK && wtype == PIB_TYPE_BF16 && !exact) rc = pib_tc_check(nullptr);
        if (rc == PIB_OK) cudaMemcpy(Y, dY, (size_t) y_elems * 4, cudaMemcpyDeviceToHost);
    } else pib_set_error("dense matmul: out of memory for the test buffers");
    for (void * p : { dW, (void *) dX, (void *) dY, (void *) dR, (void *) dZ }) if (p) cudaFree(p);
    return rc;
}
