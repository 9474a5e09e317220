// act_quant.cu -- activation quantisation (K2), fused with the producer that precedes each matmul (K4 / K8).
//
// The reference's CPU matmul first quantises every activation row to the weight type's "vec_dot type" (reference
// ggml.c:9493-9509): Q8_0 blocks for Q4_0 / Q8_0 weights (ggml-quants.c:632; on x86 the AVX2 branch :701-760:
// d = max|x| / 127 stored as fp16, q = round-half-even(x * (127 / max|x|))) and Q8_K super-blocks for Q4_K weights
// (ggml-quants.c:2329-2363: iscale = -128 / (signed value of the first max-|x| element), q = min(127, rne(iscale*x)),
// d = 1 / iscale, 16-wide bsums).  Greedy parity needs exactly this integer arithmetic, so it is reproduced bit for
// bit; only the layout differs (planes instead of blocks, see pib_act_layout in pib_common.cuh).
//
// A warp per 256 values of a row, eight neighbours per lane.  Prologues (template PRO):
//   PRO_PLAIN     v = x
//   PRO_RMSNORM   v = (x * 1/sqrtf(mean(x^2) + eps)) * w        (ggml.c:9028 with the double accumulator, then ggml_mul)
//   PRO_LAYERNORM v = (x - mean) * 1/sqrtf(var + eps) * w + b   (ggml.c:8959-9020, two double sums)
//   PRO_SILU_MUL  v = silu_f16lut(x) * x2                        (ggml.c:1490 table look-up, then ggml_mul; llama.cpp:3680)
//   PRO_GELU      v = gelu_f16lut(x)                             (ggml.c:1433; falcon MLP)
#include "pib_common.cuh"
#include "q8k_quant.cuh"

#include <algorithm>

enum { PRO_PLAIN = 0, PRO_RMSNORM = 1, PRO_SILU_MUL = 2, PRO_GELU = 3, PRO_LAYERNORM = 4 };

struct aq_args {
    const float *    x, * x2, * addend, * addend2, * bias;      // x2: norm weights, or the other factor of a gated product (x2_per_row)
    float *          sum_out, * vout;
    const uint16_t * lut;
    const int *      cancel;
    int64_t          K, xstride;
    double           inv_k;                                     // 1 / K where that is exact, else 0
    float            eps;
    int              per;                                       // units that a block quantises of a normed row
    int              x2_per_row, vec;                           // vec: every row of every operand starts on 16 bytes
    int8_t *         qs, * bs8, * qsp, * q6p, * b16;
    float *          d, * dxo;
    void *           bs;
    int2 *           qsl;
    int16_t *        sbs;
    __half *         xh;
};

__device__ __forceinline__ void aq_load8(const float * p, int vec, float (&v)[8]) {
    if (vec) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = p[j];
    }
}
__device__ __forceinline__ void aq_store8(float * p, int vec, const float (&v)[8]) {
    if (vec) {
        *reinterpret_cast<float4 *>(p)     = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) p[j] = v[j];
    }
}

// Grid: a row per blockIdx.x.  Without a norm the row's warps are spread over blockIdx.y.  With one, up to 32 warps of a block have the whole row in registers (longer rows take turns)
// and nothing is read twice; of a decode batch, blocks of eight units each (blockIdx.y) form the row's sum for themselves and quantise and write their own units: what a unit stores
// keeps an SM busy (4 rows of 8192: 3.4 us behind the wait with one block per row, 2.1 with four).
// The unit that a warp quantises stays in its registers from the sum on also where it is the warp's second of the row (with a matmul of 1712 rows, one token of 10240 9.65 -> 8.86 us, of 14848
// 12.0 -> 11.2; read again 0.6 us behind the sum otherwise).
// What bounds it: a chain of round trips behind the launch in front (operands 0.35 .. 0.6 us, the sum's two reductions and its barrier 0.3, the quants 0.25, their stores 0.4) and
// instructions that no earlier launch left in the cache (6 .. 9 clocks each).  Before (a warp's lanes on 32 neighbours for 32-element blocks, passes of up to four pieces per warp) / now,
// us that a launch adds to its chain: Q8_0 blocks, norm, 4 rows of 4096 4.6 / 2.7; Q8_K, norm, one row of 2048 3.2 / 2.8, plain 1.9 / 1.5; prompts of 700 rows, norm 4096 14.1 / 10.2.
// XH: 0 the planes of a decode batch; 1 a prompt pass, the rows go to xh as the tensor-core GEMM's fp16 operand and nowhere else; 2 more rows than a decode batch has: xh, quants, scales
// and sums, but none of the planes that only decode matmuls read; 3 a decode batch of which the caller knows that only the tensor-core matmuls of the family's own type
// (Q4_K; Q4_0, Q8_0) read it: their planes (three stores of a super-block's ten)
template <bool Q8K, int PRO, int XH>
__global__ void __launch_bounds__(1024) act_quant_kernel(const aq_args a) {
    constexpr bool NORM = PRO == PRO_RMSNORM || PRO == PRO_LAYERNORM;
    const int     row  = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const pib_oct oct  = pib_oct_of(row, (int) gridDim.x);
    const int     K = (int) a.K, units = (K + 255) / 256, u0 = NORM ? warp : blockIdx.y * W + warp, step = NORM ? W : gridDim.y * W;
    const float * xr   = a.x + (size_t) row * a.xstride;
    const float * x2r  = a.x2_per_row ? a.x2 + (size_t) row * a.xstride : a.x2;
    const int     i00  = u0 * 256 + lane * 8;
    const int     u_lo = NORM ? blockIdx.y * a.per : 0, u_hi = NORM ? min(units, u_lo + a.per) : units;      // the units that this block quantises
    float v[8] = { 0, 0, 0, 0, 0, 0, 0, 0 }, w[8] = { 0, 0, 0, 0, 0, 0, 0, 0 }, bi[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
    // the first unit that this warp quantises stays in registers; its norm weights are immutable: fetched before the wait on the producer of x
    const int uo = NORM && u0 < u_lo ? u0 + (u_lo - u0 + step - 1) / step * step : u0, io = uo * 256 + lane * 8;
    if (NORM && io < K) {
        aq_load8(x2r + io, a.vec, w);
        if (PRO == PRO_LAYERNORM) aq_load8(a.bias + io, a.vec, bi);
    }
    pib_pdl_wait();
    pib_pdl_trigger();
    if (PIB_CANCELLED(a.cancel)) return;

    float scale = 1.0f, mean = 0.0f;
    if (NORM) {
        __shared__ double red[2][32];
        // optional residual add fused in front (reference ggml_add, llama.cpp:3944 / :3962): sum_out = x + addend [+ addend2]
        auto fetch = [&](int i, float (&y)[8]) {
            const bool own = (unsigned) ((i >> 8) - u_lo) < (unsigned) (u_hi - u_lo);
            aq_load8(xr + i, a.vec, y);
            if (a.addend) {
                float z[8];
                aq_load8(a.addend + (size_t) row * K + i, a.vec, z);
#pragma unroll
                for (int j = 0; j < 8; j++) y[j] = __fadd_rn(y[j], z[j]);
                if (PRO == PRO_LAYERNORM && a.addend2) {
                    aq_load8(a.addend2 + (size_t) row * K + i, a.vec, z);
#pragma unroll
                    for (int j = 0; j < 8; j++) y[j] = __fadd_rn(y[j], z[j]);
                }
                if (own) aq_store8(a.sum_out + (size_t) row * K + i, a.vec, y);
            }
        };
        // the sum of f(value) over the row, known to every thread
        auto total = [&](double s, double * r) -> double {
            s = warp_sum_d(s);
            if (lane == 0) r[warp] = s;
            __syncthreads();
            s = lane < W ? r[lane] : 0.0;
            if (W > 8) { s += __shfl_xor_sync(0xffffffffu, s, 16); s += __shfl_xor_sync(0xffffffffu, s, 8); }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            return __shfl_sync(0xffffffffu, s, 0);
        };
        auto mean_of = [&](double s) -> float { return (float) (a.inv_k != 0.0 ? s * a.inv_k : s / (double) K); };
        auto term = [&](float y) -> double { return PRO == PRO_LAYERNORM ? (double) y : (double) __fmul_rn(y, y); };
        double s = 0.0;
        if (i00 < K) {
            fetch(i00, v);
#pragma unroll
            for (int j = 0; j < 8; j++) s += term(v[j]);
        }
#pragma unroll 1
        for (int i = i00 + step * 256; i < K; i += step * 256) {
            float y[8];
            fetch(i, y);
#pragma unroll
            for (int j = 0; j < 8; j++) s += term(y[j]);
            if (i == io) {
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = y[j];
            }
        }
        const float m = mean_of(total(s, red[0]));
        if (PRO == PRO_RMSNORM) scale = 1.0f / sqrtf(m + a.eps);
        else {
            // LayerNorm (reference norm_f32, ggml.c:8959-9020): mean from the double sum, then the double sum of the float
            // squares of (x - mean), scale = 1 / sqrtf(variance + eps)
            mean = m;
            s = 0.0;
            auto square = [&](float y) -> double { const float t = __fsub_rn(y, mean); return (double) __fmul_rn(t, t); };
#pragma unroll 1
            for (int i = i00; i < K; i += step * 256) {
                float y[8];
                if (i != io) fetch(i, y);
                else {
#pragma unroll
                    for (int j = 0; j < 8; j++) y[j] = v[j];
                }
#pragma unroll
                for (int j = 0; j < 8; j++) s += square(y[j]);
            }
            scale = 1.0f / sqrtf(mean_of(total(s, red[1])) + a.eps);
        }
        if (a.addend) xr = a.sum_out + (size_t) row * K;          // later units are read again: what this thread itself wrote
    }

#pragma unroll 1
    for (int u = uo; u < u_hi; u += step) {
        const int  i  = u * 256 + lane * 8;
        const bool in = Q8K || i < K;                             // the last group of 32-element blocks may end before 256: zeros
        if (!NORM || u != uo) {
            if (in) aq_load8(xr + i, a.vec, v);
            if (PRO == PRO_SILU_MUL || NORM) { if (in) aq_load8(x2r + i, a.vec, w); }
            if (PRO == PRO_LAYERNORM) { if (in) aq_load8(a.bias + i, a.vec, bi); }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (PRO == PRO_RMSNORM)        v[j] = __fmul_rn(__fmul_rn(v[j], scale), w[j]);
            // reference norm_f32: y = (x - mean) * scale, then ggml_mul by the weight, ggml_add of the bias
            else if (PRO == PRO_LAYERNORM) v[j] = __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(v[j], mean), scale), w[j]), bi[j]);
            else if (PRO == PRO_SILU_MUL)  v[j] = __fmul_rn(pib_h2f(a.lut[pib_f2h(v[j])]), w[j]);
            else if (PRO == PRO_GELU)      v[j] = pib_h2f(a.lut[pib_f2h(v[j])]);
            if (!in) v[j] = 0.f;
        }
        if (a.vout && in) aq_store8(a.vout + (size_t) row * K + i, a.vec, v);
        if (Q8K) {
            const int    nsb = units;
            const size_t rs  = (size_t) row * nsb + u;
            if (XH == 1) q8k_quantise_sb(v, lane, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, a.xh + (size_t) row * K + u * PIB_QK_K);
            else if (XH == 2) q8k_quantise_sb(v, lane, a.qs + (size_t) row * K + u * PIB_QK_K, nullptr, (int16_t *) a.bs + rs * 16, nullptr, nullptr, nullptr, a.d + rs, nullptr, nullptr,
                                              a.xh + (size_t) row * K + u * PIB_QK_K);
            else if (XH == 3) {
                const size_t os = (size_t) oct.before * nsb + (size_t) u * oct.gs + oct.g;
                q8k_quantise_sb(v, lane, nullptr, a.qsp + (size_t) oct.before * K + (size_t) u * oct.gs * PIB_QK_K + oct.g * 64, nullptr, a.bs8 + os * 16, nullptr, nullptr, nullptr,
                                nullptr, nullptr, nullptr, 64 * oct.gs, a.dxo + os);
            } else {
                const size_t os = (size_t) oct.before * nsb + (size_t) u * oct.gs + oct.g, of = (size_t) oct.before * K + (size_t) u * oct.gs * PIB_QK_K + oct.g * 64;
                q8k_quantise_sb(v, lane, a.qs + (size_t) row * K + u * PIB_QK_K, a.qsp + of, (int16_t *) a.bs + rs * 16, a.bs8 + os * 16, a.sbs + rs * 8, a.qsl + rs * 64, a.d + rs,
                                a.q6p + of, a.b16 + os * 32, nullptr, 64 * oct.gs, a.dxo + os);
            }
        } else {
            // four lanes per block of 32: d = max|x| / 127, q = round(x * (127 / max|x|))
            const int nb = K / PIB_QK, blk = u * 8 + (lane >> 2), j = lane >> 2;
            float amax = 0.f;
#pragma unroll
            for (int k = 0; k < 8; k++) amax = fmaxf(amax, fabsf(v[k]));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            const float d = amax / 127.f;
            float       id = amax != 0.0f ? 127.f / amax : 0.0f;
            if (id > 3.4028235e38f) {                                 // overflow (scale 0): the reference's conversion gives the lowest whole number for every element
                id = 128.f;
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] = -1.f;
            }
            int q[8];
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = __float2int_rn(__fmul_rn(v[k], id));
            const int2 p = make_int2(q8k_pack(q[0], q[1], q[2], q[3]), q8k_pack(q[4], q[5], q[6], q[7]));
            int sum = 0;
            if (XH != 3) {
                sum = __dp4a(p.x, 0x01010101, __dp4a(p.y, 0x01010101, 0));
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            }
            if (XH != 3 && in) *reinterpret_cast<int2 *>(a.qs + (size_t) row * K + i) = p;
            // fragment-order copy for the tensor-core GEMV (gemv_blk32.cu): element e = 16 h + 4 t + i of block j of a group
            // of eight is byte 8 (j & 1) + 4 h + i of quarter t of piece j >> 1; this lane holds quarters 2 (lane & 1) and the next of half h = (lane & 3) / 2
            int8_t * o = a.qsp + (size_t) oct.before * units * 256 + (((size_t) u * 4 + (j >> 1)) * oct.gs + oct.g) * 64 + (lane & 1) * 32 + (j & 1) * 8 + ((lane & 3) >> 1) * 4;
            *reinterpret_cast<int *>(o)      = p.x;
            *reinterpret_cast<int *>(o + 16) = p.y;
            if ((lane & 3) == 0) {
                reinterpret_cast<__half *>(a.bs8)[(size_t) oct.before * units * 8 + ((size_t) u * oct.gs + oct.g) * 8 + j] = __float2half_rn(d);
                if (XH != 3 && in) {
                    a.d[(size_t) row * nb + blk]               = pib_h2f(pib_f2h(d));   // the reference stores d as fp16
                    ((int32_t *) a.bs)[(size_t) row * nb + blk] = sum;
                }
            }
        }
    }
}

// The gated product of a prompt pass -> the GEMM's fp16 rows, the table in shared memory: one block per SM takes it in front of the launch wait, then its warps go over the rows'
// super-blocks.  In act_quant_kernel a warp's eight look-ups go to 32 places each and L1 gives one line a clock: 700 rows of 11008 31 us a launch, here 15.
#define AQ_TABLE_BYTES (65536 * 2)
__global__ void __launch_bounds__(1024) silu_rows_kernel(const float * __restrict__ gate, const float * __restrict__ up, int64_t stride, int b, int nsb, const uint16_t * __restrict__ lut,
                                                         __half * __restrict__ xh, const int * __restrict__ cancel) {
    extern __shared__ __align__(16) uint16_t aq_table[];
    for (int i = threadIdx.x; i < AQ_TABLE_BYTES / 16; i += 1024) reinterpret_cast<uint4 *>(aq_table)[i] = __ldg(reinterpret_cast<const uint4 *>(lut) + i);
    __syncthreads();
    pib_pdl_wait();
    pib_pdl_trigger();
    if (PIB_CANCELLED(cancel)) return;
    const int lane = threadIdx.x & 31, n = b * nsb, step = gridDim.x * 32;
    int u = blockIdx.x * 32 + (threadIdx.x >> 5);
    float x[8], w[8];
    auto load = [&](int k) {
        const size_t at = (size_t) (k / nsb) * stride + (k % nsb) * 256 + lane * 8;
        aq_load8(gate + at, 1, x);
        aq_load8(up + at, 1, w);
    };
    if (u < n) load(u);
#pragma unroll 1
    for (; u < n; u += step) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = __fmul_rn(pib_h2f(aq_table[pib_f2h(x[j])]), w[j]);
        if (u + step < n) load(u + step);                         // the next one's values are on their way meanwhile
        q8k_quantise_sb(v, lane, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, xh + (size_t) u * 256);
    }
}

template <int PRO>
static int launch_aq(int wtype, const float * x, const float * x2, int x2_per_row, float eps, int b, int64_t K, void * act,
                     float * vout, const uint16_t * lut, cudaStream_t st, const float * addend = nullptr,
                     float * sum_out = nullptr, const int * cancel = nullptr, int64_t xstride = 0, const float * bias = nullptr,
                     const float * addend2 = nullptr, void * xhat = nullptr, bool lean = false) {
    if (xstride == 0) xstride = K;
    const pib_act_layout L = pib_act_layout_of(wtype, K, b);
    uint8_t * act8 = (uint8_t *) act;
    aq_args a;
    a.x = x; a.x2 = x2; a.addend = addend; a.addend2 = addend2; a.bias = bias; a.sum_out = sum_out; a.vout = vout; a.lut = lut; a.cancel = cancel;
    a.K = K; a.xstride = xstride; a.eps = eps; a.inv_k = (K & (K - 1)) == 0 ? 1.0 / (double) K : 0.0; a.x2_per_row = x2_per_row;
    a.qs = (int8_t *) act8 + L.qs_off; a.d = (float *) (act8 + L.d_off); a.bs = act8 + L.bs_off; a.bs8 = (int8_t *) act8 + L.bs8_off; a.qsp = (int8_t *) act8 + L.qsp_off;
    a.qsl = (int2 *) (act8 + L.qsl_off); a.sbs = (int16_t *) (act8 + L.sbs_off); a.q6p = (int8_t *) act8 + L.q6p_off; a.b16 = (int8_t *) act8 + L.b16_off; a.dxo = (float *) (act8 + L.dxo_off);
    uintptr_t at = (uintptr_t) (xstride * 4);                                   // K * 4 is a multiple of 128
    for (const void * p : { (const void *) x, (const void *) x2, (const void *) addend, (const void *) addend2, (const void *) bias, (const void *) sum_out, (const void *) vout }) at |= (uintptr_t) p;
    a.vec = (at & 15) == 0;
    constexpr bool NORM = PRO == PRO_RMSNORM || PRO == PRO_LAYERNORM, PROMPT = PRO == PRO_PLAIN || PRO == PRO_RMSNORM || PRO == PRO_SILU_MUL;
    const int units = (int) ((K + 255) / 256);
    // With a norm: the row in one block, or a decode batch's row in several.  Without: up to eight warps per block, as many as leave no more than 32 blocks.  The matmul behind is
    // launched while these blocks run, and where it has a few CTAs per SM its placement follows the room that they leave: a warp on most SMs of the machine sends a third and fourth CTA to
    // the others (us with the matmul, 1 / 2 / 4 / 8 warps per block: Q4_0 5024 x 16128, 2 tokens 21.8 18.3 15.4 15.4; 4992 x 14336, 4 tokens 19.5 18.6 16.9 14.2; Q5_K 5520 x 9984, 6 tokens
    // 16.2 16.3 16.0 13.5; Q4_K 8192 x 28672, 64 rows 61.9 57.8 54.8 54.3), while eight warps of one block cost a small row more than eight blocks (2048, one token 3.85 / 4.05).
    int W = std::min(32, units), parts = 1;
    if (NORM) {
        a.per = b <= PIB_MAX_BATCH ? 8 : units;
        parts = (units + a.per - 1) / a.per;
    } else {
        W = 1;
        while (W < 8 && W < units && b * ((units + W - 1) / W) > 32) W *= 2;
        parts = (units + W - 1) / W;
    }
    // a prompt's gated product: from a super-block per warp of the machine on
    if (PRO == PRO_SILU_MUL && xhat && wtype == PIB_TYPE_Q4_K && a.vec && (int64_t) b * units >= 32 * pib_num_sms()) {
        static pib_per_device attrs;
        PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(silu_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AQ_TABLE_BYTES); }));
        PIB_CHECK(pib_launch(silu_rows_kernel, dim3((unsigned) pib_num_sms()), dim3(1024), AQ_TABLE_BYTES, st, x, x2, xstride, b, units, lut, (__half *) xhat, cancel));
        return PIB_OK;
    }
    const dim3 grid(b, (unsigned) parts), block(32 * W);
#define AQ_GO(Q8K, XH) a.xh = (__half *) (XH == 2 ? (void *) a.qsl : xhat); PIB_CHECK(pib_launch(act_quant_kernel<Q8K, PRO, XH>, grid, block, 0, st, a))
    // more rows than a decode matmul takes: the GEMM's operand takes the place of the qsl plane (pib_act_layout) and of the GEMM's own conversion (4 us a launch)
    lean = lean && PROMPT && b <= PIB_MAX_BATCH;
    if (wtype != PIB_TYPE_Q4_K)   { if (lean) { AQ_GO(false, (PROMPT ? 3 : 0)); } else { AQ_GO(false, 0); } }
    else if (PROMPT && xhat)      { AQ_GO(true, (PROMPT ? 1 : 0)); }
    else if (b > PIB_MAX_BATCH)   { AQ_GO(true, 2); }
    else if (lean)                { AQ_GO(true, (PROMPT ? 3 : 0)); }
    else                          { AQ_GO(true, 0); }
#undef AQ_GO
    return PIB_OK;
}

static int check_args(int wtype, int b, int64_t K) {
    const int blk = wtype == PIB_TYPE_Q4_K ? PIB_QK_K : PIB_QK;
    if ((wtype != PIB_TYPE_Q4_0 && wtype != PIB_TYPE_Q8_0 && wtype != PIB_TYPE_Q4_K) || b < 1 || K < blk || K % blk != 0) {
        pib_set_error("act quantise: bad arguments (type %d, b %d, K %lld)", wtype, b, (long long) K);
        return PIB_ERR_ARG;
    }
    return PIB_OK;
}

extern "C" size_t pib_act_bytes(int wtype, int64_t K, int b) { return pib_act_layout_of(wtype, K, b).total; }

extern "C" int pib_quantize_act(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, pib_stream s) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_PLAIN>(wtype, x_dev, nullptr, 0, 0.f, b, K, act_dev, nullptr, nullptr, (cudaStream_t) s);
}

extern "C" int pib_norm_quantize_act(int wtype, int norm_kind, const float * x_dev, const float * norm_w_dev, float eps, int b,
                                     int64_t K, void * act_dev, float * xnorm_dev, pib_stream s) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    if (norm_kind != 1) { pib_set_error("pib_norm_quantize_act: only RMSNorm (1) is implemented"); return PIB_ERR_UNSUPP; }
    return launch_aq<PRO_RMSNORM>(wtype, x_dev, norm_w_dev, 0, eps, b, K, act_dev, xnorm_dev, nullptr, (cudaStream_t) s);
}

// ---- internal (engine) entry points ---------------------------------------------------------------------------------
// xhat (Q8_K only): the rows go there as the tensor-core GEMM's fp16 operand instead of into the planes of act_dev
// lean: of the planes only those that the tensor-core decode matmuls of the family's own type read
// silu(gate) * up -> quantised activations for the down projection; gate_up: [b][2*K] rows = {gate[K], up[K]}
int pib_silu_mul_quantize_act(int wtype, const float * gate_dev, const float * up_dev, int64_t row_stride, int b, int64_t K,
                              void * act_dev, const int * cancel, cudaStream_t st, void * xhat, bool lean) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_SILU_MUL>(wtype, gate_dev, up_dev, 1, 0.f, b, K, act_dev, nullptr, pib_get_luts().silu_f16, st,
                                   nullptr, nullptr, cancel, row_stride, nullptr, nullptr, xhat, lean);
}

int pib_quantize_act_c(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, const int * cancel, cudaStream_t st, void * xhat, bool lean) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_PLAIN>(wtype, x_dev, nullptr, 0, 0.f, b, K, act_dev, nullptr, nullptr, st, nullptr, nullptr, cancel, 0, nullptr, nullptr, xhat, lean);
}

// [sum_out = x + addend;] act = quantise(rmsnorm(sum or x) * w)
int pib_add_rmsnorm_quantize_act(int wtype, const float * x_dev, const float * addend_dev, float * sum_out_dev,
                                 const float * norm_w_dev, float eps, int b, int64_t K, void * act_dev, const int * cancel,
                                 cudaStream_t st, void * xhat, bool lean) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_RMSNORM>(wtype, x_dev, norm_w_dev, 0, eps, b, K, act_dev, nullptr, nullptr, st, addend_dev, sum_out_dev,
                                  cancel, 0, nullptr, nullptr, xhat, lean);
}

// falcon: [sum_out = (x + addend) + addend2;] act = quantise(layernorm(sum or x) * w + bias)
int pib_add_layernorm_quantize_act(int wtype, const float * x_dev, const float * addend_dev, const float * addend2_dev,
                                   float * sum_out_dev, const float * norm_w_dev, const float * norm_b_dev, float eps, int b,
                                   int64_t K, void * act_dev, const int * cancel, cudaStream_t st) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_LAYERNORM>(wtype, x_dev, norm_w_dev, 0, eps, b, K, act_dev, nullptr, nullptr, st, addend_dev, sum_out_dev,
                                    cancel, 0, norm_b_dev, addend2_dev);
}

// falcon: act = quantise(gelu(x)) through the reference's fp16 table (ggml.c:8676)
int pib_gelu_quantize_act(int wtype, const float * x_dev, int b, int64_t K, void * act_dev, const int * cancel, cudaStream_t st) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    return launch_aq<PRO_GELU>(wtype, x_dev, nullptr, 0, 0.f, b, K, act_dev, nullptr, pib_get_luts().gelu_f16, st, nullptr, nullptr, cancel);
}

extern "C" int pib_act_to_blocks(int wtype, const void * act_dev, int b, int64_t K, void * out) {
    if (check_args(wtype, b, K) != PIB_OK) return PIB_ERR_ARG;
    const pib_act_layout L = pib_act_layout_of(wtype, K, b);
    uint8_t * h = (uint8_t *) malloc(L.total);
    cudaError_t e = cudaMemcpy(h, act_dev, L.total, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { free(h); PIB_CHECK(e); }
    uint8_t * o = (uint8_t *) out;
    if (wtype == PIB_TYPE_Q4_K) {
        const int64_t nsb = K / 256;
        for (int t = 0; t < b; t++)
            for (int64_t s = 0; s < nsb; s++) {
                uint8_t * blk = o + ((size_t) t * nsb + s) * 292;
                memcpy(blk, h + L.d_off + ((size_t) t * nsb + s) * 4, 4);
                memcpy(blk + 4, h + L.qs_off + (size_t) t * K + s * 256, 256);
                memcpy(blk + 260, h + L.bs_off + ((size_t) t * (K / 16) + s * 16) * 2, 32);
            }
    } else {
        const int64_t nb = K / 32;
        for (int t = 0; t < b; t++)
            for (int64_t s = 0; s < nb; s++) {
                uint8_t * blk = o + ((size_t) t * nb + s) * 34;
                float     d;
                memcpy(&d, h + L.d_off + ((size_t) t * nb + s) * 4, 4);
                const __half hd = __float2half_rn(d);
                memcpy(blk, &hd, 2);
                memcpy(blk + 2, h + L.qs_off + (size_t) t * K + s * 32, 32);
            }
    }
    free(h);
    return PIB_OK;
}
