// q8k_quant.cuh -- one Q8_K super-block (256 values) quantised by one warp, lane l holding values 8l .. 8l+7; shared by the
// activation-quantiser kernels (act_quant.cu) and by the GEMV that quantises its own activations in its prologue (gemv_mma.cu),
// so that the two produce the same bytes.  Reference: quantize_row_q8_K (ggml-quants.c:2329-2363): iscale = -128 / (signed value
// of the first max-|x| element), q = min(127, rne(iscale * x)), d = 1 / iscale, 16-wide bsums.
#pragma once
#include "pib_common.cuh"

// place of element e of a 64-wide chunk in the fp16 rows that the tensor-core GEMM multiplies (gemm_q4k_tc.cu): the weight record's low nibbles (e < 32) come first,
// a lane quarter's eight as two runs of four, the middle two of each run swapped (one mask of a word of nibble bytes gives the pairs (e0, e2) and (e1, e3))
__host__ __device__ __forceinline__ int tg_kpos(int e) { return (e & 32) + ((e >> 2) & 1) * 16 + ((e >> 3) & 3) * 4 + ((e & 1) << 1 | ((e >> 1) & 1)); }

// four whole numbers as the bytes of a word, saturated to -128 .. 127
__device__ __forceinline__ int q8k_pack(int a, int b, int c, int d) {
    int w;
    asm("{\n\t.reg .b32 t;\n\tcvt.pack.sat.s8.s32.b32 t, %4, %3, 0;\n\tcvt.pack.sat.s8.s32.b32 %0, %2, %1, t;\n\t}" : "=r"(w) : "r"(a), "r"(b), "r"(c), "r"(d));
    return w;
}

// Every pointer addresses this super-block's part of its plane (see pib_act_layout) and may be null:
//   qs   [256] int8   quants in element order           qsp  int8   the same in B-fragment order of mma.m16n8k32: four pieces of 64, `cs` bytes apart
//   bs   [16]  int16  sums of 16                         bs8 [16]  int8   sub-block (32) sums split as 64 hi + lo: hi[8], lo[8]
//   sbs  [8]   int16  sub-block sums                     qsl [64]  int2   B registers of the lane-exact kernel     d [1] float
//   xh   [256] fp16   quants times d in the GEMM's order (tg_kpos)
//   q6p  int8   quants in the k16 B-fragment order of the Q6_K kernel, pieces as qsp's      b16 [32] int8   sums of 16 split as 64 hi + lo: hi[16], lo[16]
__device__ __forceinline__ void q8k_quantise_sb(const float (&v)[8], int lane, int8_t * qs, int8_t * qsp, int16_t * bs, int8_t * bs8,
                                                int16_t * sbs, int2 * qsl, float * d, int8_t * q6p = nullptr, int8_t * b16 = nullptr, __half * xh = nullptr, int cs = 64, float * dxo = nullptr) {
    // first element (in index order) with the largest |x|: strict '>' scan, ties keep the lower index; a lane's elements are neighbours, so the first lane that has the
    // warp's maximum holds it (one reduction instruction and a vote; five rounds of three shuffles took 0.2 us)
    float amax = 0.0f, mx = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float ax = fabsf(v[j]);
        if (ax > amax) { amax = ax; mx = v[j]; }
    }
    float wmax;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(wmax) : "f"(amax));
    mx   = __shfl_sync(0xffffffffu, mx, __ffs(__ballot_sync(0xffffffffu, amax == wmax)) - 1);
    amax = wmax;
    int   q[8];
    float dval = 0.0f;
    if (amax <= 0x1p-121f) {                                               // zeros, or -128 / mx overflows: the reference's whole numbers are 0 then, its scale 1 / iscale
#pragma unroll
        for (int j = 0; j < 8; j++) q[j] = 0;
        if (amax != 0.0f) dval = copysignf(0.0f, -mx);
    } else {
        const float iscale = -128.f / mx;
#pragma unroll
        for (int j = 0; j < 8; j++) q[j] = __float2int_rn(__fmul_rn(iscale, v[j]));          // -128 .. 128, 127 at most below
        dval = 1.0f / iscale;
    }
    int2 packed;
    packed.x = q8k_pack(q[0], q[1], q[2], q[3]);
    packed.y = q8k_pack(q[4], q[5], q[6], q[7]);
    if (xh) {                                                              // this lane's eight elements are two runs of one 64-wide chunk
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = __fmul_rn((float) min(127, q[4 * u + j]), dval);
            const __half2 p[2] = { __floats2half2_rn(w[0], w[2]), __floats2half2_rn(w[1], w[3]) };
            *reinterpret_cast<uint2 *>(xh + (lane >> 3) * 64 + tg_kpos((lane & 7) * 8 + 4 * u)) = *reinterpret_cast<const uint2 *>(p);
        }
    }
    if (qs) *reinterpret_cast<int2 *>(qs + lane * 8) = packed;
    // fragment-order copy for the tensor-core GEMV: lane = 8c + 4h + t  ->  piece c, offset 16t + 8h
    if (qsp) *reinterpret_cast<int2 *>(qsp + (lane >> 3) * cs + (lane & 3) * 16 + ((lane >> 2) & 1) * 8) = packed;
    // lane l holds elements 8l .. 8l+7 = group l / 2, offsets 8 (l & 1) ..: quarters t = 2 (l & 1) and 2 (l & 1) + 1
    if (q6p) {
        int8_t * o = q6p + (lane >> 3) * cs + (2 * (lane & 1)) * 16 + ((lane >> 1) & 3) * 4;
        *reinterpret_cast<int *>(o)      = packed.x;
        *reinterpret_cast<int *>(o + 16) = packed.y;
    }
    const int s8  = __dp4a(packed.x, 0x01010101, __dp4a(packed.y, 0x01010101, 0));
    const int s16 = s8 + __shfl_xor_sync(0xffffffffu, s8, 1);
    if (bs && (lane & 1) == 0) bs[lane >> 1] = (int16_t) s16;
    if (b16 && (lane & 1) == 0) { b16[lane >> 1] = (int8_t) (s16 >> 6); b16[16 + (lane >> 1)] = (int8_t) (s16 & 63); }
    const int s32 = s16 + __shfl_xor_sync(0xffffffffu, s16, 2);        // the 32-element sub-block sum (lanes 4j..4j+3)
    if ((lane & 3) == 0) {
        if (bs8) { bs8[lane >> 2] = (int8_t) (s32 >> 6); bs8[8 + (lane >> 2)] = (int8_t) (s32 & 63); }
        if (sbs) sbs[lane >> 2] = (int16_t) s32;
    }
    // lane-group copy for the lane-exact kernel: this lane holds lane groups 2 (lane % 4) and 2 (lane % 4) + 1 of sub-block lane / 4
    if (qsl) {
        int2 * o = qsl + 2 * (lane & 3) * 8 + (lane >> 2);
        o[0] = make_int2(packed.x, 0);
        o[8] = make_int2(0, packed.y);
    }
    if (d && lane == 0) *d = dval;
    if (dxo && lane == 0) *dxo = dval;
}
