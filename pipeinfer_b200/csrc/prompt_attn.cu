// prompt_attn.cu -- RoPE + KV store and masked attention for ALL tokens of a wide prompt pass (up to PIB_PROMPT_MAX) at once.
//
// The decode attention (attention.cu) gives a CTA to every (query head, token) and keeps the reference's order of every fp32 sum.  A prompt pass
// whose matmuls already run on the tensor cores has no use for that order, and paid for it: sixteen dependent launches per layer, each walking the
// whole cache for every token (57 us a launch at 700 cells and 32 heads of 128: 10.5 ms of a 13.3 ms prompt of 700 tokens through four 4096-wide layers).
// Here a pass is two launches per layer:
//   prompt_rope_kernel   rotates Q and K, writes K and V of the pass to the cache and Q as fp16 -- the values and roundings of attention.cu;
//   prompt_attn_kernel   a CTA per (64 tokens, query head): scores and weighted sums as fp16 matrix products with fp32 accumulation.
// Arithmetic against the reference's (llama.cpp:3698 llm_build_kqv): fp16 Q, K, V and fp32 sums as there; exp is formed in fp32 from the unrounded
// difference (there: a table over fp16 differences), weights are rounded to fp16 before they are divided by their sum (there: after), the sum is held
// in double.  So nothing is rounded more often than there, and only the order of the fp32 sums differs.
//
// What bounds it: the launch has 4 MFLOP per (head, 64 tokens, 64 cells) and at most a few hundred CTAs, so it is latency: warps walk their tiles one after the
// other (256 tokens, 32 heads of 128, up to 700 cells: 33 us with one group of four warps per CTA, 25 with two that take the tiles in turn, the rotation 7; the sixteen
// launches before: 913).  mma.sync on register operands is taken rather than tcgen05: a tile's scores go straight from the accumulator registers through exp into the
// next product's A operand, and at 0.1 of a prompt's time the trip through tensor memory has nothing to win.
#include "pib_common.cuh"
#include "desc.cuh"
#include "engine.cuh"

#define PA_ROWS   64                 // tokens per CTA: 4 warps x 16, twice
#define PA_CELLS  64                 // cells per tile
#define PA_TILES  1024               // tiles of the visibility bitmap: contexts of up to 65536 cells

// what a pass needs from its chunks' descriptors, token after token: ids | positions | cells | sequence bitsets
__global__ void prompt_gather_kernel(const uint8_t * __restrict__ desc_base, size_t stride, pib_prompt_slots sl, int ntok, int W, int32_t * __restrict__ tok,
                                     int32_t * __restrict__ pos, int32_t * __restrict__ cell, uint32_t * __restrict__ bits) {
    const int t = blockIdx.x, k = t / PIB_CHUNK, i = t % PIB_CHUNK;
    if (t >= ntok) return;
    const uint8_t * d = desc_base + (size_t) sl.slot[k] * stride;
    if (threadIdx.x == 0) {
        tok[t]  = reinterpret_cast<const int32_t *>(d + PIB_DESC_TOK_OFF)[i];
        pos[t]  = reinterpret_cast<const int32_t *>(d + PIB_DESC_POS_OFF)[i];
        cell[t] = reinterpret_cast<const int32_t *>(d + PIB_DESC_HDR_OFF)[PIB_DH_KVHEAD] + i;
    }
    const uint32_t * b = reinterpret_cast<const uint32_t *>(d + PIB_DESC_BITS_OFF) + (size_t) i * W;
    for (int w = threadIdx.x; w < W; w += blockDim.x) bits[(size_t) t * W + w] = b[w];
}

int pib_prompt_gather(const uint8_t * desc_base, size_t stride, const pib_prompt_slots & sl, int ntok, int W, int32_t * tok, int32_t * pos, int32_t * cell, uint32_t * bits,
                      cudaStream_t st) {
    prompt_gather_kernel<<<ntok, 32, 0, st>>>(desc_base, stride, sl, ntok, W, tok, pos, cell, bits);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

// a thread takes four consecutive values of a token's q | k | v row: two rotated pairs (2j, 2j + 1), or four values of v
__global__ void __launch_bounds__(256) prompt_rope_kernel(const float * __restrict__ qkv, const int32_t * __restrict__ pos, const int32_t * __restrict__ cell, const float2 * __restrict__ rope,
                                                          int rope_n_pos, int E, int GQA, int hd, __half * __restrict__ q16, __half * __restrict__ kc, __half * __restrict__ vc,
                                                          const int * __restrict__ cancel) {
    pib_pdl_wait();
    pib_pdl_trigger();
    if (PIB_CANCELLED(cancel)) return;
    const int t = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 4, row = E + 2 * GQA;
    if (i >= row) return;
    const float4 x = *reinterpret_cast<const float4 *>(qkv + (size_t) t * row + i);
    __half2 o[2];
    if (i < E + GQA) {
        const int    j = (i % hd) / 2;
        const float4 cs = *reinterpret_cast<const float4 *>(rope + (size_t) min(pos[t], rope_n_pos - 1) * (hd / 2) + j);      // {cos, sin} of pairs j, j + 1
        o[0] = __halves2half2(__float2half_rn(__fsub_rn(__fmul_rn(x.x, cs.x), __fmul_rn(x.y, cs.y))), __float2half_rn(__fadd_rn(__fmul_rn(x.x, cs.y), __fmul_rn(x.y, cs.x))));
        o[1] = __halves2half2(__float2half_rn(__fsub_rn(__fmul_rn(x.z, cs.z), __fmul_rn(x.w, cs.w))), __float2half_rn(__fadd_rn(__fmul_rn(x.z, cs.w), __fmul_rn(x.w, cs.z))));
    } else {
        o[0] = __floats2half2_rn(x.x, x.y);
        o[1] = __floats2half2_rn(x.z, x.w);
    }
    __half * dst = i < E ? q16 + (size_t) t * E + i : i < E + GQA ? kc + (size_t) cell[t] * GQA + (i - E) : vc + (size_t) cell[t] * GQA + (i - E - GQA);
    *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(o);
}

__device__ __forceinline__ void pa_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void pa_ldsm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pa_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// bits i = 0..15: cell c + i is seen (its mask byte is 0 and it lies inside the attended range)
__device__ __forceinline__ uint32_t pa_seen16(const uint8_t * __restrict__ mrow, int c, int n, bool vec) {
    if (c >= n) return 0;
    uint32_t hid = 0;
    if (vec) {
        const uint4 m = *reinterpret_cast<const uint4 *>(mrow + c);
        // four bytes of 0 / 1 -> four neighbouring bits: byte i lands on bit 24 + i
        hid = ((m.x * 0x01020408u) >> 24 & 15u) | ((m.y * 0x01020408u) >> 24 & 15u) << 4 | ((m.z * 0x01020408u) >> 24 & 15u) << 8 | ((m.w * 0x01020408u) >> 24 & 15u) << 12;
    } else {
        for (int i = 0; i < 16 && c + i < n; i++) hid |= (uint32_t) mrow[c + i] << i;
    }
    const uint32_t in = n - c >= 16 ? 0xffffu : (1u << (n - c)) - 1u;
    return ~hid & in;
}

// two groups of four warps take the tiles in turn, each with its own stages and running state, and meet at the end
__device__ __forceinline__ void pa_group_sync(int grp) { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); }
__device__ __forceinline__ bool pa_group_any(int grp, bool v) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\tbar.red.or.pred q, %1, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(grp + 1), "r"((int) v) : "memory");
    return r != 0;
}

template <int HD>
__global__ void __launch_bounds__(256, HD == 64 ? 2 : 1)
prompt_attn_kernel(const __half * __restrict__ q16, const __half * __restrict__ kc, const __half * __restrict__ vc, const uint8_t * __restrict__ mask, const int32_t * __restrict__ scalars,
                   int ntok, int E, int GQA, int gdiv, int n_ctx, float kq_scale, float * __restrict__ out, const int * __restrict__ cancel) {
    constexpr int CH = HD / 8, ROWB = HD * 2, TILEB = PA_CELLS * ROWB;            // 16-byte pieces and bytes of a cache row, bytes of a tile
    extern __shared__ __align__(128) uint8_t pa_sm[];                            // per group K[2 stages] | V[2 stages]; at the end group 1's state
    __shared__ uint32_t seen_tiles[PA_TILES / 32];
    const int grp = threadIdx.x >> 7, tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int head = blockIdx.x, row0 = (gridDim.y - 1 - blockIdx.y) * PA_ROWS;   // the last rows see most cells: they start first
    const uint8_t * own = pa_sm + grp * 4 * TILEB;
    const uint32_t  sm = (uint32_t) __cvta_generic_to_shared(own);
    const bool vec = (n_ctx & 15) == 0;
    pib_pdl_wait();
    pib_pdl_trigger();
    // one decision for the block: the flag can change while its warps read it, and the groups' barriers count on every thread
    if (__syncthreads_or(PIB_CANCELLED(cancel))) return;
    const int n = min(scalars[2], n_ctx), n_tiles = (n + PA_CELLS - 1) / PA_CELLS;
    const __half * kh = kc + (size_t) (head / gdiv) * HD, * vh = vc + (size_t) (head / gdiv) * HD;

    // tiles that some row of the block sees (a prompt's later cells, other sequences' cells: none)
    if (threadIdx.x < PA_TILES / 32) seen_tiles[threadIdx.x] = 0;
    __syncthreads();
    {
        const int rows = min(PA_ROWS, ntok - row0), per = (n + 15) / 16;
        for (int i = threadIdx.x; i < rows * per; i += 256) {
            const int r = i / per, c = (i - r * per) * 16;
            if (pa_seen16(mask + (size_t) (row0 + r) * n_ctx, c, n, vec)) atomicOr(&seen_tiles[c / PA_CELLS / 32], 1u << (c / PA_CELLS % 32));
        }
    }
    __syncthreads();
    auto next_tile = [&](int i) {                     // first seen tile at or behind i, n_tiles when there is none
        while (i < n_tiles) {
            const uint32_t w = seen_tiles[i / 32] >> (i % 32);
            if (w) return min(i + __ffs((int) w) - 1, n_tiles);
            i = (i / 32 + 1) * 32;
        }
        return n_tiles;
    };
    auto load_tile = [&](int tile, int stage) {       // rows behind the attended range repeat its last one: their scores are masked
        for (int i = tid; i < PA_CELLS * CH; i += 128) {
            const int r = i / CH, ch = i - r * CH;
            const size_t   src = (size_t) min(tile * PA_CELLS + r, n - 1) * GQA + ch * 8;
            const uint32_t dst = sm + (uint32_t) (stage * TILEB + r * ROWB + ((ch ^ (r & 7)) << 4));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(kh + src) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 2 * TILEB), "l"(vh + src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int ra = row0 + warp * 16 + g, rb = ra + 8;                            // this lane's two rows
    const int rac = min(ra, ntok - 1), rbc = min(rb, ntok - 1);
    uint32_t qf[HD / 16][4];
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
        const __half * qa = q16 + (size_t) rac * E + head * HD + ks * 16 + 2 * t4, * qb = q16 + (size_t) rbc * E + head * HD + ks * 16 + 2 * t4;
        qf[ks][0] = *reinterpret_cast<const uint32_t *>(qa);     qf[ks][1] = *reinterpret_cast<const uint32_t *>(qb);
        qf[ks][2] = *reinterpret_cast<const uint32_t *>(qa + 8); qf[ks][3] = *reinterpret_cast<const uint32_t *>(qb + 8);
    }
    float  o[HD / 8][4], m_a = -INFINITY, m_b = -INFINITY;
    double l_a = 0.0, l_b = 0.0;
#pragma unroll
    for (int i = 0; i < HD / 8; i++) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    constexpr float LOG2E = 1.44269504088896340736f;

    int tile = next_tile(0), stage = 0;
    if (grp) tile = next_tile(tile + 1);
    if (tile < n_tiles) load_tile(tile, 0);
    while (tile < n_tiles) {
        const int nxt = next_tile(next_tile(tile + 1) + 1);
        if (nxt < n_tiles) load_tile(nxt, stage ^ 1);
        const uint32_t bits_a = pa_seen16(mask + (size_t) rac * n_ctx, tile * PA_CELLS + 16 * t4, n, vec);
        const uint32_t bits_b = pa_seen16(mask + (size_t) rbc * n_ctx, tile * PA_CELLS + 16 * t4, n, vec);
        if (nxt < n_tiles) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else               asm volatile("cp.async.wait_group 0;" ::: "memory");
        pa_group_sync(grp);
        const uint32_t sk = sm + (uint32_t) (stage * TILEB), sv = sk + 2 * TILEB;
        // a value that is no number (or infinite) must not reach rows that do not see its cell: 0 x inf.  Rare, so the tile then takes its products one by one
        int odd = 0;
        for (int i = tid; i < PA_CELLS * CH; i += 128) {
            const uint4 v = *reinterpret_cast<const uint4 *>(own + stage * TILEB + 2 * TILEB + i * 16);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t w = q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w;
                odd |= ((w & 0x7c00u) == 0x7c00u) | ((w & 0x7c000000u) == 0x7c000000u);
            }
        }
        odd = pa_group_any(grp, odd);

        float s[8][4];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
            for (int k2 = 0; k2 < HD / 32; k2++) {
                uint32_t b[4];
                const int r = j * 8 + (lane & 7), ch = k2 * 4 + (lane >> 3);
                pa_ldsm(b, sk + (uint32_t) (r * ROWB + ((ch ^ (r & 7)) << 4)));
                pa_mma(s[j], qf[2 * k2], b[0], b[1]);
                pa_mma(s[j], qf[2 * k2 + 1], b[2], b[3]);
            }
        }
        float x_a = -INFINITY, x_b = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t wa = __shfl_sync(0xffffffffu, bits_a, (lane & ~3) + j / 2) >> ((j & 1) * 8 + 2 * t4);
            const uint32_t wb = __shfl_sync(0xffffffffu, bits_b, (lane & ~3) + j / 2) >> ((j & 1) * 8 + 2 * t4);
            s[j][0] = wa & 1 ? s[j][0] * kq_scale : -INFINITY; s[j][1] = wa & 2 ? s[j][1] * kq_scale : -INFINITY;
            s[j][2] = wb & 1 ? s[j][2] * kq_scale : -INFINITY; s[j][3] = wb & 2 ? s[j][3] * kq_scale : -INFINITY;
            x_a = fmaxf(x_a, fmaxf(s[j][0], s[j][1]));
            x_b = fmaxf(x_b, fmaxf(s[j][2], s[j][3]));
        }
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) { x_a = fmaxf(x_a, __shfl_xor_sync(0xffffffffu, x_a, d)); x_b = fmaxf(x_b, __shfl_xor_sync(0xffffffffu, x_b, d)); }
        x_a = fmaxf(x_a, m_a); x_b = fmaxf(x_b, m_b);
        const float u_a = x_a == -INFINITY ? 0.f : x_a, u_b = x_b == -INFINITY ? 0.f : x_b;      // rows that have seen nothing yet
        const float al_a = exp2f((m_a - u_a) * LOG2E), al_b = exp2f((m_b - u_b) * LOG2E);
        m_a = x_a; m_b = x_b;
        uint32_t p[8][2];
        float    t_a = 0.f, t_b = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const __half2 pa = __floats2half2_rn(exp2f((s[j][0] - u_a) * LOG2E), exp2f((s[j][1] - u_a) * LOG2E));
            const __half2 pb = __floats2half2_rn(exp2f((s[j][2] - u_b) * LOG2E), exp2f((s[j][3] - u_b) * LOG2E));
            t_a += __low2float(pa) + __high2float(pa);                            // the weights as they enter the product
            t_b += __low2float(pb) + __high2float(pb);
            p[j][0] = *reinterpret_cast<const uint32_t *>(&pa); p[j][1] = *reinterpret_cast<const uint32_t *>(&pb);
        }
        l_a = l_a * (double) al_a + (double) t_a;
        l_b = l_b * (double) al_b + (double) t_b;
        if (__any_sync(0xffffffffu, al_a != 1.f || al_b != 1.f)) {
#pragma unroll
            for (int i = 0; i < HD / 8; i++) { o[i][0] *= al_a; o[i][1] *= al_a; o[i][2] *= al_b; o[i][3] *= al_b; }
        }
        if (!odd) {
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                const uint32_t a[4] = { p[2 * kk][0], p[2 * kk][1], p[2 * kk + 1][0], p[2 * kk + 1][1] };
#pragma unroll
                for (int i = 0; i < HD / 16; i++) {
                    uint32_t b[4];
                    const int r = kk * 16 + (lane & 15), ch = 2 * i + (lane >> 4);
                    pa_ldsm_t(b, sv + (uint32_t) (r * ROWB + ((ch ^ (r & 7)) << 4)));
                    pa_mma(o[2 * i], a, b[0], b[1]);
                    pa_mma(o[2 * i + 1], a, b[2], b[3]);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++)
                for (int e = 0; e < 8; e++) {                                     // cell 8 j + e: its weights sit in lane e / 2 of the quad
                    const uint32_t wa = __shfl_sync(0xffffffffu, p[j][0], (lane & ~3) + e / 2), wb = __shfl_sync(0xffffffffu, p[j][1], (lane & ~3) + e / 2);
                    const float    fa = pib_h2f((uint16_t) (e & 1 ? wa >> 16 : wa)), fb = pib_h2f((uint16_t) (e & 1 ? wb >> 16 : wb));
                    const int      r = j * 8 + e;
#pragma unroll
                    for (int i = 0; i < HD / 8; i++) {
                        const uint32_t v = *reinterpret_cast<const uint32_t *>(own + stage * TILEB + 2 * TILEB + r * ROWB + ((i ^ (r & 7)) << 4) + t4 * 4);
                        const float    v0 = pib_h2f((uint16_t) v), v1 = pib_h2f((uint16_t) (v >> 16));
                        if (fa != 0.f) { o[i][0] = fmaf(fa, v0, o[i][0]); o[i][1] = fmaf(fa, v1, o[i][1]); }
                        if (fb != 0.f) { o[i][2] = fmaf(fb, v0, o[i][2]); o[i][3] = fmaf(fb, v1, o[i][3]); }
                    }
                }
        }
        pa_group_sync(grp);                                                       // the stage is free for the tile after next
        tile = nxt;
        stage ^= 1;
    }
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) { l_a += __shfl_xor_sync(0xffffffffu, l_a, d); l_b += __shfl_xor_sync(0xffffffffu, l_b, d); }
    // group 1 leaves its state per row and its sums; group 0 adds them, both brought to the common maximum
    __syncthreads();
    float *  po = reinterpret_cast<float *>(pa_sm) + tid;                         // [HD / 2][128 threads]
    float *  pm = reinterpret_cast<float *>(pa_sm) + HD / 2 * 128 + tid * 2;
    double * pl = reinterpret_cast<double *>(pa_sm + HD / 2 * 512 + 1024) + tid * 2;
    if (grp) {
#pragma unroll
        for (int i = 0; i < HD / 8; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) po[(i * 4 + e) * 128] = o[i][e];
        pm[0] = m_a; pm[1] = m_b; pl[0] = l_a; pl[1] = l_b;
    }
    __syncthreads();
    if (grp) return;
    const float x_a = fmaxf(m_a, pm[0]), x_b = fmaxf(m_b, pm[1]), u_a = x_a == -INFINITY ? 0.f : x_a, u_b = x_b == -INFINITY ? 0.f : x_b;
    const float f_a = exp2f((m_a - u_a) * LOG2E), f_b = exp2f((m_b - u_b) * LOG2E), h_a = exp2f((pm[0] - u_a) * LOG2E), h_b = exp2f((pm[1] - u_b) * LOG2E);
    l_a = l_a * (double) f_a + pl[0] * (double) h_a;
    l_b = l_b * (double) f_b + pl[1] * (double) h_b;
#pragma unroll
    for (int i = 0; i < HD / 8; i++) {
        o[i][0] = fmaf(po[(i * 4) * 128], h_a, o[i][0] * f_a);     o[i][1] = fmaf(po[(i * 4 + 1) * 128], h_a, o[i][1] * f_a);
        o[i][2] = fmaf(po[(i * 4 + 2) * 128], h_b, o[i][2] * f_b); o[i][3] = fmaf(po[(i * 4 + 3) * 128], h_b, o[i][3] * f_b);
    }
    const float i_a = (float) (1.0 / l_a), i_b = (float) (1.0 / l_b);
#pragma unroll
    for (int i = 0; i < HD / 8; i++) {
        const int c = head * HD + i * 8 + 2 * t4;
        if (ra < ntok) *reinterpret_cast<float2 *>(out + (size_t) ra * E + c) = make_float2(o[i][0] * i_a, o[i][1] * i_a);
        if (rb < ntok) *reinterpret_cast<float2 *>(out + (size_t) rb * E + c) = make_float2(o[i][2] * i_b, o[i][3] * i_b);
    }
}

// contexts the kernel's visibility bitmap holds; heads are 64 or 128 coordinates for every context (pib_attention_supported)
bool pib_prompt_attention_supported(int hd, int n_ctx) { return (hd == 64 || hd == 128) && n_ctx <= PA_TILES * PA_CELLS; }

template <int HD>
static int pa_launch(const __half * q16, const __half * kc, const __half * vc, const uint8_t * mask, const int32_t * scalars, int ntok, int n_head, int n_head_kv, int n_ctx, float * out,
                     const int * cancel, cudaStream_t st) {
    constexpr size_t smem = (size_t) 8 * PA_CELLS * HD * sizeof(__half);
    PIB_CHECK(cudaFuncSetAttribute(prompt_attn_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    pib_launch(prompt_attn_kernel<HD>, dim3(n_head, (ntok + PA_ROWS - 1) / PA_ROWS), dim3(256), smem, st, q16, kc, vc, mask, scalars, ntok, n_head * HD, n_head_kv * HD, n_head / n_head_kv,
               n_ctx, 1.0f / sqrtf((float) HD), out, cancel);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

// attention of the pass: qkv [ntok][E + 2 GQA] -> out [ntok][E]; q16 = scratch of ntok * E halves.  Two launches.
int pib_prompt_attention(const float * qkv, const int32_t * pos, const int32_t * cell, const float2 * rope, int rope_n_pos, __half * q16, __half * kc, __half * vc, const uint8_t * mask,
                         const int32_t * scalars, int ntok, int n_head, int n_head_kv, int hd, int n_ctx, float * out, const int * cancel, cudaStream_t st) {
    const int E = n_head * hd, GQA = n_head_kv * hd;
    pib_launch(prompt_rope_kernel, dim3((unsigned) (((E + 2 * GQA) / 4 + 255) / 256), (unsigned) ntok), dim3(256), 0, st, qkv, pos, cell, rope, rope_n_pos, E, GQA, hd, q16, kc, vc, cancel);
    PIB_CHECK(cudaGetLastError());
    if (hd == 128) return pa_launch<128>(q16, kc, vc, mask, scalars, ntok, n_head, n_head_kv, n_ctx, out, cancel, st);
    return pa_launch<64>(q16, kc, vc, mask, scalars, ntok, n_head, n_head_kv, n_ctx, out, cancel, st);
}
