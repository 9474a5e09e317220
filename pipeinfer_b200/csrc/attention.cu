// attention.cu -- RoPE + KV store (K5, K6) and multi-sequence masked attention over the KV cache (K7).
//
// Reference op chain (llama.cpp:3913-3944 build_llama, :3546 llm_build_kv_store, :3698 llm_build_kqv; CPU kernels
// ggml.c:11006 rope, :6528 dup f32->f16, :1200 vec_dot_f16, :9937 scale, :10551 soft_max):
//   Q,K <- rope(pos)             theta_i = pos * base^(-2i/d) by repeated multiply, cosf/sinf of the host libm
//   cache K (f16), cache V (f16)  at cells kv_head + t
//   S = (K . fp16(Q)) * 1/sqrt(d)   fp32 accumulate of exact fp16 products
//   S += mask (0 / -inf)            cell visible iff it shares a sequence id with the token and cell.pos <= token.pos
//   P = softmax(S)                  exp through the fp16 table on fp16(S - max), sum in double, P = val * (float)(1/sum)
//   O = V . fp16(P)
// Everything that is rounded in the reference is rounded identically here (fp16 Q, fp16 K/V, fp16 exp table, fp16 P);
// the double sum of fp16 values is exact in any order, so only the fp32 dot-product association differs.
//
// cos/sin come from a table built on the host with the reference's recurrence (rope_table_build), so RoPE itself is
// bit-exact.  The V cache is kept [cell][n_embd_gqa] (not transposed as in the reference, llama.cpp:3569): the layout
// is private and this one is coalesced for both the store and the P.V pass.
#include "pib_common.cuh"
#include "desc.cuh"

#include <math.h>

#include <algorithm>
#include <vector>

// ---- RoPE table -----------------------------------------------------------------------------------------------------
// tab[pos][i] = {cos(theta), sin(theta)}, theta as in reference rope_f32 (ggml.c:11062, 11111-11123) with ext_factor 0:
// theta_base = pos; per pair: theta = freq_scale * theta_base; theta_base *= theta_scale.  mode 2 (NeoX) pre-multiplies
// theta_base by freq_scale once more (ggml.c:11137).
void rope_table_build(std::vector<float2> & tab, int n_pos, int n_dims, int mode, float freq_base, float freq_scale) {
    const float theta_scale = powf(freq_base, -2.0f / n_dims);
    tab.resize((size_t) n_pos * (n_dims / 2));
    if (mode & 4) {
        // direct form: the angle of pair i at position p is p * base^(-2i / n_dims), each from its own power (no running product),
        // evaluated in double and rounded once; pairs are (i, i + n_dims / 2)
        for (int i = 0; i < n_dims / 2; i++) {
            const double f = pow((double) freq_base, -2.0 * i / n_dims) * freq_scale;
            for (int p = 0; p < n_pos; p++) tab[(size_t) p * (n_dims / 2) + i] = make_float2((float) cos(p * f), (float) sin(p * f));
        }
        return;
    }
    for (int p = 0; p < n_pos; p++) {
        float theta_base = (float) p;
        if (mode & 2) theta_base *= freq_scale;
        for (int i = 0; i < n_dims / 2; i++) {
            const float theta = freq_scale * theta_base;
            tab[(size_t) p * (n_dims / 2) + i] = make_float2(cosf(theta), sinf(theta));
            theta_base *= theta_scale;
        }
    }
}

// ---- attention ------------------------------------------------------------------------------------------------------
// RoPE, KV store and attention of one (query head, token), by one block.
//
// att_prefetch fetches what does not depend on the QKV projection: descriptor words, RoPE entries, mask bytes and K rows of the first cells (registers), V rows of
// up to `vcap` cells (cp.async into shared memory).  att_compute does the rest.
//
// What bounds it: the block is alone on its SM for one token, a chain of round trips and barriers between which a few warps work.  300 cells, heads of 64, clocks of the
// parts behind the projection before / now: rotation of the batch's rows 1290 / 780 (two passes of loads, now one), scores 1880 / 1170, maximum 380 / 310, exponentials
// and weights 1470 / 1280 (a thread's score stays in a register), weighted V rows 3870 / 950 (a pair of coordinates and a choice of three places for each row; now four
// coordinates, one place), reduction and the cells behind the last multiple of 32 3020 / 980 (a chain of loads; now only the additions are one).
struct att_args {
    const float *    qkv;            // [n_tokens][rstride]: query heads | key heads [| value heads]
    const float *    vsep;           // value heads of layers whose Wv is a matrix of its own, else null
    const uint8_t *  desc;
    const float2 *   rope;
    int              rope_n_pos, mode;
    __half *         kcache, * vcache;
    const uint8_t *  mask;           // [n_tokens][n_ctx], 0 = visible
    const int32_t *  scalars;
    const uint16_t * exp_lut;
    int              E, GQA, n_ctx, gdiv, vcap;
    float            kq_scale;
    float *          out;            // [n_tokens][E]
};

// shared memory of a block, in bytes: scores, the 32 partial sums and V rows; the batch's K and V rows, the query and the warps' maxima and sums
__host__ __device__ inline size_t att_fixed_smem(int hd) { return (size_t) 2 * PIB_CHUNK * hd * 2 + (size_t) hd * 4 + 16 * 4 + 16 * 8; }
__host__ __device__ inline size_t att_core_smem(int hd, int n_ctx, int vcap) {
    return (((size_t) n_ctx * 4 + 15) & ~(size_t) 15) + (size_t) 32 * hd * 4 + (size_t) (n_ctx < vcap ? n_ctx : vcap) * hd * 2 + att_fixed_smem(hd);
}

template <int HD, int THREADS>
struct att_smem {
    float *  s;                      // [n_ctx] scores, then weights
    float *  red;                    // [32][HD]
    __half * vs;                     // [vcap][HD]
    __half * kb, * vb;               // [PIB_CHUNK][HD] this KV head's rows of the batch's tokens
    float *  sq;                     // [HD]
    float *  redf;                   // [16]
    double * redd;                   // [16]
    __device__ __forceinline__ att_smem(uint8_t * base, int n_ctx, int vcap) {
        s    = reinterpret_cast<float *>(base);
        red  = reinterpret_cast<float *>(base + (((size_t) n_ctx * 4 + 15) & ~(size_t) 15));
        vs   = reinterpret_cast<__half *>(red + 32 * HD);
        kb   = vs + (size_t) min(n_ctx, vcap) * HD;
        vb   = kb + PIB_CHUNK * HD;
        sq   = reinterpret_cast<float *>(vb + PIB_CHUNK * HD);
        redd = reinterpret_cast<double *>(sq + HD);
        redf = reinterpret_cast<float *>(redd + 16);
    }
};

// phase 1 works on cell tid / 2 (+ THREADS / 2 per round), two lanes per cell; PRE rounds of K half-rows are held in registers
template <int HD, int THREADS>
struct att_pre {
    static constexpr int PRE = THREADS / 256;
    int    n, ntok, cell0;
    uint4  k[PRE][HD / 16];
    bool   live[PRE];
    float2 cs[2];
};

template <int HD, int THREADS>
__device__ __forceinline__ void att_prefetch(const att_args & a, const att_smem<HD, THREADS> & sm, int head, int t, att_pre<HD, THREADS> & p) {
    constexpr int   half = HD / 2, CH = HD * 2 / 16;                           // pairs per head; 16-byte chunks per cache row
    const int       tid  = threadIdx.x, kvh = head / a.gdiv, hsel = tid & 1;
    const uint8_t * mrow = a.mask + (size_t) t * a.n_ctx;
    const int32_t * hdr  = reinterpret_cast<const int32_t *>(a.desc + PIB_DESC_HDR_OFF);
    const int32_t * tpos = reinterpret_cast<const int32_t *>(a.desc + PIB_DESC_POS_OFF);
    const __half *  vhead = a.vcache + (size_t) kvh * HD;
    const __half *  khead = a.kcache + (size_t) kvh * HD;
    p.n = min(a.scalars[2], a.n_ctx); p.ntok = hdr[PIB_DH_NTOK]; p.cell0 = hdr[PIB_DH_KVHEAD];
    {
        const int      nst  = min(p.n, a.vcap);
        const uint32_t vs_a = (uint32_t) __cvta_generic_to_shared(sm.vs);
        for (int i = tid; i < nst * CH; i += THREADS) {
            const int c = i / CH, ch = i - c * CH;
            if (c >= p.cell0 && c < p.cell0 + p.ntok) continue;                // the batch's own rows are written by att_compute
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vs_a + (uint32_t) (c * HD * 2 + ch * 16)), "l"(vhead + (size_t) c * a.GQA + ch * 8) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int rd = 0; rd < p.PRE; rd++) {
        const int  i = rd * (THREADS / 2) + (tid >> 1), ic = max(min(i, p.n - 1), 0), bi = ic - p.cell0;
        const bool use = i < p.n && !(bi >= 0 && bi < p.ntok);
        const uint4 * kr = reinterpret_cast<const uint4 *>(khead + (size_t) ic * a.GQA);
#pragma unroll
        for (int q = 0; q < HD / 16; q++) p.k[rd][q] = use ? kr[(q >> 1) * 4 + 2 * (q & 1) + hsel] : make_uint4(0, 0, 0, 0);
        p.live[rd] = i < p.n && !mrow[ic];
    }
    // RoPE entries of this thread's first two rotation items (covers batches of up to 2 * THREADS / half - 1 tokens)
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int i = tid + it * THREADS, r = i / half, j = i - r * half;
        p.cs[it] = make_float2(1.f, 0.f);
        if (r <= p.ntok) p.cs[it] = a.rope[(size_t) min(tpos[r < p.ntok ? r : t], a.rope_n_pos - 1) * half + j];
    }
}

template <int HD, int THREADS>
__device__ __forceinline__ void att_compute(const att_args & a, const att_smem<HD, THREADS> & sm, int head, int t, const att_pre<HD, THREADS> & p) {
    constexpr int   half = HD / 2, PRE = att_pre<HD, THREADS>::PRE, NW = THREADS / 32;
    const int       tid  = threadIdx.x, lane = tid & 31, warp = tid >> 5, kvh = head / a.gdiv, hsel = tid & 1;
    const int       n = p.n, ntok = p.ntok, cell0 = p.cell0;
    const uint8_t * mrow = a.mask + (size_t) t * a.n_ctx;
    const int32_t * tpos = reinterpret_cast<const int32_t *>(a.desc + PIB_DESC_POS_OFF);
    const int       rstride = a.E + (a.vsep ? 1 : 2) * a.GQA;
    const __half *  vhead = a.vcache + (size_t) kvh * HD;
    const __half *  khead = a.kcache + (size_t) kvh * HD;
    float *         s = sm.s;

    // ---- rotate: pair j of a head = elements (2j, 2j+1), or (j, j + HD/2) in NeoX mode; unfused multiplies as the reference (-std=c11).  Items: K rows of the batch's
    // tokens, this block's query (row ntok), V rows of the batch's tokens -- one pass of loads
    {
        int       it = 0;
        const int nrot = (ntok + 1) * half, nall = nrot + ntok * half;
        for (int i = tid; i < nall; i += THREADS, it++) {
            if (i < nrot) {
                const int     r = i / half, j = i - r * half;
                const int     tok = r < ntok ? r : t;
                const float * src = a.qkv + (size_t) tok * rstride + (r < ntok ? a.E + (size_t) kvh * HD : (size_t) head * HD);
                const float2  cs  = it == 0 ? p.cs[0] : it == 1 ? p.cs[1] : a.rope[(size_t) min(tpos[tok], a.rope_n_pos - 1) * half + j];
                const int     i0 = (a.mode & 2) ? j : 2 * j, i1 = (a.mode & 2) ? j + half : 2 * j + 1;
                const float   x0 = src[i0], x1 = src[i1];
                const __half  y0 = __float2half_rn(__fsub_rn(__fmul_rn(x0, cs.x), __fmul_rn(x1, cs.y)));
                const __half  y1 = __float2half_rn(__fadd_rn(__fmul_rn(x0, cs.y), __fmul_rn(x1, cs.x)));
                if (r < ntok) { sm.kb[r * HD + i0] = y0; sm.kb[r * HD + i1] = y1; }
                else          { sm.sq[i0] = __half2float(y0); sm.sq[i1] = __half2float(y1); }
            } else {
                const int     k = i - nrot, r = k / half, d = 2 * (k - r * half), c = cell0 + r;
                const float * v = a.vsep ? a.vsep + (size_t) r * a.GQA : a.qkv + (size_t) r * rstride + a.E + a.GQA;
                const __half2 h = __floats2half2_rn(v[(size_t) kvh * HD + d], v[(size_t) kvh * HD + d + 1]);
                *reinterpret_cast<__half2 *>(sm.vb + r * HD + d) = h;
                if (c < min(n, a.vcap)) *reinterpret_cast<__half2 *>(sm.vs + (size_t) c * HD + d) = h;       // in the place that the prefetch left open
            }
        }
    }
    __syncthreads();
    if (head == kvh * a.gdiv) {                         // first query head of the group: this token's K / V row goes to the cache
        const size_t co = (size_t) (cell0 + t) * a.GQA + (size_t) kvh * HD;
        if (tid < HD / 8) reinterpret_cast<uint4 *>(a.kcache + co)[tid] = reinterpret_cast<const uint4 *>(sm.kb + t * HD)[tid];
        else if (tid < HD / 4) reinterpret_cast<uint4 *>(a.vcache + co)[tid - HD / 8] = reinterpret_cast<const uint4 *>(sm.vb + t * HD)[tid - HD / 8];
    }

    // ---- phase 1: scores, in the reference's order (ggml_vec_dot_f16, ggml.c:1200-1235 with the AVX2 reduce macro :772-790):
    // 32 fp32 accumulators, element e of the head goes to accumulator e mod 32, then ((0+2)+(1+3)) over the four 8-lane
    // vectors, low half + high half, two horizontal adds.
    // A cell is shared by two neighbouring lanes: the even one forms vectors 0 and 2 of the four, the odd one 1 and 3, and the
    // first addition of the reduce -- (0 + 2) and (1 + 3) -- happens before the halves meet through one shuffle per lane; both lanes then know the score.
    auto score = [&](int ic, bool live, const uint4 (&kg)[HD / 16]) -> float {
        if (!__any_sync(0xffffffffu, live)) return -INFINITY;
        const int bi = ic - cell0;
        uint4 kreg[HD / 16];
#pragma unroll
        for (int q = 0; q < HD / 16; q++) kreg[q] = kg[q];
        if (bi >= 0 && bi < ntok) {
            const uint4 * kr = reinterpret_cast<const uint4 *>(sm.kb + bi * HD);
#pragma unroll
            for (int q = 0; q < HD / 16; q++) kreg[q] = kr[(q >> 1) * 4 + 2 * (q & 1) + hsel];
        }
        float acc[2][8];
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int l = 0; l < 8; l++) acc[j][l] = 0.f;
#pragma unroll
        for (int st = 0; st < HD / 32; st++)
#pragma unroll
            for (int jj = 0; jj < 2; jj++) {
                const int     j  = 2 * jj + hsel;
                const uint4   k8 = kreg[st * 2 + jj];
                const __half2 h0 = *reinterpret_cast<const __half2 *>(&k8.x), h1 = *reinterpret_cast<const __half2 *>(&k8.y);
                const __half2 h2 = *reinterpret_cast<const __half2 *>(&k8.z), h3 = *reinterpret_cast<const __half2 *>(&k8.w);
                const float4  qa = *reinterpret_cast<const float4 *>(sm.sq + st * 32 + j * 8), qb = *reinterpret_cast<const float4 *>(sm.sq + st * 32 + j * 8 + 4);
                acc[jj][0] = fmaf(__low2float(h0), qa.x, acc[jj][0]); acc[jj][1] = fmaf(__high2float(h0), qa.y, acc[jj][1]);
                acc[jj][2] = fmaf(__low2float(h1), qa.z, acc[jj][2]); acc[jj][3] = fmaf(__high2float(h1), qa.w, acc[jj][3]);
                acc[jj][4] = fmaf(__low2float(h2), qb.x, acc[jj][4]); acc[jj][5] = fmaf(__high2float(h2), qb.y, acc[jj][5]);
                acc[jj][6] = fmaf(__low2float(h3), qb.z, acc[jj][6]); acc[jj][7] = fmaf(__high2float(h3), qb.w, acc[jj][7]);
            }
        float r[8];
#pragma unroll
        for (int l = 0; l < 8; l++) {
            r[l] = __fadd_rn(acc[0][l], acc[1][l]);                                     // even lane: 0 + 2, odd lane: 1 + 3
            const float o = __shfl_xor_sync(0xffffffffu, r[l], 1);
            r[l] = hsel ? __fadd_rn(o, r[l]) : __fadd_rn(r[l], o);                      // (0 + 2) + (1 + 3)
        }
        const float t0 = __fadd_rn(r[0], r[4]), t1 = __fadd_rn(r[1], r[5]), t2 = __fadd_rn(r[2], r[6]), t3 = __fadd_rn(r[3], r[7]);
        const float sc = __fmul_rn(__fadd_rn(__fadd_rn(t0, t1), __fadd_rn(t2, t3)), a.kq_scale);
        return live ? sc : -INFINITY;
    };
    // of every two rounds the even lane keeps the first one's score and the odd lane the second one's: a thread owns cell `mine`, held in a register
    // for the first THREADS cells and in s[] beyond
    const int mine = hsel * (THREADS / 2) + (tid >> 1);
    float     own = -INFINITY, lmax;
#pragma unroll
    for (int rd = 0; rd < 2; rd++) {
        if (rd * (THREADS / 2) >= n) break;
        const int i = rd * (THREADS / 2) + (tid >> 1), ic = max(min(i, n - 1), 0);
        float sc;
        if (rd < PRE) sc = score(ic, p.live[rd < PRE ? rd : 0], p.k[rd < PRE ? rd : 0]);
        else {
            // the row's address does not depend on the mask byte, both loads go out together
            uint4 kg[HD / 16];
            const uint4 * kr = reinterpret_cast<const uint4 *>(khead + (size_t) ic * a.GQA);
            const bool    inb = ic >= cell0 && ic < cell0 + ntok;
#pragma unroll
            for (int q = 0; q < HD / 16; q++) kg[q] = inb ? make_uint4(0, 0, 0, 0) : kr[(q >> 1) * 4 + 2 * (q & 1) + hsel];
            sc = score(ic, i < n && !mrow[ic], kg);
        }
        if (rd == hsel) own = sc;
    }
    lmax = own;
#pragma unroll 1
    for (int i0 = THREADS; i0 < n; i0 += THREADS / 2) {
        const int     i = i0 + (tid >> 1), ic = max(min(i, n - 1), 0);
        const bool    inb = ic >= cell0 && ic < cell0 + ntok;
        uint4         kg[HD / 16];
        const uint4 * kr = reinterpret_cast<const uint4 *>(khead + (size_t) ic * a.GQA);
#pragma unroll
        for (int q = 0; q < HD / 16; q++) kg[q] = inb ? make_uint4(0, 0, 0, 0) : kr[(q >> 1) * 4 + 2 * (q & 1) + hsel];
        const float sc = score(ic, i < n && !mrow[ic], kg);
        if (i < n && !hsel) s[i] = sc;
        lmax = fmaxf(lmax, sc);
    }
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(lmax) : "f"(lmax));
    if (lane == 0) sm.redf[warp] = lmax;
    __syncthreads();
    float mx = sm.redf[0];
#pragma unroll
    for (int w = 1; w < NW; w++) mx = fmaxf(mx, sm.redf[w]);

    // ---- phase 2: exp through the fp16 table, exact double sum (of fp16 values, the same in any order), fp16-rounded probabilities
    double sum = 0.0;
    float  ev = 0.f;
    if (own != -INFINITY) { ev = pib_h2f(a.exp_lut[pib_f2h(__fsub_rn(own, mx))]); sum = (double) ev; }
    for (int i = THREADS + tid; i < n; i += THREADS) {
        const float x = s[i];
        float       v = 0.0f;
        if (x != -INFINITY) { v = pib_h2f(a.exp_lut[pib_f2h(__fsub_rn(x, mx))]); sum += (double) v; }
        s[i] = v;
    }
    sum = warp_sum_d(sum);
    if (lane == 0) sm.redd[warp] = sum;
    asm volatile("cp.async.wait_all;" ::: "memory");              // this thread's V chunks have landed; the barrier publishes them
    __syncthreads();
    double tot[4] = { 0.0, 0.0, 0.0, 0.0 };
#pragma unroll
    for (int w = 0; w < NW; w++) tot[w & 3] += sm.redd[w];
    const float inv = (float) (1.0 / ((tot[0] + tot[1]) + (tot[2] + tot[3])));
    if (mine < n) s[mine] = __half2float(__float2half_rn(__fmul_rn(ev, inv)));
    for (int i = THREADS + tid; i < n; i += THREADS) s[i] = __half2float(__float2half_rn(__fmul_rn(s[i], inv)));
    __syncthreads();

    // ---- phase 3: O = V . P in the reference's order (the same ggml_vec_dot_f16, now over the cells): cell c < np = n & ~31 goes
    // to accumulator c mod 32, each accumulator a sequential fma chain over its cells; then the same tree per output element;
    // the n - np cells left over are added one by one in double.  A thread owns four coordinates and APG of the 32
    // accumulators; the 32 x HD partial sums meet in shared memory.
    constexpr int LPR = HD / 4, NGR = THREADS / LPR, APG = 32 / NGR;           // 512 threads: 1 accumulator for heads of 64, 2 for 128; 256: 4
    const int grp = tid / LPR, d4 = (tid % LPR) * 4;
    const int np  = n & ~31, nv = min(n, a.vcap);
    // four halves of cell c's row, staged, of the batch or in the cache; a weight of 0 leaves the sums as they are (and the row may never have been written)
    auto vrow = [&](int c, float pw) -> uint2 {
        const int      bi = c - cell0;
        const __half * vr = c < nv ? sm.vs + (size_t) c * HD : bi >= 0 && bi < ntok ? sm.vb + bi * HD : vhead + (size_t) c * a.GQA;
        uint2          v  = make_uint2(0, 0);
        if (pw != 0.f) v = *reinterpret_cast<const uint2 *>(vr + d4);
        return v;
    };
    float o[APG][4];
#pragma unroll
    for (int u = 0; u < APG; u++) { o[u][0] = o[u][1] = o[u][2] = o[u][3] = 0.f; }
    auto add = [&](int u, const uint2 v, float pw) {
        const float2 a0 = __half22float2(*reinterpret_cast<const __half2 *>(&v.x)), a1 = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
        o[u][0] = fmaf(a0.x, pw, o[u][0]); o[u][1] = fmaf(a0.y, pw, o[u][1]); o[u][2] = fmaf(a1.x, pw, o[u][2]); o[u][3] = fmaf(a1.y, pw, o[u][3]);
    };
    const int ns = min(np, nv & ~31);                                          // staged rows of whole groups of 32
#pragma unroll 4
    for (int base = 0; base < ns; base += 32)
#pragma unroll
        for (int u = 0; u < APG; u++) {
            const int   c  = base + grp * APG + u;
            const float pw = s[c];
            const uint2 v  = *reinterpret_cast<const uint2 *>(sm.vs + (size_t) c * HD + d4);
            add(u, pw == 0.f ? make_uint2(0, 0) : v, pw);
        }
#pragma unroll 4
    for (int base = ns; base < np; base += 32)
#pragma unroll
        for (int u = 0; u < APG; u++) {
            const int   c  = base + grp * APG + u;
            const float pw = s[c];
            add(u, vrow(c, pw), pw);
        }
#pragma unroll
    for (int u = 0; u < APG; u++) *reinterpret_cast<float4 *>(sm.red + (grp * APG + u) * HD + d4) = make_float4(o[u][0], o[u][1], o[u][2], o[u][3]);
    __syncthreads();
    if (tid < HD) {
        float r[8];
#pragma unroll
        for (int l = 0; l < 8; l++)
            r[l] = __fadd_rn(__fadd_rn(sm.red[(0 * 8 + l) * HD + tid], sm.red[(2 * 8 + l) * HD + tid]), __fadd_rn(sm.red[(1 * 8 + l) * HD + tid], sm.red[(3 * 8 + l) * HD + tid]));
        const float t0 = __fadd_rn(r[0], r[4]), t1 = __fadd_rn(r[1], r[5]), t2 = __fadd_rn(r[2], r[6]), t3 = __fadd_rn(r[3], r[7]);
        double sumf = (double) __fadd_rn(__fadd_rn(t0, t1), __fadd_rn(t2, t3));
        // eight products at a time, only the additions wait for one another; -0 leaves every sum as it is
        if (n <= nv) {
            const __half * v0 = sm.vs + tid;
            for (int c0 = np; c0 < n; c0 += 8) {
                float x[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int   c  = min(c0 + k, n - 1);
                    const float pw = s[c], m = __fmul_rn(__half2float(v0[c * HD]), pw);
                    x[k] = c0 + k < n && pw != 0.f ? m : -0.f;
                }
#pragma unroll
                for (int k = 0; k < 8; k++) sumf += (double) x[k];
            }
        } else
            for (int c = np; c < n; c++) {
                const float    pw = s[c];
                const int      bi = c - cell0;
                const __half * vr = c < nv ? sm.vs + (size_t) c * HD : bi >= 0 && bi < ntok ? sm.vb + bi * HD : vhead + (size_t) c * a.GQA;
                if (pw != 0.f) sumf += (double) __fmul_rn(__half2float(vr[tid]), pw);
            }
        a.out[(size_t) t * a.E + (size_t) head * HD + tid] = (float) sumf;
    }
}

// grid (n_head, n_tokens), 256 or 512 threads; one CTA per (query head, token).  Every fp32 sum is formed in the reference's order
// (ggml_vec_dot_f16 for both K.Q and V.P), so the output is bit-identical to the CPU's: phase 1 gives two threads a cell
// (a K row in 128-bit loads, the 32 lane accumulators of the reference in registers); phase 3 gives every thread four
// output dims and a share of the 32 accumulators, each a sequential chain over its cells.  K/V of a KV head are re-read by its
// G query heads through L2 -- a few MB per layer at these context lengths.  Masked cells are never loaded.
#define ATQ_VCAP_MIN 256
#define ATQ_VCAP(hd) ((hd) == 64 ? 704 : 384)     /* V rows staged in shared memory; later cells are read from global memory (512 cells, heads of 64: 5.4 us with 384 rows, 4.4 with 704) */
// RoPE, KV store and attention in one launch.  A CTA rotates its own query head itself, rotates / converts the K and V rows of
// ALL tokens of the batch for its KV head into shared memory (<= 16 rows: the batch's cells are the contiguous range starting at
// the descriptor's kv head, and a token of a tree batch attends to earlier tokens of the same batch), and the first query head
// of each KV group also writes its token's K / V row to the cache.  Cells of the batch are therefore never read from global
// memory, cells outside it never written: no ordering between CTAs is needed.  Values and roundings are the reference's
// (rope_f32 ggml.c:11006, dup f32 -> f16 :6528).
//
// The kernel is a chain of dependent memory round trips, not of arithmetic, so everything that does not depend on the QKV
// projection is fetched BEFORE the wait on it: the descriptor words and positions, the RoPE entries, the mask bytes and K rows of
// the first 512 or 128 cells (registers), and the V rows of up to ATQ_VCAP cells (cp.async into shared memory).  All of it was final
// before this launch's predecessor started: cache rows of earlier decodes, and the mask / scalars of the pass's first kernels.
//
// 512 threads: two rounds of K rows in flight and half the rounds.  Heads of 128 coordinates take 512 threads while a CTA per SM serves the launch and 256 with two CTAs
// per SM beyond.  A chain of launches, us each, before / after the parts behind the projection were shortened: 32 heads of 64, one token, 301 / 931 cells 7.6 / 4.2 and
// 15.3 / 8.8, 16 tokens 512 / 931 cells 26.4 / 17.0 and 43.7 / 29.2; heads of 128, 204 cells, 1 / 4 tokens 8.9 / 4.3 and 9.9 / 5.9, 301 cells, 16 tokens 34.8 / 25.1.
template <int HD, int ATQ_THREADS>
__global__ void __launch_bounds__(ATQ_THREADS, HD == 64 || ATQ_THREADS == 256 ? 2 : 1) attention_qh_kernel(const att_args a, const int * __restrict__ cancel) {
    extern __shared__ __align__(16) uint8_t att_sm[];
    const att_smem<HD, ATQ_THREADS> sm(att_sm, a.n_ctx, a.vcap);
    const int head = blockIdx.x, t = blockIdx.y;
    att_pre<HD, ATQ_THREADS> p;
    att_prefetch(a, sm, head, t, p);
    pib_pdl_wait();
    pib_pdl_trigger();
    if (PIB_CANCELLED(cancel)) { asm volatile("cp.async.wait_all;" ::: "memory"); return; }
    att_compute(a, sm, head, t, p);
}

// V rows staged by a context: the larger number unless a long score row needs the room
#define ATQ_SMEM_MAX(hd) (200 * 1024 + att_fixed_smem(hd))
template <int HD, int ATQ_THREADS>
static int launch_att_qh(const float * qkv, const float * vsep, const uint8_t * desc, const float2 * rope, int rope_n_pos, int mode, __half * kc, __half * vc,
                         const uint8_t * mask, const int32_t * scalars, int E, int GQA, int n_ctx, int n_tokens, int n_head, int gdiv, float * out,
                         const int * cancel, cudaStream_t st) {
    // as many V rows as are worth it while two CTAs of heads of 64 share an SM (a long score row leaves room for fewer)
    int vcap = ATQ_VCAP_MIN;
    if (ATQ_THREADS == 512) {
        vcap = ATQ_VCAP(HD);
        if (HD == 64 && 2 * (att_core_smem(HD, n_ctx, vcap) + 1024) > 228 * 1024) vcap = 384;
        if (att_core_smem(HD, n_ctx, vcap) > ATQ_SMEM_MAX(HD)) vcap = ATQ_VCAP_MIN;
    }
    vcap = std::min(n_ctx, vcap);
    const size_t smem = att_core_smem(HD, n_ctx, vcap);   // scores + 32 x HD partial sums + staged V rows
    static pib_per_device attrs;
    // several CTAs per SM (a verification batch of 3+ tokens is more CTAs than SMs): ask for the large shared-memory carve-out
    PIB_CHECK(attrs.once(smem, [&] {
        const cudaError_t e = cudaFuncSetAttribute(attention_qh_kernel<HD, ATQ_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) std::max(smem, (size_t) 32 * 1024));
        return e != cudaSuccess ? e : cudaFuncSetAttribute(attention_qh_kernel<HD, ATQ_THREADS>, cudaFuncAttributePreferredSharedMemoryCarveout, (int) cudaSharedmemCarveoutMaxShared);
    }));
    att_args a = { qkv, vsep, desc, rope, rope_n_pos, mode, kc, vc, mask, scalars, pib_get_luts().exp_f16, E, GQA, n_ctx, gdiv, vcap, 1.0f / sqrtf((float) HD), out };
    PIB_CHECK(pib_launch(attention_qh_kernel<HD, ATQ_THREADS>, dim3(n_head, n_tokens), dim3(ATQ_THREADS), smem, st, a, cancel));
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

bool pib_attention_supported(int hd, int n_head, int n_head_kv, int n_ctx) {
    if (hd != 64 && hd != 128) return false;
    if (n_head % n_head_kv) return false;
    return att_core_smem(hd, n_ctx, ATQ_VCAP_MIN) <= ATQ_SMEM_MAX(hd);      // the scores of one (head, token) live in shared memory
}

// RoPE (mode 0: adjacent pairs, 2: NeoX) + KV store + attention of one chunk: qkv = the fused projection's output [n_tokens][E + 2 GQA]
// (or [E + GQA] with V in vsep)
int pib_attention(const float * qkv, const float * vsep, const uint8_t * desc, const float2 * rope, int rope_n_pos, int mode, __half * kc, __half * vc,
                  const uint8_t * mask, const int32_t * scalars, int n_tokens, int n_head, int n_head_kv, int hd, int n_ctx, float * out,
                  const int * cancel, cudaStream_t st) {
    const int E = n_head * hd, GQA = n_head_kv * hd, G = n_head / n_head_kv;
#define ATQ_GO(HD, NT) return launch_att_qh<HD, NT>(qkv, vsep, desc, rope, rope_n_pos, mode, kc, vc, mask, scalars, E, GQA, n_ctx, n_tokens, n_head, G, out, cancel, st)
    if (hd == 128) { if (n_head * n_tokens <= pib_num_sms()) ATQ_GO(128, 512); else ATQ_GO(128, 256); }
    if (hd == 64)  ATQ_GO(64, 512);
#undef ATQ_GO
    pib_set_error("attention: unsupported head_dim %d", hd);
    return PIB_ERR_UNSUPP;
}
