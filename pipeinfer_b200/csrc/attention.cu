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
#include "attention_core.cuh"

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
// grid (n_head, n_tokens), 256 or 512 threads; one CTA per (query head, token).  Every fp32 sum is formed in the reference's order
// (ggml_vec_dot_f16 for both K.Q and V.P), so the output is bit-identical to the CPU's: phase 1 gives two threads a cell
// (a K row in 128-bit loads, the 32 lane accumulators of the reference in registers); phase 3 gives every thread four
// output dims and a share of the 32 accumulators, each a sequential chain over its cells (attention_core.cuh).  K/V of a KV head are re-read by its
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
    auto cpwait = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
    if (PIB_CANCELLED(cancel)) { cpwait(); return; }
    att_compute(a, sm, head, t, p, [] { __syncthreads(); }, cpwait);
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
