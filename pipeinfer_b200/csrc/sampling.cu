// sampling.cu -- device-side token acceptance inputs (K10 / R9): per-row argmax and sorted top-8 probabilities.
//
// The reference pulls n_vocab floats per sampled row to the host and runs std::sort over the whole vocabulary there
// (common/sampling.cpp:131, llama.cpp:7019-7046 llama_sample_softmax, :7496 llama_sample_token_greedy).  Here the
// logits stay in HBM; per row the host receives 8 x {id, logit, p} (the llama_token_data the scheduler consumes at
// speculative.cpp:977-1010), entry 0 being the greedy token:
//   id    first index of the maximum (std::max_element semantics)
//   p_i   expf(l_i - max) / sum_j expf(l_j - max); the sum is accumulated in double (the reference adds floats in
//         sorted order), so p agrees to ~1e-7 relative -- the ids are exact.
// logit_bias entries (e.g. EOS = -inf under --ignore-eos, common.cpp:1061-1063 / sampling.cpp:134-136) are applied
// in the kernel before anything else, in place, as the reference does.
#include "engine.cuh"

#include <cooperative_groups.h>

// A row is divided over P blocks of a thread-block cluster (contiguous slices of the vocabulary); each finds the best eight and, once the cluster knows the maximum,
// the exponentials' sum of its slice, and the first block merges the P sorted lists and sums through distributed shared memory.
// What bounds it: chains of block-wide rounds.  One block of 1024 threads per row took 27 us for a row of 32 000 (16 for 8 000), whatever the number of rows.
#define SMP_THREADS 256
#define SMP_TOPK    8
#define SMP_PARTS   8
#define SMP_REG     32
#define SMP_NONE    0x7fffffff

// b is ahead of a: larger, or equal and earlier (std::max_element semantics); places without an element come last
__device__ __forceinline__ bool smp_ahead(float bv, int bi, float av, int ai) { return bi != SMP_NONE && (ai == SMP_NONE || bv > av || (bv == av && bi < ai)); }

__global__ void __launch_bounds__(SMP_THREADS) sample_topk_kernel(float * __restrict__ logits, int n_vocab,
                                                                  const int32_t * __restrict__ bias_ids, const float * __restrict__ bias_val,
                                                                  int n_bias, pib_row_result * __restrict__ out, const int * __restrict__ cancel) {
    pib_pdl_wait();
    pib_pdl_trigger();
    constexpr int NW = SMP_THREADS / 32;
    __shared__ float  s_val[2][NW], s_top[SMP_TOPK];
    __shared__ int    s_idx[2][NW], s_topi[SMP_TOPK];
    __shared__ double s_sum[NW], s_total;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int P = gridDim.y, part = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *   l = logits + (size_t) blockIdx.x * n_vocab;
    // a cancelled run's blocks have nothing to do but stay for the cluster's barriers
    const bool off = PIB_CANCELLED(cancel);
    const int  lo = (int) ((long long) n_vocab * part / P), hi = off ? lo : (int) ((long long) n_vocab * (part + 1) / P);
    for (int k = tid; k < n_bias; k += SMP_THREADS) if (bias_ids[k] >= lo && bias_ids[k] < hi) l[bias_ids[k]] += bias_val[k];
    __syncthreads();
    // A thread keeps its elements in registers when they are at most SMP_REG (all loads in flight together) and looks for its best one only; otherwise one pass keeps
    // the 8 largest of its strided elements, sorted (value descending, index ascending: the indices a thread sees only grow, so strict comparisons keep the
    // earlier one of two equal values in front)
    const bool few = hi - lo <= SMP_REG * SMP_THREADS;
    float tv[SMP_REG];
    int   ti[SMP_TOPK];
    auto best_of = [&](float & bv, int & bi) {                    // few: the best element left; taken ones are marked in `gone`
        bv = -INFINITY; bi = SMP_NONE;
#pragma unroll
        for (int j = 0; j < SMP_REG; j++) {
            const int i = lo + tid + j * SMP_THREADS;
            if (i < hi && !((uint32_t) ti[0] >> j & 1u) && (bi == SMP_NONE || tv[j] > bv)) { bv = tv[j]; bi = i; }
        }
    };
    float hv;
    int   hidx;
    if (few) {
#pragma unroll
        for (int j = 0; j < SMP_REG; j++) { const int i = lo + tid + j * SMP_THREADS; tv[j] = i < hi ? l[i] : -INFINITY; }
        ti[0] = 0;                                                // bit j: element j has been taken
        best_of(hv, hidx);
    } else {
#pragma unroll
        for (int j = 0; j < SMP_TOPK; j++) { tv[j] = -INFINITY; ti[j] = SMP_NONE; }
#pragma unroll 4
        for (int i = lo + tid; i < hi; i += SMP_THREADS) {
            const float v = l[i];
            if (v > tv[SMP_TOPK - 1] || ti[SMP_TOPK - 1] == SMP_NONE) {
                tv[SMP_TOPK - 1] = v; ti[SMP_TOPK - 1] = i;
#pragma unroll
                for (int j = SMP_TOPK - 1; j > 0; j--) {
                    if (tv[j] > tv[j - 1] || ti[j - 1] == SMP_NONE) {
                        const float fv = tv[j]; tv[j] = tv[j - 1]; tv[j - 1] = fv;
                        const int   fi = ti[j]; ti[j] = ti[j - 1]; ti[j - 1] = fi;
                    }
                }
            }
        }
        hv = tv[0]; hidx = ti[0];
    }
    // eight rounds over the heads of the per-thread lists; every warp finds the block's best from the warps' (two sets of places: one barrier per round)
    for (int k = 0; k < SMP_TOPK; k++) {
        float bv = hv;
        int   bi = hidx;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int   oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (smp_ahead(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { s_val[k & 1][warp] = bv; s_idx[k & 1][warp] = bi; }
        __syncthreads();
        bv = s_val[k & 1][lane % NW]; bi = s_idx[k & 1][lane % NW];
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int   oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (smp_ahead(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (tid == 0) { s_top[k] = bv; s_topi[k] = bi; }
        if (hidx == bi && bi != SMP_NONE) {                       // the winner pops its head
            if (few) {
                ti[0] |= 1u << ((bi - lo - tid) / SMP_THREADS);
                best_of(hv, hidx);
            } else {
#pragma unroll
                for (int j = 0; j < SMP_TOPK - 1; j++) { tv[j] = tv[j + 1]; ti[j] = ti[j + 1]; }
                tv[SMP_TOPK - 1] = -INFINITY; ti[SMP_TOPK - 1] = SMP_NONE;
                hv = tv[0]; hidx = ti[0];
            }
        }
    }
    if (P > 1) cl.sync(); else __syncthreads();
    // the row's maximum: lane p looks at part p's best (one remote load each, not P in a row)
    float max_l = lane >= P ? -INFINITY : P > 1 ? *cl.map_shared_rank(s_top, lane) : s_top[0];
    {
        int mi = lane >= P ? SMP_NONE : P > 1 ? *cl.map_shared_rank(s_topi, lane) : s_topi[0];
#pragma unroll
        for (int o = SMP_PARTS / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, max_l, o);
            const int   oi = __shfl_xor_sync(0xffffffffu, mi, o);
            if (smp_ahead(ov, oi, max_l, mi)) { max_l = ov; mi = oi; }
        }
        max_l = __shfl_sync(0xffffffffu, max_l, 0);
    }
    double sum = 0.0;
    if (few) {
#pragma unroll
        for (int j = 0; j < SMP_REG; j++) if (lo + tid + j * SMP_THREADS < hi) sum += (double) expf(tv[j] - max_l);
    } else for (int i = lo + tid; i < hi; i += SMP_THREADS) sum += (double) expf(l[i] - max_l);
    sum = warp_sum_d(sum);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < NW; w++) t += s_sum[w];
        s_total = t;
    }
    if (P > 1) cl.sync(); else __syncthreads();
    if (part == 0 && warp == 0) {
        // lane p < P walks part p's sorted list
        const float * pv = P > 1 ? cl.map_shared_rank(s_top, lane < P ? lane : 0) : s_top;
        const int *   pi = P > 1 ? cl.map_shared_rank(s_topi, lane < P ? lane : 0) : s_topi;
        float mv[SMP_TOPK];
        int   mi[SMP_TOPK];
#pragma unroll
        for (int j = 0; j < SMP_TOPK; j++) { mv[j] = lane < P ? pv[j] : -INFINITY; mi[j] = lane < P ? pi[j] : SMP_NONE; }
        const double mine = lane >= P ? 0.0 : P > 1 ? *cl.map_shared_rank(&s_total, lane) : s_total;
        double t = 0.0;
#pragma unroll
        for (int p = 0; p < SMP_PARTS; p++) t += __shfl_sync(0xffffffffu, mine, p);
        for (int k = 0; k < SMP_TOPK; k++) {
            float bv = mv[0];
            int   bi = mi[0];
#pragma unroll
            for (int o = SMP_PARTS / 2; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int   oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (smp_ahead(ov, oi, bv, bi)) { bv = ov; bi = oi; }
            }
            if (lane == 0 && !off) {
                out[blockIdx.x].id[k]    = bi == SMP_NONE ? 0 : bi;
                out[blockIdx.x].logit[k] = bv;
                out[blockIdx.x].p[k]     = (float) ((double) expf(bv - max_l) / t);
            }
            if (mi[0] == bi && bi != SMP_NONE) {
#pragma unroll
                for (int j = 0; j < SMP_TOPK - 1; j++) { mv[j] = mv[j + 1]; mi[j] = mi[j + 1]; }
                mv[SMP_TOPK - 1] = -INFINITY; mi[SMP_TOPK - 1] = SMP_NONE;
            }
        }
    }
    if (P > 1) cl.sync();                                         // the other blocks' lists have been read
}

int pib_sample_topk(float * logits_dev, int n_rows, int n_vocab, const int32_t * bias_ids_dev, const float * bias_val_dev,
                    int n_bias, void * out_dev, const uint8_t * desc, const int * cancel, cudaStream_t st) {
    (void) desc;
    // as many parts as the register form needs (8192 elements each), more while the machine has room for the blocks and a thread would have more than four elements
    int P = 1;
    while (P < SMP_PARTS && (n_vocab > P * SMP_REG * SMP_THREADS || ((long long) n_rows * P * 2 <= 4LL * pib_num_sms() && n_vocab >= P * 8 * SMP_THREADS))) P <<= 1;
    if (P > 1) pib_launch_cluster(sample_topk_kernel, dim3((unsigned) n_rows, (unsigned) P), dim3(SMP_THREADS), dim3(1, (unsigned) P, 1), 0, st, logits_dev, n_vocab, bias_ids_dev, bias_val_dev, n_bias,
                                  (pib_row_result *) out_dev, cancel);
    else       pib_launch(sample_topk_kernel, dim3((unsigned) n_rows), dim3(SMP_THREADS), 0, st, logits_dev, n_vocab, bias_ids_dev, bias_val_dev, n_bias, (pib_row_result *) out_dev, cancel);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

// ---- acceptance walk (reference speculative.cpp:439-560, greedy) ----------------------------------------------------------------
// The verification loop of the scheduler, on the device that holds the sampled rows: start on branch `keep` at depth 0; sample the
// target's token at that branch's row; every active branch whose drafted token at this depth differs is dropped, the first that
// agrees becomes the branch to follow; stop at the first depth where none agrees.  Only the ids sampled along the way (and the
// branch kept) cross to the host: 8 + 4 * n_ids bytes instead of 96 bytes per row.
__global__ void accept_walk_kernel(const pib_row_result * __restrict__ rows, const uint8_t * __restrict__ desc, pib_accept_result * __restrict__ out,
                                   const int * __restrict__ cancel) {
    pib_pdl_wait();
    pib_pdl_trigger();
    if (threadIdx.x != 0) return;
    const int32_t * hdr = reinterpret_cast<const int32_t *>(desc + PIB_DESC_HDR_OFF);
    const int np = hdr[PIB_DH_TREE_NP];
    if (np <= 0 || PIB_CANCELLED(cancel)) { out->n_ids = 0; out->s_keep = 0; return; }
    const int32_t * len = reinterpret_cast<const int32_t *>(desc + PIB_DESC_TREE_OFF);
    const int32_t * trow = len + PIB_TREE_NP, * ttok = trow + PIB_TREE_NP * PIB_TREE_DEPTH;
    int  keep = hdr[PIB_DH_TREE_KEEP], n = 0, i = 0;
    bool act[PIB_TREE_NP];
    for (int s = 0; s < PIB_TREE_NP; s++) act[s] = s < np && len[s] >= 0;
    while (n < PIB_CHUNK + 2 && i < PIB_TREE_DEPTH) {
        const int id = rows[trow[keep * PIB_TREE_DEPTH + i]].id[0];
        out->ids[n++] = id;
        if (!hdr[PIB_DH_TREE_SPEC]) break;
        bool matches = false;
        for (int s = 0; s < np; s++) {
            if (!act[s]) continue;
            if (i < len[s] && id == ttok[s * PIB_TREE_DEPTH + i]) { if (!matches) keep = s; matches = true; }
            else act[s] = false;
        }
        if (!matches) break;
        i++;
    }
    out->n_ids = n;
    out->s_keep = keep;
}

int pib_accept_walk(const void * rows_dev, const uint8_t * desc, void * out_dev, const int * cancel, cudaStream_t st) {
    pib_launch(accept_walk_kernel, dim3(1), dim3(32), 0, st, (const pib_row_result *) rows_dev, desc, (pib_accept_result *) out_dev, cancel);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}
