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
// What bounds it: chains of rounds; a round is two reductions in hardware (redux on order-preserving keys), a thread looks for its best two only, eight lanes write the eight results.
// A few rows: every warp finds its own best eight without a barrier, one warp the best of the warps' lists (two places per lane), and up to 32 values per thread wait in registers for
// the exponentials (behind cold rows, us, before / now: one row of 32 000 12.7 / 11.1, 4 rows of 8 000 12.2 / 10.2; between a matmul and a copy 10.8 / 8.9).  Many rows: rounds of the
// block with a barrier each, since a warp's eight come from the same thread often enough for its look behind its best two to cost (700 rows of 32 000 56 us, 137 with lists per
// warp); with the results by eight lanes 256 rows of 32 000 36 -> 25, 1 512 of 8 000 41 -> 28.
#define SMP_THREADS 256
#define SMP_TOPK    8
#define SMP_PARTS   8
#define SMP_NONE    0x7fffffff

// order-preserving keys: larger value, larger key, the two zeros one key (the sum is +0 for both); what is no number comes last, but in front of places without an element (0)
__device__ __forceinline__ uint32_t smp_key(float v) {
    const uint32_t u = __float_as_uint(v + 0.0f);
    return v != v ? 1u : (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
// the warp's best (key, index): the largest key, the smallest index among equals
__device__ __forceinline__ void smp_warp_best(uint32_t & key, int & idx) {
    const uint32_t k = __reduce_max_sync(0xffffffffu, key);
    idx = __reduce_min_sync(0xffffffffu, key == k ? idx : SMP_NONE);
    key = k;
}

// the best SMP_TOPK of the warp's candidates in order, lane r gets the r-th (key 0, SMP_NONE behind the last): a lane offers (k0, i0), then (k1, i1), then what `more` finds behind a given one
template <typename F> __device__ __forceinline__ void smp_warp_top(uint32_t k0, int i0, uint32_t k1, int i1, int lane, uint32_t & key, int & idx, F more) {
    key = 0; idx = SMP_NONE;
#pragma unroll 1
    for (int r = 0; r < SMP_TOPK; r++) {
        uint32_t bk = k0;
        int      bi = i0;
        smp_warp_best(bk, bi);
        if (bi == SMP_NONE) break;
        if (lane == r) { key = bk; idx = bi; }
        if (i0 == bi) {                                           // the winner gives its best away
            const uint32_t gk = k0;
            const int      gi = i0;
            k0 = k1; i0 = i1; k1 = 0; i1 = SMP_NONE;
            if (i0 == SMP_NONE) more(gk, gi, k0, i0);
        }
    }
}

// E: values that a thread keeps in registers; 0: slices of more, which are read again from memory
template <int E>
__global__ void __launch_bounds__(SMP_THREADS) sample_topk_kernel(float * __restrict__ logits, int n_vocab,
                                                                  const int32_t * __restrict__ bias_ids, const float * __restrict__ bias_val,
                                                                  int n_bias, pib_row_result * __restrict__ out, const int * __restrict__ cancel) {
    pib_pdl_wait();
    pib_pdl_trigger();
    constexpr int NW = SMP_THREADS / 32;
    __shared__ uint32_t s_key[NW * SMP_TOPK], s_topk[SMP_TOPK];
    __shared__ int      s_idx[NW * SMP_TOPK], s_topi[SMP_TOPK];
    __shared__ double   s_sum[NW], s_total;
    __shared__ float    s_best;                                   // the slice's maximum
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int P = gridDim.y, part = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *   l = logits + (size_t) blockIdx.x * n_vocab;
    // a cancelled run's blocks have nothing to do but stay for the cluster's barriers
    const bool off = PIB_CANCELLED(cancel);
    const int  lo = (int) ((long long) n_vocab * part / P), hi = off ? lo : (int) ((long long) n_vocab * (part + 1) / P);
    if (n_bias > 0) {
        for (int k = tid; k < n_bias; k += SMP_THREADS) if (bias_ids[k] >= lo && bias_ids[k] < hi) l[bias_ids[k]] += bias_val[k];
        __syncthreads();
    }
    float v[E ? E : 1];
    if (E) {
#pragma unroll
        for (int e = 0; e < E; e++) { const int i = lo + tid + e * SMP_THREADS; v[e] = i < hi ? l[i] : 0.f; }
    }
    // A thread walks its strided elements for the best two (key descending, index ascending: indices only grow, so strict comparisons keep the earlier one of equals in
    // front).  One that gives away both looks for its next among the elements behind the last one it gave: after it in (key descending, index ascending) order.
    uint32_t k0 = 0, k1 = 0;
    int      i0 = SMP_NONE, i1 = SMP_NONE;
    if (E) {
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int      i = lo + tid + e * SMP_THREADS;
            const uint32_t k = i < hi ? smp_key(v[e]) : 0u;
            if (k > k0) { k1 = k0; i1 = i0; k0 = k; i0 = i; }
            else if (k > k1) { k1 = k; i1 = i; }
        }
        auto behind = [&](uint32_t gk, int gi, uint32_t & nk, int & ni) {
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int      i = lo + tid + e * SMP_THREADS;
                const uint32_t k = i < hi ? smp_key(v[e]) : 0u;
                if ((k < gk || (k == gk && i > gi)) && k > nk) { nk = k; ni = i; }
            }
        };
        uint32_t wk;
        int      wi;
        smp_warp_top(k0, i0, k1, i1, lane, wk, wi, behind);
        if (lane < SMP_TOPK) { s_key[warp * SMP_TOPK + lane] = wk; s_idx[warp * SMP_TOPK + lane] = wi; }
        __syncthreads();
        if (warp == 0) {
            // the warps' lists, two places per lane
            uint32_t a = s_key[lane], b = s_key[lane + 32], tk;
            int      ai = s_idx[lane], bi = s_idx[lane + 32], ti;
            const bool swap = b > a || (b == a && bi < ai);
            smp_warp_top(swap ? b : a, swap ? bi : ai, swap ? a : b, swap ? ai : bi, lane, tk, ti, [](uint32_t, int, uint32_t &, int &) {});
            if (lane < SMP_TOPK) { s_topk[lane] = tk; s_topi[lane] = ti; }
            if (lane == 0) s_best = ti == SMP_NONE ? -INFINITY : l[ti];
        }
    } else {
#pragma unroll 8
        for (int i = lo + tid; i < hi; i += SMP_THREADS) {
            const uint32_t k = smp_key(l[i]);
            if (k > k0) { k1 = k0; i1 = i0; k0 = k; i0 = i; }
            else if (k > k1) { k1 = k; i1 = i; }
        }
        // eight rounds of the block; every warp finds the block's best from the warps' (two sets of places: one barrier per round)
        for (int r = 0; r < SMP_TOPK; r++) {
            uint32_t bk = k0;
            int      bi = i0;
            smp_warp_best(bk, bi);
            if (lane == 0) { s_key[(r & 1) * NW + warp] = bk; s_idx[(r & 1) * NW + warp] = bi; }
            __syncthreads();
            bk = s_key[(r & 1) * NW + lane % NW]; bi = s_idx[(r & 1) * NW + lane % NW];
            smp_warp_best(bk, bi);
            if (tid == 0) { s_topk[r] = bk; s_topi[r] = bi; if (r == 0) s_best = bi == SMP_NONE ? -INFINITY : l[bi]; }
            if (bi != SMP_NONE && i0 == bi) {                     // the winner gives its best away
                const uint32_t gk = k0;
                const int      gi = i0;
                k0 = k1; i0 = i1; k1 = 0; i1 = SMP_NONE;
                if (i0 == SMP_NONE) {
                    for (int i = lo + tid; i < hi; i += SMP_THREADS) {
                        const uint32_t k = smp_key(l[i]);
                        if ((k < gk || (k == gk && i > gi)) && k > k0) { k0 = k; i0 = i; }
                    }
                }
            }
        }
    }
    if (P > 1) cl.sync(); else __syncthreads();
    // the row's maximum: lane p looks at part p's best (one remote load each, not P in a row)
    float max_l = s_best;
    if (P > 1) {
        const int p = lane < P ? lane : 0;
        uint32_t  bk = *cl.map_shared_rank(s_topk, p);
        int       bi = *cl.map_shared_rank(s_topi, p);
        const float x = *cl.map_shared_rank(&s_best, p);
        if (lane >= P) { bk = 0; bi = SMP_NONE; }
        const uint32_t mine = bk;
        const int      idx = bi;
        smp_warp_best(bk, bi);
        const unsigned who = __ballot_sync(0xffffffffu, mine == bk && idx == bi);
        max_l = __shfl_sync(0xffffffffu, x, __ffs((int) who) - 1);
    }
    double sum = 0.0;
    if (E) {
#pragma unroll
        for (int e = 0; e < E; e++) if (lo + tid + e * SMP_THREADS < hi) sum += (double) expf(v[e] - max_l);
    } else {
#pragma unroll 8
        for (int i = lo + tid; i < hi; i += SMP_THREADS) sum += (double) expf(l[i] - max_l);
    }
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
        uint32_t rk = lane < SMP_TOPK ? s_topk[lane] : 0u;
        int      ri = lane < SMP_TOPK ? s_topi[lane] : SMP_NONE;
        double   t = s_total;
        if (P > 1) {
            // the parts' lists, two places per lane (8 P are at most 64)
            const int p0 = lane / SMP_TOPK, p1 = p0 + 32 / SMP_TOPK, j = lane % SMP_TOPK;
            uint32_t a = 0, b = 0;
            int      ai = SMP_NONE, bi = SMP_NONE;
            if (p0 < P) { a = cl.map_shared_rank(s_topk, p0)[j]; ai = cl.map_shared_rank(s_topi, p0)[j]; }
            if (p1 < P) { b = cl.map_shared_rank(s_topk, p1)[j]; bi = cl.map_shared_rank(s_topi, p1)[j]; }
            const double mine = lane < P ? *cl.map_shared_rank(&s_total, lane) : 0.0;
            t = 0.0;
#pragma unroll
            for (int q = 0; q < SMP_PARTS; q++) t += __shfl_sync(0xffffffffu, mine, q);
            const bool swap = b > a || (b == a && bi < ai);
            smp_warp_top(swap ? b : a, swap ? bi : ai, swap ? a : b, swap ? ai : bi, lane, rk, ri, [](uint32_t, int, uint32_t &, int &) {});
        }
        if (lane < SMP_TOPK && !off) {
            const float x = ri == SMP_NONE ? -INFINITY : l[ri];
            out[blockIdx.x].id[lane]    = ri == SMP_NONE ? 0 : ri;
            out[blockIdx.x].logit[lane] = x;
            out[blockIdx.x].p[lane]     = (float) ((double) expf(x - max_l) / t);
        }
    }
    if (P > 1) cl.sync();                                         // the other blocks' lists have been read
}

int pib_sample_topk(float * logits_dev, int n_rows, int n_vocab, const int32_t * bias_ids_dev, const float * bias_val_dev,
                    int n_bias, void * out_dev, const uint8_t * desc, const int * cancel, cudaStream_t st) {
    (void) desc;
    // Parts while a thread has more than four elements and all blocks run at once: three per SM, less a sixteenth that packing clusters loses (us of 2 / 4 / 8 parts of 32 000
    // values: 48 rows 15.5 / 13.1 / 13.3, 56 15.5 / 15.5 / 22.7, 100 20.7 / 15.7 / 33.5, 148 22.9 / 27.5 / 45.2).  However many rows there are, long ones need several
    // blocks to have enough loads in flight (256 rows of 128 000, 1 / 2 / 4 parts: 203 / 115 / 100; of 65 000 57 / 52 / 56; of 32 000 32 / 35 / 40).
    int P = n_vocab > 96000 ? 4 : n_vocab > 48000 ? 2 : 1;
    while (P < SMP_PARTS && 16LL * n_rows * P * 2 <= 45LL * pib_num_sms() && n_vocab >= P * 8 * SMP_THREADS) P <<= 1;
    const int per = ((n_vocab + P - 1) / P + SMP_THREADS - 1) / SMP_THREADS;     // values per thread
#define SMP_GO(E) do {                                                                                                                                                                     \
        if (P > 1) PIB_CHECK(pib_launch_cluster(sample_topk_kernel<E>, dim3((unsigned) n_rows, (unsigned) P), dim3(SMP_THREADS), dim3(1, (unsigned) P, 1), 0, st, logits_dev, n_vocab,      \
                                                bias_ids_dev, bias_val_dev, n_bias, (pib_row_result *) out_dev, cancel));                                                                  \
        else       PIB_CHECK(pib_launch(sample_topk_kernel<E>, dim3((unsigned) n_rows), dim3(SMP_THREADS), 0, st, logits_dev, n_vocab, bias_ids_dev, bias_val_dev, n_bias,                 \
                                        (pib_row_result *) out_dev, cancel));                                                                                                              \
    } while (0)
    const bool few = (int64_t) n_rows * P <= 2 * pib_num_sms();
    if (few && per <= 16) SMP_GO(16); else if (few && per <= 32) SMP_GO(32); else SMP_GO(0);
#undef SMP_GO
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
