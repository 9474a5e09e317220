// flash_attn.cu -- attention of long portions over cached key / value heads (served mode) with scores and weights in tensor memory.
//
// One launch takes the portions of up to FA_SEGS segments (a sequence's consecutive tokens).  One block takes 128 query rows of one problem (key / value head, map) of one
// portion: rows are (token, head of the group), the `rep` heads that share the keys next to each other; the blocks with the most keys start first.
// It walks the key columns its tokens can see in tiles of 64 with one pass and running maxima:
//   warp 0       one lane brings the query rows once and every tile's keys and values by TMA (two stages each)
//   warp 1       an elected lane issues tcgen05.mma: scores S = Q K^T of a tile, then O += P V of the tile before the last
//   warps 2..9   two groups of 128 threads, one for the even and one for the odd tiles, a thread per query row: scores from tensor memory, cap, distance bias and
//                mask, running maximum, weights as two bfloat16 parts back into tensor memory (the first operand of the second product).  Each group has its own accumulator,
//                rescaled only when a maximum has grown by more than 2^FA_LAZY; both are merged on the way out
// Scores keep fp32 accuracy on bfloat16 operands: queries and keys enter as their bfloat16 part and the remainder of that rounding, three products are summed
// (hi.hi + lo.hi + hi.lo); weights enter as two parts against the bfloat16 values.  The sink is the running state's start (maximum = sink, denominator = 1).
// The result leaves in token order, divided by the denominator and (optionally) gated.
// Operands: fa_gather_kernel lays out, for every portion, key columns [kept first positions (n_front) | positions j0, j0 + 1, ... | zeros up to 64], values transposed, query rows;
// tiles nobody in the block sees are not visited.  Every wait is bounded (tc_common.cuh).
// What bounds it: the score products (24 MMAs of 64 keys a tile, 57 clocks each: a tile takes 2650 clocks), and with few tiles a block's start and end: code that runs once comes from far
// away, 9 clocks an instruction.  Three portions of 517, 504 and 491 tokens, 16 heads of 128 over 4: one launch 34 us with slopes, 48 with a bias table and a gate (a launch per
// portion, weights through shared memory, the table read from memory, a lane's own row written by it: 88 and 153).
#include <cuda_bf16.h>

#include <algorithm>

#include "tc_common.cuh"

#define FA_ROWS    128
#define FA_KEYS    64
#define FA_THREADS 320
#define FA_LAZY    8.0f
#define FA_LOG2E   1.4426950408889634f
#define FA_SEGS    32
#define FA_REL_LOW 192       // a row's distance to a column of a tile that its block visits: more than -(FA_ROWS + FA_KEYS)
#define FA_REL_TOP 128       // and less than this above the table's end where the tile is not wholly behind it
#define FA_REL_MAX (24 * 1024)

struct fa_args {
    int rep, maps, H, V, VN, Z, n_segs;              // heads per problem, maps per head, query rows per token, value size (rounded up to 16: VN), problems, portions
    int window, mask, keep, vec_out, rel_smem;       // vec_out: outputs and gates in pieces of 16 bytes; rel_smem: entries per head of the bias table's copy in shared memory (0: read from memory)
    float softcap;
    const float * sink, * slopes, * rel; int n_rel;
    const float * gate; int ldg;
    float * out; int out_bf16;                       // out_bf16: out holds bfloat16 rows
    int * err;
    pib_attn_block seg[FA_SEGS];                     // portions, those with the most row blocks first
};
__device__ __forceinline__ float fa_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ int fa_low(const fa_args & A, int p) { return A.mask == PIB_MASK_CHUNK ? p - p % A.window : max(0, p - A.window + 1); }

template <int NC> struct fa_cfg {                    // NC: 64-wide column chunks of a head (1 or 2)
    static constexpr int Q_TILE = FA_ROWS * 128, K_TILE = FA_KEYS * 128, V_TILE = 128 * 128;
    static constexpr int Q_BYTES = 2 * NC * Q_TILE, K_BYTES = 2 * NC * K_TILE, STAGE = K_BYTES + V_TILE;
    static constexpr size_t SMEM = (size_t) Q_BYTES + 2 * STAGE + 2 * FA_ROWS * 8 + 16 * 8 + 32 + 1024;    // behind the stages: the groups' maxima and denominators; then the bias table
};

// A in tensor memory, B in shared memory; called by a converged warp
__device__ __forceinline__ void fa_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

__device__ __forceinline__ void fa_st16(uint32_t taddr, const uint32_t * v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                   "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}

template <int NC>
__global__ void __launch_bounds__(FA_THREADS)
flash_attn_kernel(const __grid_constant__ CUtensorMap qh, const __grid_constant__ CUtensorMap ql, const __grid_constant__ CUtensorMap kh, const __grid_constant__ CUtensorMap kl,
                  const __grid_constant__ CUtensorMap vm, const __grid_constant__ fa_args A) {
    pib_pdl_wait();
    pib_pdl_trigger();
    using C = fa_cfg<NC>;
    extern __shared__ __align__(1024) uint8_t fa_dsm[];
    uint8_t *  sQ  = fa_dsm + ((1024u - (dt_smem(fa_dsm) & 1023u)) & 1023u);
    uint8_t *  sKV = sQ + C::Q_BYTES;
    float2 *   ml  = reinterpret_cast<float2 *>(sKV + 2 * C::STAGE);
    uint64_t * bar = reinterpret_cast<uint64_t *>(ml + 2 * FA_ROWS);
    uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(bar + 16);
    volatile int * abort_s = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *    srel = reinterpret_cast<float *>(tmem_slot + 8);
    // barriers: queries; keys arrived / read, values arrived / read (per stage); scores ready, weights written, product done (per group)
    const uint32_t b0 = dt_smem(bar), bar_q = b0, bar_k = b0 + 8, bar_kf = b0 + 24, bar_v = b0 + 40, bar_vf = b0 + 56, bar_s = b0 + 72, bar_p = b0 + 88, bar_o = b0 + 104;
    // the portion and row block: the last row blocks (the most keys) of all portions first; z the problem
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, z = blockIdx.x % A.Z;
    int at = blockIdx.x / A.Z, k_seg = 1;
    for (; k_seg < A.n_segs; k_seg++) {              // the first k_seg portions have row blocks of the numbers [blocks of the next one, blocks of the last of these)
        const int n = (A.seg[k_seg - 1].row_blocks - A.seg[k_seg].row_blocks) * k_seg;
        if (at < n) break;
        at -= n;
    }
    const pib_attn_block & G = A.seg[at % k_seg];
    const int row0 = (A.seg[k_seg - 1].row_blocks - 1 - at / k_seg) * FA_ROWS, n_rows = G.nq * A.rep, p0 = G.p0, j0 = G.j0, n_front = G.n_front;
    // the tiles this block's tokens see: [0, front) hold kept positions, [first, last] the window
    const int pa = p0 + row0 / A.rep, pb = p0 + min(n_rows - 1, row0 + FA_ROWS - 1) / A.rep;
    const int first = (n_front + fa_low(A, pa) - j0) / FA_KEYS, last = (n_front + pb - j0) / FA_KEYS;
    const int kept = n_front > 0 ? n_front : min(A.keep, pb + 1), front = (kept + FA_KEYS - 1) / FA_KEYS;
    const bool joined = front >= first;
    const int n_tiles = joined ? last + 1 : front + last - first + 1;
    auto tile_of = [&](int j) { return joined || j < front ? j : first + j - front; };

    if (threadIdx.x == 0) {
        dt_mbar_init(bar_q, 1);
        for (int k = 0; k < 2; k++) {
            for (uint32_t b : { bar_k, bar_kf, bar_v, bar_vf, bar_s, bar_o }) dt_mbar_init(b + 8 * k, 1);
            dt_mbar_init(bar_p + 8 * k, FA_ROWS);
        }
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dt_smem(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    dt_fence_before();
    __syncthreads();
    dt_fence_after();
    const uint32_t tmem = *tmem_slot, tm_p = tmem + 128, tm_o = tmem + 256;          // columns: scores 0..63 and 64..127, weights 128..191 and 192..255 (32 of each part), outputs 256..383 and 384..511

    if (warp == 0) {
        if (lane == 0) {
            dt_mbar_expect_tx(bar_q, C::Q_BYTES);
            for (int c = 0; c < NC; c++) {
                dt_tma_3d(dt_smem(sQ + c * C::Q_TILE), &qh, bar_q, c * 64, G.row0 + row0, z);
                dt_tma_3d(dt_smem(sQ + (NC + c) * C::Q_TILE), &ql, bar_q, c * 64, G.row0 + row0, z);
            }
            auto keys = [&](int j) {
                const int k = 8 * (j & 1), col = G.col0 + tile_of(j) * FA_KEYS;
                uint8_t * st = sKV + (j & 1) * C::STAGE;
                if (j >= 2 && !dt_mbar_wait(bar_kf + k, ((j >> 1) - 1) & 1, abort_s)) return false;
                dt_mbar_expect_tx(bar_k + k, C::K_BYTES);
                for (int c = 0; c < NC; c++) {
                    dt_tma_3d(dt_smem(st + c * C::K_TILE), &kh, bar_k + k, c * 64, col, z);
                    dt_tma_3d(dt_smem(st + (NC + c) * C::K_TILE), &kl, bar_k + k, c * 64, col, z);
                }
                return true;
            };
            bool ok = keys(0);
            for (int j = 0; j < n_tiles && ok; j++) {               // the keys run one tile ahead: their place is free as soon as the scores before are formed
                const int k = 8 * (j & 1);
                if (j + 1 < n_tiles && !(ok = keys(j + 1))) break;
                if (j >= 2 && !dt_mbar_wait(bar_vf + k, ((j >> 1) - 1) & 1, abort_s)) break;
                dt_mbar_expect_tx(bar_v + k, A.VN * 128);
                dt_tma_3d(dt_smem(sKV + (j & 1) * C::STAGE + C::K_BYTES), &vm, bar_v + k, G.col0 + tile_of(j) * FA_KEYS, 0, z);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t id_s = dt_idesc(FA_ROWS, FA_KEYS);
        const uint32_t id_o = dt_idesc(FA_ROWS, A.VN);
        const uint64_t dq = dt_desc(dt_smem(sQ));
        auto scores = [&](int j) {                             // S(j), once its keys are there: three products over the head's columns
            if (!__all_sync(0xffffffffu, dt_mbar_wait(bar_k + 8 * (j & 1), (j >> 1) & 1, abort_s))) return false;
            dt_fence_after();
            const uint64_t dk = dt_desc(dt_smem(sKV + (j & 1) * C::STAGE));
            bool acc = false;
#pragma unroll
            for (int part = 0; part < 3; part++) {
                const uint64_t a = dq + (part == 1 ? (uint64_t) (NC * C::Q_TILE >> 4) : 0), b = dk + (part == 2 ? (uint64_t) (NC * C::K_TILE >> 4) : 0);
#pragma unroll
                for (int c = 0; c < NC; c++)
#pragma unroll
                    for (int k = 0; k < 4; k++) { dt_mma(tmem + 64 * (j & 1), a + (c * C::Q_TILE >> 4) + 2 * k, b + (c * C::K_TILE >> 4) + 2 * k, id_s, acc); acc = true; }
            }
            dt_commit(bar_s + 8 * (j & 1));
            dt_commit(bar_kf + 8 * (j & 1));
            return true;
        };
        bool ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_q, 0, abort_s)) && scores(0) && (n_tiles < 2 || scores(1));
        for (int j = 0; j < n_tiles && ok; j++) {
            ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_p + 8 * (j & 1), (j >> 1) & 1, abort_s));       // the group has read its scores, too: their columns are free
            if (!ok) break;
            if (j + 2 < n_tiles && !(ok = scores(j + 2))) break;
            ok = __all_sync(0xffffffffu, dt_mbar_wait(bar_v + 8 * (j & 1), (j >> 1) & 1, abort_s));
            if (!ok) break;
            dt_fence_after();
            const uint64_t dv = dt_desc(dt_smem(sKV + (j & 1) * C::STAGE + C::K_BYTES));
            const uint32_t tp = tm_p + 64 * (j & 1);
#pragma unroll
            for (int part = 0; part < 2; part++)                   // the weights' parts
#pragma unroll
                for (int k = 0; k < 4; k++) fa_mma_ts(tm_o + 128 * (j & 1), tp + 32 * part + 8 * k, dv + 2 * k, id_o, (j > 1) | ((part | k) != 0));
            dt_commit(bar_o + 8 * (j & 1));
            dt_commit(bar_vf + 8 * (j & 1));
        }
    } else {
        const int w = (warp - 2) >> 2, q4 = warp & 3, rt = q4 * 32 + lane, R = row0 + rt, Rc = min(R, n_rows - 1);
        const int p = p0 + Rc / A.rep, h = (z / A.maps * A.rep + Rc % A.rep) * A.maps + z % A.maps;
        const int pmin = p0 + min(n_rows - 1, row0 + q4 * 32) / A.rep, pmax = p0 + min(n_rows - 1, row0 + q4 * 32 + 31) / A.rep;      // of this warp's rows
        const uint32_t lane_off = (uint32_t) (q4 * 32) << 16;
        const float slope2 = A.slopes ? A.slopes[h] * FA_LOG2E : 0.f;
        const float * rel = A.rel ? A.rel + (size_t) h * A.n_rel : nullptr;
        const float * rels = srel + (Rc % A.rep) * A.rel_smem + FA_REL_LOW;              // the same in units of log2, continued at both ends
        if (A.rel_smem) {
            for (int hr = 0; hr < A.rep; hr++) {
                const float * src = A.rel + (size_t) ((z / A.maps * A.rep + hr) * A.maps + z % A.maps) * A.n_rel;
#pragma unroll 4
                for (int i = threadIdx.x - 64; i < A.n_rel + FA_REL_LOW + FA_REL_TOP; i += 256) srel[hr * A.rel_smem + i] = src[min(max(i - FA_REL_LOW, 0), A.n_rel - 1)] * FA_LOG2E;
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        const bool sunk = A.sink && w == 0;                                                                                              // the sink counts once
        float m = sunk ? A.sink[h] * FA_LOG2E : -INFINITY, l = sunk ? 1.f : 0.f;                                                         // maximum in units of log2
        const uint32_t tm_s = tmem + lane_off + 64 * w, tm_w = tm_o + lane_off + 128 * w;
        const uint32_t tm_pw = tm_p + lane_off + 64 * w;
        bool ok = true;
        for (int j = w; j < n_tiles; j += 2) {
            const int c0 = tile_of(j) * FA_KEYS, xb = j0 + c0 - n_front;       // column c0 + i holds position xb + i (i when it is a kept column in front)
            ok = dt_mbar_wait(bar_s + 8 * w, (j >> 1) & 1, abort_s);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            dt_fence_after();
            float t[FA_KEYS];
            dt_ld32(tm_s, reinterpret_cast<uint32_t *>(t));
            dt_ld32(tm_s + 32, reinterpret_cast<uint32_t *>(t) + 32);
            dt_wait_ld();
            if (A.softcap > 0.f) {
                const float ic = 1.0f / A.softcap;
#pragma unroll
                for (int i = 0; i < FA_KEYS; i++) t[i] = A.softcap * FA_LOG2E * tanhf(t[i] * ic);
            }                                                        // without a cap the queries carry the factor log2 e
            if (c0 >= n_front) {                                   // no kept column in this tile
                const int d0 = p - xb;
                if (A.slopes) {
                    const float f0 = (float) d0;
#pragma unroll
                    for (int i = 0; i < FA_KEYS; i++) t[i] = fmaf(-slope2, f0 - (float) i, t[i]);
                }
                if (rel) {
                    if (pmin - xb - (FA_KEYS - 1) >= A.n_rel - 1) {  // the whole tile lies where the table has come to its end
                        const float e = rel[A.n_rel - 1];
#pragma unroll
                        for (int i = 0; i < FA_KEYS; i++) t[i] = fmaf(e, FA_LOG2E, t[i]);
                    } else if (A.rel_smem) {
                        const float * e = rels + d0;
#pragma unroll
                        for (int i = 0; i < FA_KEYS; i++) t[i] += e[-i];
                    } else {
#pragma unroll
                        for (int i = 0; i < FA_KEYS; i++) t[i] = fmaf(rel[min(max(d0 - i, 0), A.n_rel - 1)], FA_LOG2E, t[i]);
                    }
                }
                const bool all_seen = xb + FA_KEYS - 1 <= pmin && xb >= fa_low(A, pmax);
                if (!all_seen) {
                    const int lo = fa_low(A, p) - xb;                // columns lo .. d0, and those of kept positions
                    const int ka = A.keep - xb;
#pragma unroll
                    for (int i = 0; i < FA_KEYS; i++) t[i] = i <= d0 && (i >= lo || i < ka) ? t[i] : -INFINITY;
                }
            } else {
                const int lo = fa_low(A, p);
#pragma unroll
                for (int i = 0; i < FA_KEYS; i++) {
                    const int x = c0 + i < n_front ? c0 + i : xb + i, d = p - x;
                    if (A.slopes) t[i] = fmaf(-slope2, (float) d, t[i]);
                    if (rel) t[i] = fmaf(rel[min(max(d, 0), A.n_rel - 1)], FA_LOG2E, t[i]);
                    t[i] = d >= 0 && (x >= lo || x < A.keep) ? t[i] : -INFINITY;
                }
            }
            float mt = t[0];
#pragma unroll
            for (int i = 1; i < FA_KEYS; i++) mt = fmaxf(mt, t[i]);
            const bool grow = mt > m + FA_LAZY;                      // also the first key of a row without a sink (m -inf)
            const bool rescale = __any_sync(0xffffffffu, grow);
            float f = 1.f;
            if (grow) { f = fa_exp2(m - mt); m = mt; l *= f; }
            const float ms = m == -INFINITY ? 0.f : m;
            if (j > 1) {                                             // the group's product before has read its weights and left the accumulator
                ok = dt_mbar_wait(bar_o + 8 * w, ((j >> 1) - 1) & 1, abort_s);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                dt_fence_after();                                    // also without a rescale: the weights' stores below come behind that product's reads of them
                if (rescale) {
                    for (int c = 0; c < A.VN; c += 32) {
                        uint32_t v[32];
                        dt_ld32(tm_w + c, v);
                        dt_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
                        dt_st32(tm_w + c, v);
                    }
                    dt_wait_st();
                }
            }
            float l2 = 0.f;
#pragma unroll
            for (int c = 0; c < 2; c++) {                            // 32 columns: a word holds two neighbouring ones
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float a = fa_exp2(t[32 * c + 2 * i] - ms), b = fa_exp2(t[32 * c + 2 * i + 1] - ms);
                    l += a; l2 += b;
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
                    hi[i] = *reinterpret_cast<const uint32_t *>(&h2);
                    const __nv_bfloat162 r2 = __floats2bfloat162_rn(a - __uint_as_float(hi[i] << 16), b - __uint_as_float(hi[i] & 0xffff0000u));
                    lo[i] = *reinterpret_cast<const uint32_t *>(&r2);
                }
                fa_st16(tm_pw + 16 * c, hi);
                fa_st16(tm_pw + 32 + 16 * c, lo);
            }
            l += l2;
            dt_wait_st();
            dt_fence_before();
            dt_arrive(bar_p + 8 * w);
        }
        // both groups' products are done; maxima and denominators cross through shared memory (the weights' place), then each group writes half of the columns
        const int mine = (n_tiles - 1 - w) >> 1;                     // index of the group's last tile among its own (none: -1)
        if (ok && n_tiles > w) ok = dt_mbar_wait(bar_o + 8 * w, mine & 1, abort_s);
        ok = __all_sync(0xffffffffu, ok);
        ml[w * FA_ROWS + rt] = make_float2(m, l);
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (__all_sync(0xffffffffu, ok && !*abort_s)) {
            dt_fence_after();
            const float2 o = ml[(1 - w) * FA_ROWS + rt];
            const float  M = fmaxf(m, o.x), fm = m == -INFINITY ? 0.f : fa_exp2(m - M), fo = o.x == -INFINITY ? 0.f : fa_exp2(o.x - M), inv = 1.0f / (l * fm + o.y * fo);
            const float  f0 = (w == 0 ? fm : fo) * inv, f1 = (w == 0 ? fo : fm) * inv;
            // a chunk of 32 columns turns through shared memory (the operands' place: every product is done), so that a row's values leave and its gate's arrive in one piece (a
            // lane per row took 20 us of a gated block's time)
            static_assert(8 * 2 * 32 * 36 * 4 <= C::Q_BYTES + 2 * C::STAGE, "chunks of values and gates of eight warps");
            float * buf = reinterpret_cast<float *>(sQ) + (warp - 2) * 2 * 32 * 36, * gbuf = buf + 32 * 36;
            const uint32_t gate_at = (uint32_t) (((size_t) (G.t0 + Rc / A.rep) * A.ldg + (size_t) h * A.V) / 4);
            const int row = (int) ((size_t) (G.t0 + Rc / A.rep) * A.H + h), rows = min(32, n_rows - row0 - q4 * 32);
#pragma unroll 1
            for (int c = 32 * w; c < A.VN; c += 64) {
                float v[32];
                dt_ld32(tm_o + lane_off + c, reinterpret_cast<uint32_t *>(v));
                dt_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] *= f0;
                if (n_tiles > 1) {
                    float u[32];
                    dt_ld32(tm_o + lane_off + 128 + c, reinterpret_cast<uint32_t *>(u));
                    dt_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] = fmaf(u[i], f1, v[i]);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4 *>(buf + lane * 36 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                __syncwarp();
                if (A.vec_out) {                                     // four rows at a time, eight lanes a row
                    const int cl = c + (lane & 7) * 4;
                    const bool col = cl < A.V;
                    if (A.gate) {
                        float4 g4[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const int r = 4 * k + (lane >> 3);
                            const uint32_t g_r = __shfl_sync(0xffffffffu, gate_at, r);
                            if (r < rows && col) g4[k] = *reinterpret_cast<const float4 *>(A.gate + (size_t) g_r * 4 + cl);
                        }
#pragma unroll
                        for (int k = 0; k < 8; k++) *reinterpret_cast<float4 *>(gbuf + (4 * k + (lane >> 3)) * 36 + (lane & 7) * 4) = g4[k];      // read back by the lane that wrote it
                    }
#pragma unroll 1                                                     // short code: instructions that a block runs once come from far away, 9 clocks each
                    for (int k = 0; k < 8; k++) {
                        const int r = 4 * k + (lane >> 3), rr = __shfl_sync(0xffffffffu, row, r);
                        float4 x = *reinterpret_cast<const float4 *>(buf + r * 36 + (lane & 7) * 4);
                        if (A.gate) {
                            const float4 g = *reinterpret_cast<const float4 *>(gbuf + r * 36 + (lane & 7) * 4);
                            x.x *= 1.0f / (1.0f + __expf(-g.x)); x.y *= 1.0f / (1.0f + __expf(-g.y)); x.z *= 1.0f / (1.0f + __expf(-g.z)); x.w *= 1.0f / (1.0f + __expf(-g.w));
                        }
                        if (r >= rows || !col) continue;
                        if (A.out_bf16) {
                            const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
                            *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(A.out) + (size_t) rr * A.V + cl) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
                        } else *reinterpret_cast<float4 *>(A.out + (size_t) rr * A.V + cl) = x;
                    }
                } else {
                    for (int r = 0; r < rows; r++) {
                        const int rr = __shfl_sync(0xffffffffu, row, r);
                        if (c + lane >= A.V) continue;
                        float x = buf[r * 36 + lane];
                        if (A.gate) x *= 1.0f / (1.0f + __expf(-A.gate[(size_t) (rr / A.H) * A.ldg + (size_t) (rr % A.H) * A.V + c + lane]));
                        if (A.out_bf16) reinterpret_cast<__nv_bfloat16 *>(A.out)[(size_t) rr * A.V + c + lane] = __float2bfloat16_rn(x);
                        else A.out[(size_t) rr * A.V + c + lane] = x;
                    }
                }
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
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

bool pib_flash_attention_fits(const pib_hlayer & L) {
    static const int on = getenv("PIB_FLASH_ATTN") ? atoi(getenv("PIB_FLASH_ATTN")) : 1;
    return on != 0 && L.dim % 8 == 0 && L.dim >= 8 && L.dim <= 128 && L.vdim >= 1 && L.vdim <= 128 && !(L.maps > 1 && L.sink);
}

// ---- operands ---------------------------------------------------------------------------------------------------------------------
// keys Kb [GK][C][2 D] = [hi | lo], values Vt [GK][V][C], queries Qc [GK][R][2 D], bfloat16; C columns and R rows of all portions (pib_attn_block: col0, row0)
struct fa_gather_args {
    const float * cache; int cache_row; const int32_t * cellmap; int n_ctx;
    const float * q; int ldq, vec_k, vec_q;                      // vec: four floats at a time
    int GK, maps, rep, D, V, C, R, n_segs; float scale;
    __nv_bfloat16 * Kb, * Vt, * Qc;
    pib_attn_block seg[FA_SEGS];
};
// a warp: [hi | lo] of four rows at once (src null: zeros; dst null: none); heads of up to 128 coordinates, four or one a lane and trip
__device__ __forceinline__ void fa_split_rows(const float * const (&src)[4], __nv_bfloat16 * const (&dst)[4], int D, int vec, float scale, int lane) {
    if (vec) {
        const int i = lane * 4;
        if (i >= D) return;
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = src[k] ? *reinterpret_cast<const float4 *>(src[k] + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!dst[k]) continue;
            v[k].x *= scale; v[k].y *= scale; v[k].z *= scale; v[k].w *= scale;
            const __nv_bfloat162 a = __floats2bfloat162_rn(v[k].x, v[k].y), b = __floats2bfloat162_rn(v[k].z, v[k].w);
            const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
            const __nv_bfloat162 c = __floats2bfloat162_rn(v[k].x - fa.x, v[k].y - fa.y), d = __floats2bfloat162_rn(v[k].z - fb.x, v[k].w - fb.y);
            *reinterpret_cast<uint2 *>(dst[k] + i)     = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
            *reinterpret_cast<uint2 *>(dst[k] + D + i) = make_uint2(*reinterpret_cast<const uint32_t *>(&c), *reinterpret_cast<const uint32_t *>(&d));
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            if (!dst[k]) continue;
            for (int i = lane; i < D; i += 32) {
                const float v = src[k] ? src[k][i] * scale : 0.f;
                const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                dst[k][i] = hi; dst[k][D + i] = __float2bfloat16_rn(v - __bfloat162float(hi));
            }
        }
    }
}
// grid (64 columns or 32 query rows, problem, 2 + slices of 32 value coordinates): queries, keys, values (through shared memory to come out transposed)
__global__ void __launch_bounds__(256) fa_gather_kernel(const __grid_constant__ fa_gather_args A) {
    pib_pdl_wait();
    pib_pdl_trigger();
    __shared__ float tile[64][33];
    const int z = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, what = blockIdx.z;
    const float * src[4];
    __nv_bfloat16 * dst[4];
    int s = 0;
    if (what == 0) {
        const int r0 = blockIdx.x * 32;
        if (r0 >= A.R) return;
        while (s + 1 < A.n_segs && r0 >= A.seg[s].row0 + A.seg[s].row_blocks * FA_ROWS) s++;
        const pib_attn_block & G = A.seg[s];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int i = warp * 4 + k, r = r0 + i - G.row0, h = (z / A.maps * A.rep + r % A.rep) * A.maps + z % A.maps;
            const bool live = r < G.nq * A.rep;                  // rows without a token are read and dropped by the attention
            src[k] = live ? A.q + (size_t) (G.t0 + r / A.rep) * A.ldq + (size_t) h * A.D : nullptr;
            dst[k] = live ? A.Qc + ((size_t) z * A.R + r0 + i) * 2 * A.D : nullptr;
        }
        fa_split_rows(src, dst, A.D, A.vec_q, A.scale, lane);
        return;
    }
    const int c0 = blockIdx.x * 64;
    if (c0 >= A.C) return;
    while (s + 1 < A.n_segs && c0 >= A.seg[s].col0 + A.seg[s].cols) s++;
    const pib_attn_block & G = A.seg[s];
    const int32_t * map = A.cellmap + (size_t) G.slot * A.n_ctx;
    const float * rows[8];                                       // this warp's columns warp, warp + 8, ...
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = c0 - G.col0 + warp + 8 * i;
        rows[i] = j < G.NK ? A.cache + (size_t) map[j < G.n_front ? j : G.j0 + j - G.n_front] * A.cache_row : nullptr;
    }
    if (what == 1) {
#pragma unroll
        for (int t = 0; t < 2; t++) {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                src[k] = rows[4 * t + k] ? rows[4 * t + k] + (size_t) z * A.D : nullptr;
                dst[k] = A.Kb + ((size_t) z * A.C + c0 + warp + 8 * (4 * t + k)) * 2 * A.D;
            }
            fa_split_rows(src, dst, A.D, A.vec_k, 1.f, lane);
        }
        return;
    }
    const size_t vo = (size_t) A.GK * A.D + (size_t) (z / A.maps) * A.V;
    const int v0 = (what - 2) * 32;
#pragma unroll
    for (int i = 0; i < 8; i++) tile[warp + 8 * i][lane] = rows[i] && v0 + lane < A.V ? rows[i][vo + v0 + lane] : 0.f;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = warp + 8 * i;
        if (v0 + c < A.V) *reinterpret_cast<__nv_bfloat162 *>(A.Vt + ((size_t) z * A.V + v0 + c) * A.C + c0 + 2 * lane) = __floats2bfloat162_rn(tile[2 * lane][c], tile[2 * lane + 1][c]);
    }
}

size_t pib_flash_attention_bytes(const pib_hlayer & L, long long cols, long long rows, size_t * k_bytes, size_t * v_bytes) {
    const size_t GK = (size_t) L.kv_heads * L.maps;
    *k_bytes = GK * cols * 2 * L.dim * 2;
    *v_bytes = GK * L.vdim * cols * 2;
    return GK * rows * 2 * L.dim * 2;
}
void pib_flash_attention_place(std::vector<pib_attn_block> & blocks, int rep, long long * cols, long long * rows) {
    std::stable_sort(blocks.begin(), blocks.end(), [](const pib_attn_block & a, const pib_attn_block & b) { return a.nq > b.nq; });
    long long c = 0, r = 0;
    for (pib_attn_block & g : blocks) {
        g.cols = (g.NK + FA_KEYS - 1) / FA_KEYS * FA_KEYS; g.row_blocks = (g.nq * rep + FA_ROWS - 1) / FA_ROWS;
        g.col0 = (int) c; g.row0 = (int) r;
        c += g.cols; r += (long long) g.row_blocks * FA_ROWS;
    }
    *cols = c; *rows = r;
}
int pib_flash_attention_max() { return FA_SEGS; }

int pib_flash_attention(const pib_kv_query & q, const pib_hlayer & L, const std::vector<pib_attn_block> & blocks, int C, int R, const float * cache, int cache_row, const int32_t * cellmap, int n_ctx,
                        void * Kb, void * Vt, void * Qc, float * out, cudaStream_t st, bool out_bf16) {
    const int D = L.dim, V = L.vdim, maps = L.maps, rep = L.heads / L.kv_heads, Z = L.kv_heads * maps, n = (int) blocks.size();
    if (n < 1 || n > FA_SEGS) { pib_set_error("attention: %d portions in a launch", n); return PIB_ERR_ARG; }
    fa_gather_args g = { cache, cache_row, cellmap, n_ctx, q.q, q.ldq, cache_row % 4 == 0 && ((uintptr_t) cache & 15) == 0, q.ldq % 4 == 0 && ((uintptr_t) q.q & 15) == 0,
                         Z, maps, rep, D, V, C, R, n, L.softcap > 0.f ? L.scale : L.scale * FA_LOG2E, (__nv_bfloat16 *) Kb, (__nv_bfloat16 *) Vt, (__nv_bfloat16 *) Qc, {} };
    std::copy(blocks.begin(), blocks.end(), g.seg);
    pib_launch(fa_gather_kernel, dim3((unsigned) std::max(C / 64, R / 32), (unsigned) Z, (unsigned) (2 + (V + 31) / 32)), dim3(256), (size_t) 0, st, g);
    PIB_CHECK(cudaGetLastError());
    const __nv_bfloat16 * kb = (const __nv_bfloat16 *) Kb, * qc = (const __nv_bfloat16 *) Qc, * vt = (const __nv_bfloat16 *) Vt;
    CUtensorMap qh, ql, kh, kl, vm;
    const int VN = (V + 15) & ~15;
    int rc = pib_tma_map3(&qh, qc, D, R, Z, 4 * (uint64_t) D, 4 * (uint64_t) D * R, FA_ROWS);
    if (rc == PIB_OK) rc = pib_tma_map3(&ql, qc + D, D, R, Z, 4 * (uint64_t) D, 4 * (uint64_t) D * R, FA_ROWS);
    if (rc == PIB_OK) rc = pib_tma_map3(&kh, kb, D, C, Z, 4 * (uint64_t) D, 4 * (uint64_t) D * C, FA_KEYS);
    if (rc == PIB_OK) rc = pib_tma_map3(&kl, kb + D, D, C, Z, 4 * (uint64_t) D, 4 * (uint64_t) D * C, FA_KEYS);
    if (rc == PIB_OK) rc = pib_tma_map3(&vm, vt, C, V, Z, 2 * (uint64_t) C, 2 * (uint64_t) C * V, (uint32_t) VN);
    if (rc != PIB_OK) return rc;
    int * err = pib_tc_error_word(st);
    if (!err) { pib_set_error("attention: no error word"); return PIB_ERR_NOMEM; }
    // entries per head, the heads 8 banks apart
    const int entries = L.rel ? (L.n_rel + FA_REL_LOW + FA_REL_TOP + 31) / 32 * 32 + 8 : 0, rel_smem = (size_t) entries * rep * 4 <= FA_REL_MAX ? entries : 0;
    int t_end = 0;
    for (const pib_attn_block & b : blocks) t_end = std::max(t_end, b.t0 + b.nq);
    const int vec_out = V % 4 == 0 && ((uintptr_t) out & 15) == 0 && (!q.gate || (q.ldg % 4 == 0 && ((uintptr_t) q.gate & 15) == 0 && (size_t) q.ldg * ((size_t) t_end + 1) / 4 < (1ull << 32)));
    fa_args A = { rep, maps, L.heads * maps, V, VN, Z, n, L.window, L.mask, L.keep, vec_out, rel_smem, L.softcap, L.sink, L.slopes, L.rel, L.n_rel, q.gate, q.ldg, out, out_bf16 ? 1 : 0, err, {} };
    std::copy(blocks.begin(), blocks.end(), A.seg);
    int row_blocks = 0;
    for (const pib_attn_block & b : blocks) row_blocks += b.row_blocks;
    const size_t extra = (size_t) rel_smem * rep * 4;
#define FA_GO(NC) do {                                                                                                                             \
        static pib_per_device attrs;                                                                                                                \
        PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(flash_attn_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) (fa_cfg<NC>::SMEM + FA_REL_MAX)); })); \
        pib_launch(flash_attn_kernel<NC>, dim3((unsigned) (row_blocks * Z)), dim3(FA_THREADS), fa_cfg<NC>::SMEM + extra, st, qh, ql, kh, kl, vm, A); \
    } while (0)
    if (D <= 64) FA_GO(1); else FA_GO(2);
#undef FA_GO
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}
