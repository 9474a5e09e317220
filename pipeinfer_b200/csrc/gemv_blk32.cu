// gemv_blk32.cu -- tensor-core dequant-GEMV for the 32-element block formats (Q4_0, Q8_0) at verification batch 1..16.
//
// Same arithmetic as the reference (ggml_vec_dot_q4_0_q8_0 ggml-quants.c:2426, q8_0_q8_0 :3521): per 32-element block an
// exact integer dot product of (q - 8) resp. q with the int8 activations, scaled by fp16(d_w) * d_x in fp32 and summed
// over the blocks.  Only the order of the fp32 block terms differs (per-warp partial sums, then a fixed-order reduction).
//
// Layout.  Eight consecutive blocks (256 columns) of a 16-row tile form one record, in mma.m16n8k32 A-fragment order so
// that a lane's 128-bit loads ARE its tensor-core operands:
//   Q4_0  2304 B: [pair p = 0..3][lane][16 B] = { row g blk 2p, row g+8 blk 2p, row g blk 2p+1, row g+8 blk 2p+1 } -- of each
//                 block the 4 bytes 4t..4t+3, whose low nibbles are columns 4t..4t+3 and high nibbles columns 16+4t..16+4t+3 --
//                 then [row 0..15][8 x fp16 d].
//   Q8_0  4352 B: [blk j = 0..7][lane][16 B] = { row g k 4t.., row g+8 k 4t.., row g k 16+4t.., row g+8 k 16+4t.. }, then the
//                 same 256 B of scales.
// K is padded to a multiple of 256 with zero blocks (d = 0), e.g. Falcon-7B's 4544 columns.  The activations come in a
// matching fragment order (act_quant.cu: qsp / dxp planes), zero-padded the same way.
#include <map>
#include <mutex>
#include <utility>

#include <math.h>

#include "pib_common.cuh"

#define BK_WARPS   4
#define BK_THREADS (BK_WARPS * 32)

__host__ __device__ static inline int bk_rec_bytes(int type) { return type == PIB_TYPE_Q4_0 ? 2304 : 4352; }

// ---- repack: planes -> records ------------------------------------------------------------------------------------------
__global__ void blk32_tiles_kernel(int type, const uint8_t * __restrict__ qs, const uint16_t * __restrict__ d, int64_t N, int64_t K,
                                   uint8_t * __restrict__ tiles) {
    const int64_t nb = K / 32, ngr = (K + 255) / 256, n_tiles = (N + 15) / 16;
    const int     rec = bk_rec_bytes(type), per = rec / 16, nq = per - 16;          // 16-byte pieces: quants, then 16 scale rows
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_tiles * ngr * per) return;
    const int64_t ts = i / per;
    const int     p  = (int) (i % per);
    const int64_t T = ts / ngr, G = ts % ngr;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (p < nq) {
        const int     lane = p % 32, g = lane / 4, t = lane % 4;
        const int64_t r0 = T * 16 + g, r1 = r0 + 8;
        if (type == PIB_TYPE_Q4_0) {
            const int     pr = p / 32;                                               // block pair
            const int64_t b0 = G * 8 + 2 * pr, b1 = b0 + 1;
            auto word = [&](int64_t r, int64_t b) -> uint32_t {
                return (r < N && b < nb) ? *reinterpret_cast<const uint32_t *>(qs + r * (K / 2) + b * 16 + t * 4) : 0x88888888u;   // (8 - 8) = 0
            };
            v = make_uint4(word(r0, b0), word(r1, b0), word(r0, b1), word(r1, b1));
        } else {
            const int     j = p / 32;
            const int64_t b = G * 8 + j;
            auto word = [&](int64_t r, int off) -> uint32_t {
                return (r < N && b < nb) ? *reinterpret_cast<const uint32_t *>(qs + r * K + b * 32 + off + t * 4) : 0u;
            };
            v = make_uint4(word(r0, 0), word(r1, 0), word(r0, 16), word(r1, 16));
        }
    } else {
        const int64_t r = T * 16 + (p - nq);
        uint16_t h[8];
        for (int j = 0; j < 8; j++) { const int64_t b = G * 8 + j; h[j] = (r < N && b < nb) ? d[r * nb + b] : (uint16_t) 0; }
        v = make_uint4(h[0] | ((uint32_t) h[1] << 16), h[2] | ((uint32_t) h[3] << 16), h[4] | ((uint32_t) h[5] << 16), h[6] | ((uint32_t) h[7] << 16));
    }
    *reinterpret_cast<uint4 *>(tiles + i * 16) = v;
}

int pib_weight_build_tiles_blk32(pib_weight * w) {
    if ((w->type != PIB_TYPE_Q4_0 && w->type != PIB_TYPE_Q8_0) || w->tiles) return PIB_OK;
    const int64_t ngr = (w->K + 255) / 256, n_tiles = (w->N + 15) / 16;
    const size_t  bytes = (size_t) n_tiles * ngr * bk_rec_bytes(w->type);
    if (cudaMalloc(&w->tiles, bytes) != cudaSuccess) {
        cudaGetLastError();
        pib_set_error("gemv tiles: cudaMalloc of %zu bytes failed", bytes);
        w->tiles = nullptr;
        return PIB_ERR_NOMEM;
    }
    w->tile_bytes = bytes;
    const int64_t n = (int64_t) (bytes / 16);
    blk32_tiles_kernel<<<(unsigned) ((n + 255) / 256), 256>>>(w->type, w->qs, w->d, w->N, w->K, w->tiles);
    PIB_CHECK(cudaGetLastError());
    return PIB_OK;
}

// ---- kernel -------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bk_mma_s8(int (&c)[4], int a0, int a1, int a2, int a3, int b0, int b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four nibbles 0..15 in the low half of each byte -> four int8 (q - 8): the forced high bit keeps the per-byte subtraction from
// borrowing across bytes, the final xor turns 0x78..0x87 into two's complement -8..7
__device__ __forceinline__ int bk_sub8(uint32_t nib) { return (int) (((nib | 0x80808080u) - 0x08080808u) ^ 0x80808080u); }

// grid (row tiles, k splits), BK_WARPS warps: warp w takes records sb0 + w, sb0 + w + BK_WARPS, ... of the CTA's k range;
// NT = token groups of 8 (1: b <= 8, 2: b <= 16).  The next record is prefetched into registers while the current one is
// multiplied; partial sums of the warps are reduced through shared memory in warp order; with k splits the last CTA to
// arrive adds the splits' partial sums in split order (deterministic), exactly as gemv_q4k_direct_kernel does.
// ONE: one token, whose pieces lie at distances known beforehand (Q4_0 57344 x 8192 52.9 / 50.9 us, 32000 x 4096 18.0 / 17.6; Q8_0 goes without: 32000 x 2048 11.8 / 13.7).
template <int WT, int NT, bool ONE>
__global__ void __launch_bounds__(BK_THREADS, NT == 1 ? 4 : 3)
gemv_blk32_kernel(const uint8_t * __restrict__ tiles, int ngr, int N, const int8_t * __restrict__ aqs, const __half * __restrict__ adx,
                  int b, float * __restrict__ y, float * __restrict__ partial, unsigned int * __restrict__ counters,
                  const int * __restrict__ cancel) {
    if (PIB_CANCELLED(cancel)) {
        pib_pdl_wait();
        // cancelled: no math, but the arrival protocol of the k split still runs -- the flag can flip while the grid is starting,
        // and a tile whose splits did not all arrive would leave its counter non-zero for the next launch
        if (gridDim.y > 1 && threadIdx.x == 0 && atomicAdd(&counters[blockIdx.x], 1u) == gridDim.y - 1) counters[blockIdx.x] = 0;
        return;
    }
    constexpr int REC = WT == PIB_TYPE_Q4_0 ? 2304 : 4352;
    constexpr int NQ  = WT == PIB_TYPE_Q4_0 ? 4 : 8;            // 128-bit quant loads per lane and record
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int T = blockIdx.x;
    const int nsplit = gridDim.y, split = blockIdx.y;
    const int per = (ngr + nsplit - 1) / nsplit;
    const int s0 = split * per, s1 = min(ngr, s0 + per);
    const uint8_t * qbase = tiles + (size_t) T * ngr * REC + lane * 16;
    const uint8_t * dbase = tiles + (size_t) T * ngr * REC + (REC - 256) + g * 16;

    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) { acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f; }
    const int8_t * a_q[NT];
    const __half * a_d[NT][2];
    int            gs[NT];                                      // tokens of the octet (pib_oct)
#pragma unroll
    for (int n = 0; n < NT; n++) {
        gs[n] = ONE ? 1 : min(8, b - 8 * n);
        a_q[n] = aqs + (size_t) n * 8 * ngr * 256 + min(g, gs[n] - 1) * 64 + t * 16;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            a_d[n][e] = adx + ((size_t) n * 8 * ngr + min(2 * t + e, gs[n] - 1)) * 8;
            // Two addresses of which nothing more is known: formed from one another, as neighbours allow, they cost up to 2.4 us a launch (at 2 tokens Q8_0 32000 x 2048 14.2 / 11.8,
            // 32000 x 1536 12.1 / 9.9, Q4_0 57344 x 8192 54.3 / 52.9; found by trying, instructions and bytes are the same)
            asm("" : "+l"(a_d[n][e]));
        }
    }

    int4 wq[NQ], dq[2];
    int  s = s0 + warp;
    if (s < s1) {
#pragma unroll
        for (int c = 0; c < NQ; c++) wq[c] = ld_stream_v4(qbase + (size_t) s * REC + c * 512);
        dq[0] = ld_stream_v4(dbase + (size_t) s * REC);
        dq[1] = ld_stream_v4(dbase + (size_t) s * REC + 128);
    }
    // the weights above are immutable, so their loads were issued before waiting for the kernel that produces the activations
    pib_pdl_wait();
    pib_pdl_trigger();
    for (; s < s1; s += BK_WARPS) {
        int4 wn[NQ], dn[2];
        const int sn = s + BK_WARPS;
        if (sn < s1) {
#pragma unroll
            for (int c = 0; c < NQ; c++) wn[c] = ld_stream_v4(qbase + (size_t) sn * REC + c * 512);
            dn[0] = ld_stream_v4(dbase + (size_t) sn * REC);
            dn[1] = ld_stream_v4(dbase + (size_t) sn * REC + 128);
        }
        int4 aq[NT][4];
        int4 ax[NT][2];
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const int sg = s * gs[n];
            const int4 * ap = reinterpret_cast<const int4 *>(a_q[n] + (size_t) sg * 256);
#pragma unroll
            for (int c = 0; c < 4; c++) aq[n][c] = __ldg(ap + c * 4 * gs[n]);
#pragma unroll
            for (int e = 0; e < 2; e++) ax[n][e] = __ldg(reinterpret_cast<const int4 *>(a_d[n][e] + (size_t) sg * 8));
        }
        const uint32_t dw0[4] = { (uint32_t) dq[0].x, (uint32_t) dq[0].y, (uint32_t) dq[0].z, (uint32_t) dq[0].w };   // row g:   d of blocks 2i | 2i+1
        const uint32_t dw1[4] = { (uint32_t) dq[1].x, (uint32_t) dq[1].y, (uint32_t) dq[1].z, (uint32_t) dq[1].w };   // row g+8
#pragma unroll
        for (int j = 0; j < 8; j++) {
            int a0, a1, a2, a3;
            if (WT == PIB_TYPE_Q4_0) {
                const int4     w  = wq[j >> 1];
                const uint32_t w0 = (uint32_t) ((j & 1) ? w.z : w.x), w1 = (uint32_t) ((j & 1) ? w.w : w.y);
                a0 = bk_sub8(w0 & 0x0F0F0F0Fu); a2 = bk_sub8((w0 >> 4) & 0x0F0F0F0Fu);
                a1 = bk_sub8(w1 & 0x0F0F0F0Fu); a3 = bk_sub8((w1 >> 4) & 0x0F0F0F0Fu);
            } else {
                const int4 w = wq[j & (NQ - 1)];
                a0 = w.x; a1 = w.y; a2 = w.z; a3 = w.w;
            }
            const float d0 = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? dw0[j >> 1] >> 16 : dw0[j >> 1] & 0xffffu)));
            const float d1 = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? dw1[j >> 1] >> 16 : dw1[j >> 1] & 0xffffu)));
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const int4 bq = aq[n][j >> 1];
                int c[4] = { 0, 0, 0, 0 };
                bk_mma_s8(c, a0, a1, a2, a3, (j & 1) ? bq.z : bq.x, (j & 1) ? bq.w : bq.y);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int4     xv = ax[n][e];
                    const uint32_t xw = (uint32_t) ((j >> 1) == 0 ? xv.x : (j >> 1) == 1 ? xv.y : (j >> 1) == 2 ? xv.z : xv.w);
                    const float    dx = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? xw >> 16 : xw & 0xffffu)));
                    acc[n][e]     = fmaf(__fmul_rn(d0, dx), (float) c[e], acc[n][e]);
                    acc[n][2 + e] = fmaf(__fmul_rn(d1, dx), (float) c[2 + e], acc[n][2 + e]);
                }
            }
        }
        if (sn < s1) {
#pragma unroll
            for (int c = 0; c < NQ; c++) wq[c] = wn[c];
            dq[0] = dn[0]; dq[1] = dn[1];
        }
    }

    __shared__ float red[BK_WARPS][NT * 8][16];
    __shared__ bool  s_last;
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            red[warp][n * 8 + 2 * t + e][g]     = acc[n][e];
            red[warp][n * 8 + 2 * t + e][g + 8] = acc[n][2 + e];
        }
    __syncthreads();
    for (int i = threadIdx.x; i < NT * 8 * 16; i += BK_THREADS) {
        const int tok = i / 16, r = i % 16, row = T * 16 + r;
        if (tok < b && row < N) {
            float v = red[0][tok][r];
#pragma unroll
            for (int w2 = 1; w2 < BK_WARPS; w2++) v += red[w2][tok][r];
            if (nsplit == 1) y[(size_t) tok * N + row] = v;
            else partial[((size_t) split * b + tok) * N + row] = v;
        }
    }
    if (nsplit == 1) return;
    __syncthreads();
    if (threadIdx.x == 0) { __threadfence(); s_last = atomicAdd(&counters[T], 1u) == (unsigned) nsplit - 1; }
    __syncthreads();
    if (!s_last) return;
    for (int i = threadIdx.x; i < NT * 8 * 16; i += BK_THREADS) {
        const int tok = i / 16, r = i % 16, row = T * 16 + r;
        if (tok < b && row < N) {
            float v = 0.f;
            for (int sp = 0; sp < nsplit; sp++) v += __ldcg(partial + ((size_t) sp * b + tok) * N + row);
            y[(size_t) tok * N + row] = v;
        }
    }
    if (threadIdx.x == 0) counters[T] = 0;
}

// The same without a K split, for row tiles that are there (nearly) all at once: WARPS warps per tile, every warp streams its records through a private ring in shared
// memory filled by cp.async, STAGES - 1 of them in flight (as gemv_q4k_ring_kernel).
// What bounds it: a warp's chain of memory latencies, which more warps and a deeper prefetch shorten.  4096 x 4096 Q4_0 at 8 / 16 tokens 6.2 / 12.0 -> 4.4 / 7.7 us,
// 4096 x 11008 9.8 / 20.8 -> 8.5 / 15.5, 11264 x 2048 (four warps) 7.3 -> 5.3; two token groups with two CTAs per SM instead of one: 4096 x 4096 7.0 -> 4.3,
// 4096 x 11008 12.7 -> 9.3, 8192 x 4096 13.0 -> 8.0.  With one token group and more rounds of tiles new CTAs keep arriving with their first records in flight, the
// ring's extra pass through shared memory is what counts (22016 x 4096 at 7 tokens 16.0 -> 16.5, Q8_0 18.9 -> 24.5), and gemv_blk32_kernel stays: pib_gemv_blk32.
template <int WT, int NT, int WARPS, int STAGES>
__global__ void __launch_bounds__(WARPS * 32, NT == 1 ? (WARPS == 4 ? 5 : 2) : (WARPS == 4 ? 3 : 2))
gemv_blk32_ring_kernel(const uint8_t * __restrict__ tiles, int ngr, int N, const int8_t * __restrict__ aqs, const __half * __restrict__ adx, int b, float * __restrict__ y, const int * __restrict__ cancel) {
    if (PIB_CANCELLED(cancel)) { pib_pdl_wait(); return; }
    constexpr int REC = WT == PIB_TYPE_Q4_0 ? 2304 : 4352, PIECES = (REC + 511) / 512;        // 512 bytes per warp-wide copy, the last one half
    constexpr int NQ  = WT == PIB_TYPE_Q4_0 ? 4 : 8;            // 16-byte quant pieces per lane and record
    extern __shared__ __align__(16) uint8_t bk_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int T = blockIdx.x;
    const uint8_t * tbase  = tiles + (size_t) T * ngr * REC + lane * 16;
    uint8_t *       ring   = bk_smem + warp * (STAGES * REC);
    const uint32_t  ring_a = (uint32_t) __cvta_generic_to_shared(ring) + lane * 16;
    int ps = warp;                                         // prefetch cursor
    auto issue = [&](int stage) {
        if (ps < ngr) {
            const uint8_t * src = tbase + (size_t) ps * REC;
            const uint32_t  dst = ring_a + stage * REC;
#pragma unroll
            for (int c = 0; c < PIECES; c++)
                if (c < PIECES - 1 || lane < 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * 512), "l"(src + c * 512) : "memory");
            ps += WARPS;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the weights are immutable: their copies start before the wait on the kernel that produces the activations
#pragma unroll
    for (int i = 0; i < STAGES - 1; i++) issue(i);

    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) { acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f; }
    const int8_t * a_q[NT];
    const __half * a_d[NT][2];
    int            gs[NT];                                      // tokens of the octet (pib_oct)
#pragma unroll
    for (int n = 0; n < NT; n++) {
        gs[n] = min(8, b - 8 * n);
        a_q[n] = aqs + (size_t) n * 8 * ngr * 256 + min(g, gs[n] - 1) * 64 + t * 16;
#pragma unroll
        for (int e = 0; e < 2; e++) a_d[n][e] = adx + ((size_t) n * 8 * ngr + min(2 * t + e, gs[n] - 1)) * 8;
    }
    pib_pdl_wait();
    pib_pdl_trigger();
    int stage = 0;
    for (int s = warp; s < ngr; s += WARPS) {
        int4 aq[NT][4];
        int4 ax[NT][2];
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const int sg = s * gs[n];
            const int4 * ap = reinterpret_cast<const int4 *>(a_q[n] + (size_t) sg * 256);
#pragma unroll
            for (int c = 0; c < 4; c++) aq[n][c] = __ldg(ap + c * 4 * gs[n]);
#pragma unroll
            for (int e = 0; e < 2; e++) ax[n][e] = __ldg(reinterpret_cast<const int4 *>(a_d[n][e] + (size_t) sg * 8));
        }
        __syncwarp();                                           // every lane has used the stage about to be refilled
        issue((stage + STAGES - 1) % STAGES);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        const uint8_t * rs = ring + stage * REC;
        int4 wq[NQ], dq[2];
#pragma unroll
        for (int c = 0; c < NQ; c++) wq[c] = *reinterpret_cast<const int4 *>(rs + c * 512 + lane * 16);
        dq[0] = *reinterpret_cast<const int4 *>(rs + (REC - 256) + g * 16);
        dq[1] = *reinterpret_cast<const int4 *>(rs + (REC - 256) + (g + 8) * 16);
        const uint32_t dw0[4] = { (uint32_t) dq[0].x, (uint32_t) dq[0].y, (uint32_t) dq[0].z, (uint32_t) dq[0].w };   // row g:   d of blocks 2i | 2i+1
        const uint32_t dw1[4] = { (uint32_t) dq[1].x, (uint32_t) dq[1].y, (uint32_t) dq[1].z, (uint32_t) dq[1].w };   // row g+8
#pragma unroll
        for (int j = 0; j < 8; j++) {
            int a0, a1, a2, a3;
            if (WT == PIB_TYPE_Q4_0) {
                const int4     w  = wq[j >> 1];
                const uint32_t w0 = (uint32_t) ((j & 1) ? w.z : w.x), w1 = (uint32_t) ((j & 1) ? w.w : w.y);
                a0 = bk_sub8(w0 & 0x0F0F0F0Fu); a2 = bk_sub8((w0 >> 4) & 0x0F0F0F0Fu);
                a1 = bk_sub8(w1 & 0x0F0F0F0Fu); a3 = bk_sub8((w1 >> 4) & 0x0F0F0F0Fu);
            } else {
                const int4 w = wq[j & (NQ - 1)];
                a0 = w.x; a1 = w.y; a2 = w.z; a3 = w.w;
            }
            const float d0 = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? dw0[j >> 1] >> 16 : dw0[j >> 1] & 0xffffu)));
            const float d1 = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? dw1[j >> 1] >> 16 : dw1[j >> 1] & 0xffffu)));
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const int4 bq = aq[n][j >> 1];
                int c[4] = { 0, 0, 0, 0 };
                bk_mma_s8(c, a0, a1, a2, a3, (j & 1) ? bq.z : bq.x, (j & 1) ? bq.w : bq.y);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int4     xv = ax[n][e];
                    const uint32_t xw = (uint32_t) ((j >> 1) == 0 ? xv.x : (j >> 1) == 1 ? xv.y : (j >> 1) == 2 ? xv.z : xv.w);
                    const float    dx = __half2float(__ushort_as_half((unsigned short) ((j & 1) ? xw >> 16 : xw & 0xffffu)));
                    acc[n][e]     = fmaf(__fmul_rn(d0, dx), (float) c[e], acc[n][e]);
                    acc[n][2 + e] = fmaf(__fmul_rn(d1, dx), (float) c[2 + e], acc[n][2 + e]);
                }
            }
        }
        stage = stage + 1 == STAGES ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                            // the rings are done with: their memory becomes the reduction buffer

    float (*red)[NT * 8][16] = reinterpret_cast<float (*)[NT * 8][16]>(bk_smem);
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            red[warp][n * 8 + 2 * t + e][g]     = acc[n][e];
            red[warp][n * 8 + 2 * t + e][g + 8] = acc[n][2 + e];
        }
    __syncthreads();
    for (int i = threadIdx.x; i < NT * 8 * 16; i += WARPS * 32) {
        const int tok = i / 16, r = i % 16, row = T * 16 + r;
        if (tok < b && row < N) {
            float v = red[0][tok][r];
#pragma unroll
            for (int w2 = 1; w2 < WARPS; w2++) v += red[w2][tok][r];
            y[(size_t) tok * N + row] = v;
        }
    }
}

// ---- launcher -----------------------------------------------------------------------------------------------------------
struct bk_scratch { float * partial = nullptr; unsigned int * counters = nullptr; };
static std::map<std::pair<int, cudaStream_t>, bk_scratch> g_bk_scratch;
static std::mutex                                        g_bk_mu;

// per (device, stream), sized once for every shape the split rule can produce (see gemv_mma.cu: ensure_scratch)
static int bk_ensure_scratch(cudaStream_t st, bk_scratch ** out) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_bk_mu);
    bk_scratch & s = g_bk_scratch[std::make_pair(dev, st)];
    if (!s.partial) {
        if (cudaMalloc(&s.partial, (size_t) 32 << 20) != cudaSuccess || cudaMalloc(&s.counters, 8192 * sizeof(unsigned int)) != cudaSuccess) {
            cudaGetLastError();
            return PIB_ERR_NOMEM;
        }
        cudaMemset(s.counters, 0, 8192 * sizeof(unsigned int));
    }
    *out = &s;
    return PIB_OK;
}

int pib_split_fill_target();         // gemv_mma.cu: CTA count below which a k split is worth its second phase

bool pib_gemv_blk32_supported(const pib_weight * w, int b) {
    return w && (w->type == PIB_TYPE_Q4_0 || w->type == PIB_TYPE_Q8_0) && w->tiles != nullptr && b >= 1 && b <= PIB_MAX_BATCH;
}

template <int WT, int NT, int WARPS, int STAGES>
static int bk_ring_launch(const pib_weight * w, int ngr, const int8_t * aqs, const __half * adx, int b, float * y_dev, const int * cancel, cudaStream_t st) {
    const int    n_tiles = (int) ((w->N + 15) / 16);
    const size_t ring = (size_t) WARPS * STAGES * bk_rec_bytes(WT), smem = WARPS == 8 ? pib_gemv_smem_spread(ring, n_tiles) : ring;
    static pib_per_device attrs;
    PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(gemv_blk32_ring_kernel<WT, NT, WARPS, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) (ring > PIB_GEMV_SPREAD ? ring : PIB_GEMV_SPREAD)); }));
    PIB_CHECK(pib_launch(gemv_blk32_ring_kernel<WT, NT, WARPS, STAGES>, dim3((unsigned) n_tiles), dim3(WARPS * 32), smem, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, cancel));
    return PIB_OK;
}

int pib_gemv_blk32(const pib_weight * w, const void * act_dev, int b, float * y_dev, const int * cancel, cudaStream_t st) {
    if (!pib_gemv_blk32_supported(w, b)) { pib_set_error("pib_gemv: the tensor-core variant needs Q4_0 / Q8_0 weights with tiles"); return PIB_ERR_UNSUPP; }
    const pib_act_layout L   = pib_act_layout_of(w->type, w->K, b);
    const uint8_t *      act = (const uint8_t *) act_dev;
    const int            ngr = (int) ((w->K + 255) / 256), n_tiles = (int) ((w->N + 15) / 16);
    const int8_t *       aqs = (const int8_t *) (act + L.qsp_off);
    const __half *       adx = (const __half *) (act + L.bs8_off);    // dxp plane of the 32-element block formats
    // The ring kernels or the K split below, by where each was faster (us, ring / K split).  What decides are rounds: of the ring's eight-warp CTAs an SM holds two, of its
    // four-warp CTAs five, of the K split's four.
    // One token group, eight warps: while the K split would split, since from 80 % of its slots on it runs unsplit in one round (4096 wide, 8 tokens: 444 tiles of Q4_0
    // 7.3 / 10.1, 512 tiles 7.3 / 6.7; Q8_0 8.6 / 10.6 and 8.9 / 7.2).
    // Two token groups, eight warps (where four, below, are not faster; behind a quantiser, 13 tokens): any number of tiles of Q4_0 (4096 wide, 740 tiles 12.8 / 14.6, 1376 20.9 / 23.0, 2000 27.5 / 28.8); of Q8_0 up to four tiles
    // per SM and rows from 6144 on (4096 wide, 592 tiles 13.1 / 15.8, 880 18.5 / 17.1, 1184 22.9 / 22.2; 8192 wide, 740 25.4 / 26.7, 1376 40.6 / 45.5).
    // Few tiles of long rows go to the K split, which divides a row over up to 64 warps (28672 wide, 32 tiles: 8.8 / 5.1 and, 13 tokens, 14.5 / 11.0; 64 tiles 9.2 / 6.9 and
    // 14.6 / 15.8; 80 tiles 9.3 / 9.9; 8192 wide, 16 tiles 3.3 / 3.2, 48 3.5 / 4.1).
    // Four warps (Q4_0, one token group): one round of them, where eight make a second round with little in it, where the K split would split, takes a second round, or has too few records per
    // warp (8 tokens: 28672 wide, 328 tiles 28.1, eight warps 33.5, K split 30.9, 740 tiles 43.8 / 58.6; 2048 wide, 444 tiles 4.3 / 7.3, 592 4.5 / 4.7; 3072 wide, 592 6.0 / 5.7).
    // Four warps, two token groups (three CTAs per SM; us at 9 / 16 tokens, before / four-warp ring): up to a round of them (4096 wide, 444 tiles of Q4_0 9.8 9.8 / 8.7 8.9, of Q8_0 11.7
    // 12.3 / 9.5 9.7; 2048 wide 10.6 10.7 / 7.6 7.8) but not few tiles of long rows (256 of 11008 12.8 / 15.1 at 16), and from two rounds on (4096 wide, 2000 tiles, 13 tokens: Q4_0 27.6 / 25.5,
    // Q8_0 32.5 / 28.2; 57344 x 8192 76.1 80.7 / 72.4 75.6 and 88.7 88.6 / 82.3 89.8); between, eight warps have fuller rounds (Q4_0 512 tiles 10.5 10.6 / 11.4 11.4, 640 12.1 12.4 / 12.8
    // 12.7; Q8_0 512 tiles of 8192 18.5 18.8 / 20.4 20.6), except of Q8_0 in rows up to 4096 (640 tiles 14.8 14.8 / 13.4 13.6) and of short rows (704 of 2048 at 13: 9.2 / 8.7, 10.2 / 9.7).
    // Not for Q8_0 in rows of 1024 (one round, 310 tiles at 13: 4.4 / 4.7; 444 of 1536 7.0 / 6.1) or of many records (1800 tiles of 12288 at 9 and 13: 70.3 65.7 / 72.7 73.4, of 7168 45.1 47.5 /
    // 39.7 45.2).
    // One token group of Q4_0 from 2.4 rounds of them on (four or fewer tokens, or long rows): 57344 x 8192 at 1, 4, 7 tokens 52.3 55.2 56.5 / 50.2 51.4 55.0, 57344 x 4096 at 3 30.8 / 28.9, but
    // 32000 x 4096 at 8 19.4 / 20.5.  The sums are those of the four-warp K split where it does not split.
    const int  sms = pib_num_sms(), fill = pib_split_fill_target();
    const bool two = b > 8, q8 = w->type == PIB_TYPE_Q8_0;
    const bool many = two ? (n_tiles > 2 * sms && ngr <= 16 && (n_tiles <= 3 * sms ? !q8 || ngr > 4 : q8 ? ngr > 8 || n_tiles > 4 * sms : ngr <= 8 || n_tiles > 6 * sms)) ||
                                (n_tiles > 8 * sms && (!q8 || ngr <= 28))
                          : !q8 && n_tiles > 12 * sms && (b <= 4 || ngr >= 32);
    const bool four = !q8 && !two && n_tiles > 2 * sms && n_tiles <= 5 * sms && (ngr <= 8 || 5 * n_tiles <= 12 * sms || n_tiles > 4 * sms || (ngr < 16 && n_tiles < fill));
    const bool wide = ngr == 16 || 2 * n_tiles >= 3 * ngr || (two ? 5 * n_tiles >= 2 * sms : 2 * n_tiles > sms);
    if (many) {
        if (q8) return bk_ring_launch<PIB_TYPE_Q8_0, 2, 4, 3>(w, ngr, aqs, adx, b, y_dev, cancel, st);
        return two ? bk_ring_launch<PIB_TYPE_Q4_0, 2, 4, 4>(w, ngr, aqs, adx, b, y_dev, cancel, st) : bk_ring_launch<PIB_TYPE_Q4_0, 1, 4, 4>(w, ngr, aqs, adx, b, y_dev, cancel, st);
    }
    if (four) return bk_ring_launch<PIB_TYPE_Q4_0, 1, 4, 4>(w, ngr, aqs, adx, b, y_dev, cancel, st);
    if (ngr >= 16 && wide && (two ? w->type == PIB_TYPE_Q4_0 || n_tiles <= 4 * sms || ngr >= 24 : n_tiles < fill)) {
        if (w->type == PIB_TYPE_Q4_0) return two ? bk_ring_launch<PIB_TYPE_Q4_0, 2, 8, 4>(w, ngr, aqs, adx, b, y_dev, cancel, st) : bk_ring_launch<PIB_TYPE_Q4_0, 1, 8, 4>(w, ngr, aqs, adx, b, y_dev, cancel, st);
        return two ? bk_ring_launch<PIB_TYPE_Q8_0, 2, 8, 3>(w, ngr, aqs, adx, b, y_dev, cancel, st) : bk_ring_launch<PIB_TYPE_Q8_0, 1, 8, 3>(w, ngr, aqs, adx, b, y_dev, cancel, st);
    }
    // k splits: enough CTAs to fill the machine when there are few row tiles; at least two records per warp
    int split = 1;
    while (n_tiles * split < pib_split_fill_target() && split * 2 * BK_WARPS <= ngr && split < 16) split *= 2;     // see gemv_mma.cu
    while (split > 1 && ((size_t) split * b * w->N * sizeof(float) > ((size_t) 32 << 20) || n_tiles > 8192)) split /= 2;
    bk_scratch * s = nullptr;
    if (split > 1 && bk_ensure_scratch(st, &s) != PIB_OK) { pib_set_error("pib_gemv: scratch allocation failed"); return PIB_ERR_NOMEM; }
    const dim3     grid(n_tiles, split);
    float *        pp  = s ? s->partial : nullptr;
    unsigned int * cc  = s ? s->counters : nullptr;
    cudaError_t    e;
    if (w->type == PIB_TYPE_Q4_0) {
        if (b == 1) e = pib_launch(gemv_blk32_kernel<PIB_TYPE_Q4_0, 1, true>, grid, dim3(BK_THREADS), 0, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, pp, cc, cancel);
        else if (b <= 8) e = pib_launch(gemv_blk32_kernel<PIB_TYPE_Q4_0, 1, false>, grid, dim3(BK_THREADS), 0, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, pp, cc, cancel);
        else        e = pib_launch(gemv_blk32_kernel<PIB_TYPE_Q4_0, 2, false>, grid, dim3(BK_THREADS), 0, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, pp, cc, cancel);
    } else {
        if (b <= 8) e = pib_launch(gemv_blk32_kernel<PIB_TYPE_Q8_0, 1, false>, grid, dim3(BK_THREADS), 0, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, pp, cc, cancel);
        else        e = pib_launch(gemv_blk32_kernel<PIB_TYPE_Q8_0, 2, false>, grid, dim3(BK_THREADS), 0, st, w->tiles, ngr, (int) w->N, aqs, adx, b, y_dev, pp, cc, cancel);
    }
    PIB_CHECK(e);
    return PIB_OK;
}
