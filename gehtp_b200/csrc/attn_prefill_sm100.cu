// Prefill attention on tcgen05 / TMEM: softmax(Q K^T * scale + mask) V, head_dim 128, grouped-query heads.
//
// Same op chain and the same fp16 rounding points of a score as ops_attn_prefill.cu (after the dot
// product, after the scale, after the mask); the probabilities are exp(s - rowmax) / rowsum rounded to
// fp16 before they meet V; the division by the row sum is applied to the fp32 output accumulator (the reference's
// SOFTMAX op, oplist_exec.c:1163-1194, divides first and rounds then: a difference of rounding only).
//
// One CTA = one query head x 128 query rows. Key/value tiles of 128 positions; tiles whose mask is -inf everywhere (upper
// triangle of a causal mask) are skipped, the others are dealt out in turn to two groups of four softmax warps, each with its
// own S, O, row maximum and row sum. While one group works on its scores the tensor core runs the products of the other; the
// two halves of the result are added at the end. Halving the chain of a row tile this way is what a prompt of a few hundred
// tokens needs (64 CTAs of up to four tiles at 512 tokens and 16 heads: no CTA has a second one beside it on its SM).
//
//   S = Q K^T   tcgen05.mma into TMEM
//   P           one thread per row: score roundings on half2 pairs (a scale that fp16 holds multiplies them as half2: the
//               product of two fp16 values, rounded once, is what the fp32 product rounds to), maximum, 2^(s - m) rounded to
//               fp16 and written over S
//   O += P V    tcgen05.mma with P as the A operand from TMEM
// The maximum a row is referred to is raised - and its O rescaled - only when a tile exceeds it by more than 2^8.
// Bound by the exponentials (16 a cycle and SM) and the ALU work beside them. Against two passes over the tiles (maxima first)
// by one group: 16 heads and 512 positions 16 -> 10 us a layer, 32 heads and 2048 positions 115 -> 66. With one live tile (up to 128
// positions) the second group has nothing to do, and the one pass is still ahead: prompts of four layers of 16 heads, 64 tokens
// 287 -> 270 us, 128 tokens 322 -> 297.
//
// Operands: Q, K token-major (head_dim contiguous) are K-major for S = Q K^T; for O = P V the contraction runs over key
// positions: V is read as it lies in memory ([position][head_dim]) and declared an MN-major B operand (instruction
// descriptor bit 16; boxes of 64 positions x 64 head_dim values, see umma_desc_v).
//
//   warp 0     TMA producer: Q once, then the K and V tiles, one buffer of each per group
//   warp 1     one lane issues tcgen05.mma / tcgen05.commit
//   warp 2     owns the TMEM allocation (512 columns: S / P and O of both groups)
//   warps 4-11 softmax: warp w works on TMEM lanes 32 (w % 4) .. +31, one query row per thread, group (w - 4) / 4
// Every mbarrier wait is bounded; on a timeout the CTA raises the engine's status word and winds down.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include "common.cuh"
#include "launchers_attn.h"
#include "sm100_attn.cuh"

namespace gehtp {

using namespace sm100;

namespace {

constexpr int BQ = 128, BKV = 128, HD = 128, TILE_BYTES = 128 * 64 * 2;   // one 128 x 64 fp16 box
constexpr int NTHREADS = 384;

constexpr float RAISE = 8.0f;

struct __align__(8) ABars {
    uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_full, merge;
    uint32_t tmem_base, abort_flag;
    unsigned long long live, zero;   // bit kt: tile (qt, kt) has a live entry / a mask of +0 everywhere (n_kt <= 64)
};

struct SmArgs {
    const uint16_t* mask;        // [heads or 1][seq_q][seq_k] additive fp16, or NULL
    size_t mask_head_stride;
    const uint8_t* skip;         // [ceil(seq_q/64)][ceil(seq_k/64)], 1 = 64 x 64 tile fully masked, or NULL
    const uint8_t* zero;         // same shape, 1 = the mask of the 64 x 64 tile is +0 everywhere, or NULL
    uint16_t* out;               // [seq_q][nh * 128]
    uint32_t seq_q, seq_k, nh, kvh;
    float scale;
    int scale_div;
    unsigned int* status;
};

// Two fp32 values -> one half2 word (low half = a) in one instruction, and back.
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ __half2 as_h2(uint32_t w) { return *(const __half2*)&w; }
__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *(const uint32_t*)&h; }
__device__ __forceinline__ float2 unpack_h2(uint32_t h) { return __half22float2(as_h2(h)); }
// piece `p` of row `row` (16 bytes) in a tile of 32 rows of 16 pieces: rows of a piece and pieces of a row lie on different banks
__device__ __forceinline__ uint32_t mask_at(uint32_t row, uint32_t p) { return row * 16 + (p ^ (row & 15)); }

// the scores of 32 positions of a row from its 32 dot products, as 16 half2 words
template <bool HALF_SCALE>
__device__ __forceinline__ void scores32(const uint32_t (&v)[32], uint32_t* h, bool masked, const uint4* mask, uint32_t row, uint32_t piece, float rscale, uint32_t rscale2) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
        uint32_t w = pack_h2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        if (HALF_SCALE) {
            w = as_u32(__hmul2_rn(as_h2(w), as_h2(rscale2)));
        } else {
            const float2 f = unpack_h2(w);
            w = pack_h2(__fmul_rn(f.x, rscale), __fmul_rn(f.y, rscale));
        }
        h[i] = w;
    }
    if (masked) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint4 p = mask[mask_at(row, piece + q)];
            h[4 * q] = as_u32(__hadd2_rn(as_h2(h[4 * q]), as_h2(p.x)));
            h[4 * q + 1] = as_u32(__hadd2_rn(as_h2(h[4 * q + 1]), as_h2(p.y)));
            h[4 * q + 2] = as_u32(__hadd2_rn(as_h2(h[4 * q + 2]), as_h2(p.z)));
            h[4 * q + 3] = as_u32(__hadd2_rn(as_h2(h[4 * q + 3]), as_h2(p.w)));
        }
    }
}

// true: the 128 x 128 tile (qt, kt) has no live entry
__device__ __forceinline__ bool tile_dead(const uint8_t* skip, uint32_t qt, uint32_t kt, uint32_t nq64, uint32_t nk64) {
    if (!skip) return false;
    for (uint32_t a = 0; a < 2; a++)
        for (uint32_t b = 0; b < 2; b++) {
            const uint32_t r = 2 * qt + a, c = 2 * kt + b;
            if (r < nq64 && c < nk64 && !skip[(size_t)r * nk64 + c]) return false;
        }
    return true;
}

// true: the mask of the 128 x 128 tile (qt, kt) is +0 on all its entries
__device__ __forceinline__ bool tile_zero(const uint8_t* zero, uint32_t qt, uint32_t kt, uint32_t nq64, uint32_t nk64) {
    if (!zero) return false;
    for (uint32_t a = 0; a < 2; a++)
        for (uint32_t b = 0; b < 2; b++) {
            const uint32_t r = 2 * qt + a, c = 2 * kt + b;
            if (r < nq64 && c < nk64 && !zero[(size_t)r * nk64 + c]) return false;
        }
    return true;
}

// Mask values of 32 rows (row0 on; past the last: of the last) for the 128 positions from key0 on into shared memory, by one
// warp. Positions past the sequence count as masked out; bytes outside the mask tensor are never read. Code that runs once
// in a CTA costs its fetch (about 3 ns an instruction): loops stay rolled, and the function is no part of the score loop.
__device__ __noinline__ void mask_tile(const uint16_t* mask, const uint16_t* end, uint32_t row0, uint32_t rows, uint32_t key0, uint32_t seq_k, uint4* out) {
    const uint32_t lane = threadIdx.x & 31;
    const uint4 none = make_uint4(0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u);
    if (mask && (seq_k & 7u) == 0 && ((uintptr_t)mask & 15u) == 0) {
        // pieces of 16 bytes lie inside a row or past its end; 16 lanes to a row, all requests in flight
        const uint32_t p = lane & 15, k = key0 + 8 * p;
#pragma unroll 1
        for (uint32_t r = lane >> 4; r < 32; r += 2) {
            if (k < seq_k)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(out + mask_at(r, p))), "l"(mask + (size_t)min(row0 + r, rows - 1) * seq_k + k) : "memory");
            else
                out[mask_at(r, p)] = none;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        return;
    }
    // Rows that start on no 16-byte boundary, one to a lane: five aligned pieces for 32 positions, moved into place by 8, 4 and 2
    // bytes. (One 2-byte load per position: 16 heads x 333 positions twice the time of the layer.)
    const uint16_t* mrow = mask ? mask + (size_t)min(row0 + lane, rows - 1) * seq_k : nullptr;
#pragma unroll 1
    for (uint32_t c = 0; c < 4; c++, key0 += 32) {
        uint32_t mk[16];
        const uint32_t past = seq_k > key0 ? seq_k - key0 : 0;                          // positions of the piece before the end
        const uintptr_t at = (uintptr_t)(mrow + key0), lo = at & ~(uintptr_t)15;
        if (mrow && past && lo >= (uintptr_t)mask && lo + 80 <= (uintptr_t)end) {
            const uint32_t by = (uint32_t)(at & 15);
            uint32_t w[20];
#pragma unroll
            for (int q4 = 0; q4 < 5; q4++) {
                const uint4 p = __ldg((const uint4*)lo + q4);
                w[4 * q4] = p.x; w[4 * q4 + 1] = p.y; w[4 * q4 + 2] = p.z; w[4 * q4 + 3] = p.w;
            }
#pragma unroll
            for (int i = 0; i < 18; i++) w[i] = by & 8u ? w[i + 2] : w[i];
#pragma unroll
            for (int i = 0; i < 17; i++) w[i] = by & 4u ? w[i + 1] : w[i];
#pragma unroll
            for (int i = 0; i < 16; i++) {
                uint32_t x = by & 2u ? __funnelshift_r(w[i], w[i + 1], 16) : w[i];
                if (2u * i >= past) x = 0xFC00FC00u;
                else if (2u * i + 1 >= past) x = (x & 0xFFFFu) | 0xFC000000u;
                mk[i] = x;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const uint32_t k = key0 + 2 * i;
                const uint32_t lo16 = k < seq_k ? (mrow ? mrow[k] : 0u) : 0xFC00u, hi16 = k + 1 < seq_k ? (mrow ? mrow[k + 1] : 0u) : 0xFC00u;
                mk[i] = lo16 | (hi16 << 16);
            }
        }
#pragma unroll
        for (uint32_t q4 = 0; q4 < 4; q4++) out[mask_at(lane, c * 4 + q4)] = make_uint4(mk[4 * q4], mk[4 * q4 + 1], mk[4 * q4 + 2], mk[4 * q4 + 3]);
    }
    __syncwarp();
}

// HALF_SCALE: the scale is an fp16 value
template <bool HALF_SCALE>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_prefill_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                          const __grid_constant__ CUtensorMap tmap_v, const SmArgs A) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sQ = smem;                          // 2 boxes (head_dim halves)
    unsigned char* sK = sQ + 2 * TILE_BYTES;           // 2 groups x 2 boxes
    unsigned char* sV = sK + 4 * TILE_BYTES;           // 2 groups x 2 boxes (position halves)
    unsigned char* sM = sV + 4 * TILE_BYTES;           // 2 groups x 4 warps x 32 rows x 128 mask values
    ABars* bars = (ABars*)(sM + 4 * TILE_BYTES);
    volatile uint32_t* abort_flag = &bars->abort_flag;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t qt = gridDim.y - 1 - blockIdx.y;     // the longest rows of all heads first
    const uint32_t head = blockIdx.x, kvhd = head / (A.nh / A.kvh);
    const uint32_t q0 = qt * BQ;
    const uint32_t n_kt = (A.seq_k + BKV - 1) / BKV;
    const uint32_t nq64 = (A.seq_q + 63) / 64, nk64 = (A.seq_k + 63) / 64;

    if (threadIdx.x == 0) {
        mbar_init(&bars->q_full, 1); mbar_init(&bars->o_full, 1); mbar_init(&bars->merge, 8);
        for (int s = 0; s < 2; s++) {
            mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1);
            mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], 1);
            mbar_init(&bars->s_full[s], 1); mbar_init(&bars->p_full[s], 4);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 32)
        for (const CUtensorMap* map : {&tmap_q, &tmap_k, &tmap_v}) asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    if (warp == 3) {
        // which key tiles this CTA works on, read once (the tables are constants: no need to wait for the predecessor)
        unsigned long long lv = 0, zr = 0;
        for (uint32_t kt = lane; kt < n_kt; kt += 32) {
            if (!tile_dead(A.skip, qt, kt, nq64, nk64)) lv |= 1ull << kt;
            if (tile_zero(A.zero, qt, kt, nq64, nk64)) zr |= 1ull << kt;
        }
        for (int o = 16; o; o >>= 1) { lv |= __shfl_xor_sync(0xffffffffu, lv, o); zr |= __shfl_xor_sync(0xffffffffu, zr, o); }
        if (lane == 0) { bars->live = lv; bars->zero = zr; }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars->tmem_base;
    const unsigned long long live = bars->live, zero_tiles = bars->zero;
    const uint32_t n_live = (uint32_t)__popcll(live);   // tile number i (in order) belongs to group i % 2, as its i / 2 th

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0 && n_live) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            mbar_expect_tx(&bars->q_full, 2 * TILE_BYTES);
            tma_load_2d(sQ, &tmap_q, (int)(head * HD), (int)q0, &bars->q_full);
            tma_load_2d(sQ + TILE_BYTES, &tmap_q, (int)(head * HD + 64), (int)q0, &bars->q_full);
            unsigned long long rest = live;
            uint32_t kn = 0, vn = 0;                    // tiles requested
            while (vn < n_live && !*abort_flag) {
                uint32_t kt[2];
                const uint32_t n = min(2u, n_live - vn);
                for (uint32_t t = 0; t < n; t++) { kt[t] = (uint32_t)__ffsll((long long)rest) - 1; rest &= rest - 1; }
                for (uint32_t t = 0; t < n; t++) {
                    if (!mbar_wait_or_abort(&bars->k_empty[t], ((kn >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; break; }
                    mbar_expect_tx(&bars->k_full[t], 2 * TILE_BYTES);
                    tma_load_2d(sK + t * 2 * TILE_BYTES, &tmap_k, (int)(kvhd * HD), (int)(kt[t] * BKV), &bars->k_full[t]);
                    tma_load_2d(sK + t * 2 * TILE_BYTES + TILE_BYTES, &tmap_k, (int)(kvhd * HD + 64), (int)(kt[t] * BKV), &bars->k_full[t]);
                    kn++;
                }
                for (uint32_t t = 0; t < n && !*abort_flag; t++) {
                    if (!mbar_wait_or_abort(&bars->v_empty[t], ((vn >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; break; }
                    mbar_expect_tx(&bars->v_full[t], 2 * TILE_BYTES);
                    // [position half][head_dim half][64 positions x 128 bytes]
#pragma unroll
                    for (uint32_t b4 = 0; b4 < 4; b4++)
                        tma_load_2d(sV + t * 2 * TILE_BYTES + b4 * (TILE_BYTES / 2), &tmap_v, (int)(kvhd * HD + (b4 & 1) * 64),
                                    (int)(kt[t] * BKV + (b4 >> 1) * 64), &bars->v_full[t]);
                    vn++;
                }
            }
            if (*abort_flag) {   // copies already requested must land before the CTA may go away
                mbar_wait(&bars->q_full, 0);
                for (uint32_t j = kn > 2 ? kn - 2 : 0; j < kn; j++) mbar_wait(&bars->k_full[j & 1], (j >> 1) & 1);
                for (uint32_t j = vn > 2 ? vn - 2 : 0; j < vn; j++) mbar_wait(&bars->v_full[j & 1], (j >> 1) & 1);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0 && n_live) {
            const uint32_t q_base = smem_u32(sQ), k_base = smem_u32(sK), v_base = smem_u32(sV);
            bool ok = true;
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok) ok = mbar_wait_or_abort(bar, parity, abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return ok;
            };
            // S of tile i: 2 head_dim halves x 4 steps of k16
            auto issue_s = [&](uint32_t i) {
                const uint32_t t = i & 1;
                if (!wait(&bars->k_full[t], (i >> 1) & 1)) return;
#pragma unroll
                for (uint32_t kb = 0; kb < 2; kb++)
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; k4++)
                        umma_f16(tmem + t * 128, umma_desc(q_base + kb * TILE_BYTES) + (uint64_t)(k4 * 2),
                                 umma_desc(k_base + t * 2 * TILE_BYTES + kb * TILE_BYTES) + (uint64_t)(k4 * 2), idesc_f16(128), (kb | k4) ? 1u : 0u);
                umma_commit(&bars->k_empty[t]);
                umma_commit(&bars->s_full[t]);
            };
            if (wait(&bars->q_full, 0)) {
                issue_s(0);
                if (n_live > 1) issue_s(1);
            }
            for (uint32_t i = 0; ok && i < n_live; i++) {
                const uint32_t t = i & 1, ph = (i >> 1) & 1;
                if (!wait(&bars->v_full[t], ph) || !wait(&bars->p_full[t], ph)) break;
#pragma unroll
                for (uint32_t k = 0; k < 8; k++)                // 16 positions = two 8-position groups = 2048 bytes; bit 16: B is MN-major
                    umma_f16_ta(tmem + 256 + t * 128, tmem + t * 128 + k * 8, umma_desc_v(v_base + t * 2 * TILE_BYTES + (k >> 2) * TILE_BYTES + (k & 3) * 2048),
                                idesc_f16(128) | (1u << 16), (i > 1 || k) ? 1u : 0u);
                umma_commit(&bars->v_empty[t]);
                if (i + 2 < n_live) issue_s(i + 2);             // over the P just read: products run in the order they are issued
            }
            if (ok) umma_commit(&bars->o_full);
            else *abort_flag = 1;
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------ softmax and output: one thread per query row and group
        const uint32_t quarter = warp & 3, t = (warp - 4) >> 2;
        // query row of the tile = TMEM lane = quarter * 32 + lane
        const uint32_t ts = tmem + ((quarter * 32) << 16) + t * 128, to = ts + 256;
        const uint16_t* mask = A.mask ? A.mask + (size_t)head * A.mask_head_stride : nullptr;
        const uint16_t* mask_end = mask + (size_t)A.seq_q * A.seq_k;
        uint4* mbuf = (uint4*)sM + (t * 4 + quarter) * 512;    // this warp's rows of a mask tile
        const float rscale = A.scale_div ? 1.0f / A.scale : A.scale;   // s * (1 / scale): within an fp32 step of s / scale before the fp16 rounding
        const uint32_t rscale2 = pack_h2(rscale, rscale);
        const float LOG2E = 1.4426950408889634f;
        float m = -INFINITY;                                   // in powers of two
        float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        bool ok = true;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        unsigned long long rest = live;
        for (uint32_t i = 0; i < n_live; i++) {
            const uint32_t kt = (uint32_t)__ffsll((long long)rest) - 1;
            rest &= rest - 1;
            if ((i & 1) != t) continue;
            // a tile whose mask is +0 everywhere and that lies inside the sequence needs no mask values
            const bool masked = !((!mask || ((zero_tiles >> kt) & 1ull)) && (kt + 1) * BKV <= A.seq_k);
            if (masked) mask_tile(mask, mask_end, q0 + quarter * 32, A.seq_q, kt * BKV, A.seq_k, mbuf);
            ok = !__any_sync(0xffffffffu, *abort_flag != 0) && __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->s_full[t], (i >> 1) & 1, abort_flag));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // scores, two to a word, over the columns already read (64 words: where P goes), and their maximum
            __half2 mx[4] = {as_h2(0xFC00FC00u), as_h2(0xFC00FC00u), as_h2(0xFC00FC00u), as_h2(0xFC00FC00u)};
#pragma unroll 1
            for (uint32_t c = 0; c < 2; c++) {
                uint32_t va[32], vb[32], h[32];
                tmem_ld32(ts + c * 64, va);
                tmem_ld_wait(va);
                tmem_ld32(ts + c * 64 + 32, vb);
                scores32<HALF_SCALE>(va, h, masked, mbuf, lane, c * 8, rscale, rscale2);
                tmem_ld_wait(vb);
                scores32<HALF_SCALE>(vb, h + 16, masked, mbuf, lane, c * 8 + 4, rscale, rscale2);
                tmem_st32(ts + c * 32, h);
#pragma unroll
                for (int e = 0; e < 32; e++) mx[e & 3] = __hmax2(mx[e & 3], as_h2(h[e]));
            }
            mx[0] = __hmax2(__hmax2(mx[0], mx[1]), __hmax2(mx[2], mx[3]));
            const float mt = fmaxf(__low2float(mx[0]), __high2float(mx[0])) * LOG2E;
            tmem_st_wait();
            // s_full of this tile came after this group's products of the tile before: its O is at rest
            const bool raise = mt > m + RAISE;
            if (__any_sync(0xffffffffu, raise)) {
                const float f = raise ? (m == -INFINITY ? 0.0f : ex2(m - mt)) : 1.0f;
                if (raise) m = mt;
#pragma unroll
                for (int c = 0; c < 2; c++) { l2[c].x *= f; l2[c].y *= f; }
                if (i > 1) {
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        uint32_t v[32];
                        tmem_ld32(to + c * 32, v);
                        tmem_ld_wait(v);
#pragma unroll
                        for (int e = 0; e < 32; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) * f);
                        tmem_st32(to + c * 32, v);
                    }
                    tmem_st_wait();
                }
            }
            const float off = m == -INFINITY ? 0.0f : -m;        // a row that has seen no live position yet: zeros
#pragma unroll 1
            for (uint32_t c = 0; c < 2; c++) {
                uint32_t h[32];
                tmem_ld32(ts + c * 32, h);
                tmem_ld_wait(h);
#pragma unroll
                for (int e = 0; e < 32; e++) {
                    const float2 x = fma2(unpack_h2(h[e]), make_float2(LOG2E, LOG2E), make_float2(off, off));
                    const float2 p = make_float2(ex2(x.x), ex2(x.y));
                    l2[e & 1] = add2(l2[e & 1], p);
                    h[e] = pack_h2(p.x, p.y);
                }
                tmem_st32(ts + c * 32, h);
            }
            tmem_st_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_full[t]);
        }
        // ---- the two groups' halves together: every thread takes head_dim columns 64 t .. +63 of its row out of both
        if (ok) {
            __syncwarp();                                       // the warp's mask values have been read
            ((float2*)mbuf)[lane] = make_float2(m, (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y));      // row maximum and sum, for the other group
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->merge);
            ok = __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->merge, 0, abort_flag));
        }
        if (ok && n_live) ok = __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->o_full, 0, abort_flag));
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float2 ml0 = ((const float2*)((const uint4*)sM + quarter * 512))[lane], ml1 = ((const float2*)((const uint4*)sM + (4 + quarter) * 512))[lane];
            const float M = fmaxf(ml0.x, ml1.x);
            float f0 = ml0.x == -INFINITY ? 0.0f : ex2(ml0.x - M), f1 = ml1.x == -INFINITY ? 0.0f : ex2(ml1.x - M);
            const float l = ml0.y * f0 + ml1.y * f1;
            const float inv = l == 0.0f ? 0.0f : 1.0f / l;       // a sum that is no number makes no number of the row
            f0 *= inv; f1 *= inv;
            const uint32_t ta = tmem + ((quarter * 32) << 16) + 256 + t * 64;
            // the warp's 32 rows of 128 bytes by way of shared memory: 8 lanes to a row, a request touches four (a row to a lane touched
            // 32, 1.2 us). Q has been read by all products.
            uint4* stage = (uint4*)sQ + (t * 4 + quarter) * 256;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[16], u[16];
                tmem_ld16(ta + c * 16, v);
                tmem_ld16(ta + 128 + c * 16, u);
                tmem_ld_wait(v);
                tmem_ld_wait(u);
                const bool two = n_live > 1;                     // a group without a tile has nothing in its O
                float o[16], sum = 0.0f;
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    o[e] = __uint_as_float(v[e]) * f0;
                    if (two) o[e] = fmaf(__uint_as_float(u[e]), f1, o[e]);
                    if (inv == 0.0f) o[e] = 0.0f;                // a row without a live position, whatever values it would have weighed
                    sum += o[e];
                }
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; e++) w[e] = pack_h2(o[2 * e], o[2 * e + 1]);
                if (isnan(sum)) {                                // the reference's conversion of NaN, which the instruction does not know
#pragma unroll
                    for (int e = 0; e < 8; e++) w[e] = (uint32_t)f2h(o[2 * e]) | ((uint32_t)f2h(o[2 * e + 1]) << 16);
                }
#pragma unroll
                for (int q = 0; q < 2; q++) stage[lane * 8 + ((c * 2 + q) ^ (lane & 7))] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
            }
            __syncwarp();
            const uint32_t p = lane & 7;
#pragma unroll 2
            for (uint32_t r = lane >> 3; r < 32; r += 4)
                if (q0 + quarter * 32 + r < A.seq_q)
                    ((uint4*)(A.out + ((size_t)(q0 + quarter * 32 + r) * A.nh + head) * HD + t * 64))[p] = stage[r * 8 + (p ^ (r & 7))];
        }
        if (!ok) *abort_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        if (lane == 0 && *abort_flag) raise_status(A.status, kStatusAttnTimeout);
    }
}

bool make_map(CUtensorMap* tm, const uint16_t* base, uint64_t inner, uint64_t rows, uint64_t row_stride_elems, uint32_t box_rows = 128) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    cuuint64_t dims[2] = {inner, rows};
    cuuint64_t strides[1] = {row_stride_elems * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// false: shape not taken (head_dim other than 128, more than 8192 key positions, unaligned operands, scale <= 0,
// which the general kernel takes); nothing launched.
bool k_attn_prefill_sm100(cudaStream_t st, const uint16_t* q, const uint16_t* k, const uint16_t* v, const uint16_t* mask,
                          size_t mask_head_stride, const uint8_t* skip, const uint8_t* zero, float scale, int scale_div, uint32_t seq_q,
                          uint32_t seq_k, uint32_t nh, uint32_t kvh, uint32_t hd, uint16_t* out, unsigned int* status) {
    if (hd != 128 || !seq_q || !seq_k || seq_k > 64 * BKV || !kvh || nh % kvh) return false;
    if ((((uintptr_t)q) | ((uintptr_t)k) | ((uintptr_t)v) | ((uintptr_t)out)) & 15u) return false;
    if (scale <= 0.0f) return false;
    CUtensorMap tq, tk, tv;
    if (!make_map(&tq, q, (uint64_t)nh * hd, seq_q, (uint64_t)nh * hd) || !make_map(&tk, k, (uint64_t)kvh * hd, seq_k, (uint64_t)kvh * hd) ||
        !make_map(&tv, v, (uint64_t)kvh * hd, seq_k, (uint64_t)kvh * hd, 64))
        return false;
    const size_t smem = 1024 + 14 * (size_t)TILE_BYTES + sizeof(ABars) + 16;
    const float rscale = scale_div ? 1.0f / scale : scale;
    const bool half_scale = __half2float(__float2half_rn(rscale)) == rscale;
    static int have[2][64] = {};
    auto kernel = half_scale ? attn_prefill_sm100_kernel<true> : attn_prefill_sm100_kernel<false>;
    if (!ensure_dyn_smem(kernel, smem, have[half_scale])) return false;
    SmArgs a{mask, mask_head_stride, skip, zero, out, seq_q, seq_k, nh, kvh, scale, scale_div, status};
    if (launch_pdl(kernel, dim3(nh, (seq_q + BQ - 1) / BQ), dim3(NTHREADS), smem, st, tq, tk, tv, a) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g_launches++;
    return true;
}

}  // namespace gehtp
