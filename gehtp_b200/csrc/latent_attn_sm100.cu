// Latent attention over many rows on tcgen05 / TMEM (bf16; keys of 128 + 64 rotated values, values of 128), behind the
// projection that expands keys and values of every cached position (latent_prefill.cu).
//
// One CTA = 128 query rows of a head; key / value tiles of 128 positions in turn to two groups of four softmax warps, each with
// its own S, O, row maximum and row sum; the halves of the result are added at the end (as attn_prefill_sm100.cu). The rotated
// part of the keys is read from the state rows that all heads share.
//   S = Q K^T   three boxes of 64 values, into TMEM
//   P           fp32 scores, one thread per row; 2^(s - m) as hi + lo bf16 over S (as window_attn_sm100.cu)
//   O += P V    P as the A operand from TMEM, V as it lies in memory
// Hidden keys have weight 0, which a value that is no number turns into one. A row whose result is no number although the tiles held
// keys it does not see is worked out once more over its own keys alone.
// 2048 tokens of 16 heads: 36 us a layer, 146 with mma.sync products; 1500 tokens of 32 heads 46, 140; 64 tokens 7.9, 10.9.
// Every mbarrier wait is bounded; on a timeout the CTA raises the engine's status word and winds down.
#include <cuda.h>
#include <cuda_runtime.h>
#include "launchers_rows.h"
#include "sm100_attn.cuh"

namespace gehtp {

using namespace sm100;

namespace {

constexpr uint32_t BQ = 128, BKV = 128, DIM = 128, ROT = 64, VD = 128, BOX = 64 * 64 * 2;      // bytes of a box of 64 rows x 64 values
constexpr uint32_t KB = (DIM + ROT) / 64, K_BYTES = KB * 2 * BOX, V_BYTES = 4 * BOX;
constexpr int NTHREADS = 384;
constexpr float RAISE = 8.0f;

struct __align__(8) LBars {
    uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_full, merge;
    uint32_t tmem_base, abort_flag;
    float2 ml[2][BQ];                                           // row maximum and sum of the two groups
};

// Values 64 t .. + 63 of a row's result, two a lane, over the keys up to its position alone: a key per lane for the scores, a warp per
// key for the values. Rows beside a value that is no number come here, no others.
__device__ __noinline__ float2 row_alone(const LatentArgs& A, const uint16_t* kv, uint32_t h, uint32_t row, uint32_t pos, uint32_t t, float sc) {
    const uint32_t lane = threadIdx.x & 31;
    const size_t kw = (size_t)A.heads * (DIM + VD), ls = A.ls();
    const uint4* q = (const uint4*)((const uint16_t*)A.q + ((size_t)row * A.heads + h) * (DIM + ROT));
    const uint16_t* rot = (const uint16_t*)A.state + A.rank;
    const uint16_t* val = kv + (size_t)A.heads * DIM + h * VD + t * 64 + 2 * lane;
    auto dot = [](float s, uint4 x, uint4 y) {
        const uint32_t a[4] = {x.x, x.y, x.z, x.w}, b[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
            s = fmaf(__uint_as_float(a[i] & 0xffff0000u), __uint_as_float(b[i] & 0xffff0000u), fmaf(__uint_as_float(a[i] << 16), __uint_as_float(b[i] << 16), s));
        return s;
    };
    float m = -INFINITY, l = 0.0f;
    float2 o = make_float2(0.f, 0.f);
#pragma unroll 1
    for (uint32_t j0 = 0; j0 <= pos; j0 += 32) {
        const uint32_t j = j0 + lane, n = min(32u, pos - j0 + 1);
        float s = 0.0f;
        if (lane < n) {
            const uint4 *k = (const uint4*)(kv + j * kw + h * DIM), *r = (const uint4*)(rot + j * ls);
#pragma unroll 4
            for (uint32_t i = 0; i < DIM / 8; i++) s = dot(s, __ldcg(q + i), __ldcg(k + i));
#pragma unroll 4
            for (uint32_t i = 0; i < ROT / 8; i++) s = dot(s, __ldcg(q + DIM / 8 + i), __ldcg(r + i));
        }
        s = lane < n ? s * sc : -INFINITY;
        const float mx = fmaxf(m, warp_max(s)), off = mx == -INFINITY ? 0.0f : mx, f = ex2(m - off), p = ex2(s - off);
        m = mx;
        l = l * f + p;
        o.x *= f; o.y *= f;
#pragma unroll 1
        for (uint32_t i = 0; i < n; i++) {
            const float w = __shfl_sync(0xffffffffu, p, i);
            const uint32_t v = __ldcg((const uint32_t*)(val + (j0 + i) * kw));
            o.x = fmaf(w, __uint_as_float(v << 16), o.x);
            o.y = fmaf(w, __uint_as_float(v & 0xffff0000u), o.y);
        }
    }
    const float f = A.gate[(size_t)row * A.heads + h] / warp_sum(l);
    return make_float2(o.x * f, o.y * f);
}

__global__ void __launch_bounds__(NTHREADS, 1)
latent_attn_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv, const __grid_constant__ CUtensorMap tmap_rot,
                         const __grid_constant__ LatentArgs A, const uint16_t* kv, uint32_t rows, uint32_t past) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sQ = smem;                                    // at the end the rows on their way out
    unsigned char* sK = sQ + K_BYTES;                            // a buffer per group
    unsigned char* sV = sK + 2 * K_BYTES;                        // a buffer per group: [position half][64 values][64 positions x 128 bytes]
    LBars* bars = (LBars*)(sV + 2 * V_BYTES);
    volatile uint32_t* abort_flag = &bars->abort_flag;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t h = blockIdx.x, q0 = (gridDim.y - 1 - blockIdx.y) * BQ;      // the longest rows of all heads first
    const uint32_t n_kt = (min(past + q0 + BQ, past + rows) + BKV - 1) / BKV;

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
        for (const CUtensorMap* map : {&tmap_q, &tmap_kv, &tmap_rot}) asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars->tmem_base;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            mbar_expect_tx(&bars->q_full, K_BYTES);
#pragma unroll 1
            for (uint32_t b = 0; b < 2 * KB; b++)
                tma_load_2d(sQ + b * BOX, &tmap_q, (int)(h * (DIM + ROT) + (b >> 1) * 64), (int)(q0 + (b & 1) * 64), &bars->q_full);
            uint32_t kn = 0, vn = 0;                             // tiles requested
            while (vn < n_kt && !*abort_flag) {
                const uint32_t i0 = vn, n = min(2u, n_kt - i0);
                for (uint32_t t = 0; t < n; t++) {
                    const int y = (int)((i0 + t) * BKV);
                    if (!mbar_wait_or_abort(&bars->k_empty[t], ((i0 >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; break; }
                    mbar_expect_tx(&bars->k_full[t], K_BYTES);
#pragma unroll 1
                    for (uint32_t b = 0; b < 2 * KB; b++) {
                        const uint32_t d = b >> 1;
                        tma_load_2d(sK + t * K_BYTES + b * BOX, d < DIM / 64 ? &tmap_kv : &tmap_rot, (int)(d < DIM / 64 ? h * DIM + d * 64 : A.rank), y + (int)(b & 1) * 64, &bars->k_full[t]);
                    }
                    kn++;
                }
                for (uint32_t t = 0; t < n && !*abort_flag; t++) {
                    const int y = (int)((i0 + t) * BKV);
                    if (!mbar_wait_or_abort(&bars->v_empty[t], ((i0 >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; break; }
                    mbar_expect_tx(&bars->v_full[t], V_BYTES);
#pragma unroll 1
                    for (uint32_t b = 0; b < 4; b++)
                        tma_load_2d(sV + t * V_BYTES + b * BOX, &tmap_kv, (int)(A.heads * DIM + h * VD + (b & 1) * 64), y + (int)(b >> 1) * 64, &bars->v_full[t]);
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
        if (lane == 0) {
            const uint32_t q_base = smem_u32(sQ), k_base = smem_u32(sK), v_base = smem_u32(sV);
            bool ok = true;
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok) ok = mbar_wait_or_abort(bar, parity, abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return ok;
            };
            auto issue_s = [&](uint32_t i) {
                const uint32_t t = i & 1;
                if (!wait(&bars->k_full[t], (i >> 1) & 1)) return;
#pragma unroll
                for (uint32_t d = 0; d < KB; d++)
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; k4++)
                        umma_f16(tmem + t * 128, umma_desc(q_base + d * 2 * BOX) + (uint64_t)(k4 * 2),
                                 umma_desc(k_base + t * K_BYTES + d * 2 * BOX) + (uint64_t)(k4 * 2), idesc_f16(128) | IDESC_BF16, (d | k4) ? 1u : 0u);
                umma_commit(&bars->k_empty[t]);
                umma_commit(&bars->s_full[t]);
            };
            if (wait(&bars->q_full, 0)) {
                issue_s(0);
                if (n_kt > 1) issue_s(1);
            }
            for (uint32_t i = 0; ok && i < n_kt; i++) {
                const uint32_t t = i & 1, ph = (i >> 1) & 1;
                if (!wait(&bars->v_full[t], ph) || !wait(&bars->p_full[t], ph)) break;
#pragma unroll
                for (uint32_t part = 0; part < 2; part++)
#pragma unroll
                    for (uint32_t k = 0; k < 8; k++)             // 16 positions = two 8-position groups = 2048 bytes per step
                        umma_f16_ta(tmem + 256 + t * 128, tmem + t * 128 + (k >> 1) * 32 + part * 16 + (k & 1) * 8,
                                    umma_desc_v(v_base + t * V_BYTES + (k >> 2) * (2 * BOX) + (k & 3) * 2048), idesc_f16(VD) | IDESC_BF16 | (1u << 16), (i > 1 || part || k) ? 1u : 0u);
                umma_commit(&bars->v_empty[t]);
                if (i + 2 < n_kt) issue_s(i + 2);                // over the P just read: products run in the order they are issued
            }
            if (ok) umma_commit(&bars->o_full);
            else *abort_flag = 1;
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------ softmax and output: one thread per query row and group
        const uint32_t quarter = warp & 3, t = (warp - 4) >> 2;
        const uint32_t row = q0 + quarter * 32 + lane, pos = past + row, w_first = pos - lane;
        const uint32_t ts = tmem + ((quarter * 32) << 16) + t * 128, to = ts + 256;
        const float sc = A.scale * 1.44269504088896340736f;      // scores in powers of two
        float m = -INFINITY;
        float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        bool ok = true;
        asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
        for (uint32_t i = t; i < n_kt; i += 2) {
            ok = !__any_sync(0xffffffffu, *abort_flag != 0) && __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->s_full[t], (i >> 1) & 1, abort_flag));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool edge = i * BKV + BKV - 1 > w_first;       // some key of the tile is hidden from some row
            const int hi = (int)pos - (int)(i * BKV);            // columns up to hi are visible to this row
            float mt = -INFINITY;
#pragma unroll 1
            for (int c = 0; c < 2; c++) {
                uint32_t va[32], vb[32];
                tmem_ld32(ts + c * 64, va);
                tmem_ld32(ts + c * 64 + 32, vb);
                tmem_ld_wait(va);
                tmem_ld_wait(vb);
                if (edge) mt = fmaxf(mt, fmaxf(max32<true>(va, visible32(c * 64, 0, hi)), max32<true>(vb, visible32(c * 64 + 32, 0, hi))));
                else mt = fmaxf(mt, fmaxf(max32<false>(va, 0u), max32<false>(vb, 0u)));
            }
            mt *= sc;
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
            const float off = m == -INFINITY ? 0.0f : -m;        // a row that has seen no key of this group yet: zeros
#pragma unroll 1
            for (int c = 0; c < 2; c++) {
                uint32_t va[32], vb[32], w[32];
                tmem_ld32(ts + c * 64, va);
                tmem_ld_wait(va);
                tmem_ld32(ts + c * 64 + 32, vb);
                if (edge) probs32<true>(va, w, sc, off, visible32(c * 64, 0, hi), l2);
                else probs32<false>(va, w, sc, off, 0u, l2);
                tmem_st32(ts + c * 64, w);
                tmem_ld_wait(vb);
                if (edge) probs32<true>(vb, w, sc, off, visible32(c * 64 + 32, 0, hi), l2);
                else probs32<false>(vb, w, sc, off, 0u, l2);
                tmem_st32(ts + c * 64 + 32, w);
            }
            tmem_st_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_full[t]);
        }
        // ---- the two groups' halves together: every thread takes values 64 t .. +63 of its row out of both
        const float gate = row < rows ? A.gate[(size_t)row * A.heads + h] : 0.0f;
        if (ok) {
            bars->ml[t][quarter * 32 + lane] = make_float2(m, (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y));
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->merge);
            ok = __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->merge, 0, abort_flag));
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait_or_abort(&bars->o_full, 0, abort_flag));
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float2 ml0 = bars->ml[0][quarter * 32 + lane], ml1 = bars->ml[1][quarter * 32 + lane];
            const float M = fmaxf(ml0.x, ml1.x);
            float f0 = ex2(ml0.x - M), f1 = ml1.x == -INFINITY ? 0.0f : ex2(ml1.x - M);       // key 0 is visible to every row
            const float f = gate / (ml0.y * f0 + ml1.y * f1);
            f0 *= f; f1 *= f;
            const uint32_t ta = tmem + ((quarter * 32) << 16) + 256 + t * 64;
            uint4* stage = (uint4*)sQ + (t * 4 + quarter) * 256;     // Q has been read by all products
            float sum = 0.0f;                                        // no number if one of the row's values is none
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[16], u[16], w[8];
                tmem_ld16(ta + c * 16, v);
                tmem_ld16(ta + 128 + c * 16, u);
                tmem_ld_wait(v);
                tmem_ld_wait(u);
                const bool two = n_kt > 1;                           // a group without a tile has nothing in its O
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    float x = __uint_as_float(v[2 * e]) * f0, y = __uint_as_float(v[2 * e + 1]) * f0;
                    if (two) { x = fmaf(__uint_as_float(u[2 * e]), f1, x); y = fmaf(__uint_as_float(u[2 * e + 1]), f1, y); }
                    sum += (x - x) + (y - y);
                    w[e] = pack_bf2(x, y);
                }
#pragma unroll
                for (int q = 0; q < 2; q++) stage[lane * 8 + ((c * 2 + q) ^ (lane & 7))] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
            }
            __syncwarp();
            for (uint32_t bad = __ballot_sync(0xffffffffu, sum != 0.0f && row < rows && pos + 1 < min(n_kt * BKV, past + rows)); bad; bad &= bad - 1) {
                const uint32_t r = __ffs(bad) - 1;
                const float2 x = row_alone(A, kv, h, row - lane + r, pos - lane + r, t, sc);
                ((uint32_t*)(stage + r * 8 + ((lane >> 2) ^ (r & 7))))[lane & 3] = pack_bf2(x.x, x.y);
                __syncwarp();
            }
            const uint32_t p = lane & 7;
#pragma unroll 2
            for (uint32_t r = lane >> 3; r < 32; r += 4)
                if (q0 + quarter * 32 + r < rows)
                    ((uint4*)((uint16_t*)A.out + ((size_t)(q0 + quarter * 32 + r) * A.heads + h) * VD + t * 64))[p] = stage[r * 8 + (p ^ (r & 7))];
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

bool make_map(CUtensorMap* tm, const void* base, uint64_t inner, uint64_t rows, uint64_t row_elems) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    cuuint64_t dims[2] = {inner, rows};
    cuuint64_t strides[1] = {row_elems * 2};
    cuuint32_t box[2] = {64, 64};
    cuuint32_t estr[2] = {1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// kv: expanded keys and values of positions [0, past + rows). false: sizes or alignment not taken, nothing launched
bool k_latent_sm100(cudaStream_t st, const LatentArgs& a, const uint16_t* kv, uint32_t rows, uint32_t past) {
    if (!a.bf16 || !rows || a.dim != DIM || a.rot != ROT || a.vdim != VD || a.rank % 8 || a.scale <= 0.0f) return false;
    if (((uintptr_t)a.q | (uintptr_t)a.state | (uintptr_t)a.out | (uintptr_t)kv) & 15u) return false;
    CUtensorMap tq, tkv, trot;
    const uint64_t n = past + rows, qw = (uint64_t)a.heads * (DIM + ROT), kw = (uint64_t)a.heads * (DIM + VD);
    if (!make_map(&tq, a.q, qw, rows, qw) || !make_map(&tkv, kv, kw, n, kw) || !make_map(&trot, a.state, a.ls(), n, a.ls())) return false;
    const size_t smem = 1024 + 3 * (size_t)K_BYTES + 2 * (size_t)V_BYTES + sizeof(LBars) + 16;
    static int have[64] = {};
    if (!ensure_dyn_smem(latent_attn_sm100_kernel, smem, have)) return false;
    if (launch_pdl(latent_attn_sm100_kernel, dim3(a.heads, (rows + BQ - 1) / BQ), dim3(NTHREADS), smem, st, tq, tkv, trot, a, kv, rows, past) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g_launches++;
    return true;
}

}  // namespace gehtp
