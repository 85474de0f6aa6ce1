// Pieces of the chunked gated delta rule that its kernels share (gdn_delta_mma.cu: one chunk per launch, gdn_scan.cu: the
// chunks of a sequence in two launches): decays, the triangular matrix and its inverse, the decayed q.k matrix.
#pragma once
#include "common.cuh"
#include "w4_stream.cuh"

namespace gehtp {
namespace gdn {

constexpr int C = 64;          // chunk rows (shorter chunks are padded with zero rows)
constexpr int CP = C + 8;      // row stride (halves) of [..][C] operands: rows fall on different banks

// acc += A[16 x K] . Bt[8 x K]^T ; A, Bt row-major fp16 in shared memory with K contiguous
__device__ __forceinline__ void mma_rows(float (&acc)[4], const uint16_t* A, int lda, const uint16_t* Bt, int ldb, int K, int g, int t) {
    const uint16_t* a_lo = A + g * lda + 2 * t;
    const uint16_t* a_hi = A + (g + 8) * lda + 2 * t;
    const uint16_t* b = Bt + g * ldb + 2 * t;
#pragma unroll 4
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4];
        a[0] = *(const uint32_t*)(a_lo + k0);
        a[1] = *(const uint32_t*)(a_hi + k0);
        a[2] = *(const uint32_t*)(a_lo + k0 + 8);
        a[3] = *(const uint32_t*)(a_hi + k0 + 8);
        mma16816(acc, a, *(const uint32_t*)(b + k0), *(const uint32_t*)(b + k0 + 8));
    }
}

__device__ __forceinline__ void split_store(uint16_t* hi, uint16_t* lo, float x) {
    const uint16_t h = f2h(x);
    *hi = h;
    *lo = f2h(x - h2f(h));
}

// The decays of a chunk of c tokens, by one warp: G the running sum of the log decays, eG = exp(G), wd = exp(G_last - G_i),
// bj the step sizes; zeros past c.
__device__ __forceinline__ void chunk_decays(const uint16_t* gh, const uint16_t* bh, int c, int lane, float* G, float* bj, float* eG, float* wd) {
    // running sum of g over the chunk, in token order (a warp scan would add in another order): every lane
    // adds the 64 values up itself, from registers, and keeps the two sums that are its own
    for (int i = lane; i < C; i += 32) wd[i] = i < c ? h2f(gh[i]) : 0.0f;      // wd as scratch for the raw values
    __syncwarp();
    float acc = 0.0f, mine0 = 0.0f, mine1 = 0.0f, last = 0.0f;
#pragma unroll
    for (int i = 0; i < C; i++) {
        acc += wd[i];
        if (i == lane) mine0 = acc;
        if (i == lane + 32) mine1 = acc;
        if (i == c - 1) last = acc;
    }
    __syncwarp();
    G[lane] = mine0; G[lane + 32] = mine1;
    eG[lane] = expf(mine0); eG[lane + 32] = expf(mine1);
    wd[lane] = expf(last - mine0); wd[lane + 32] = expf(last - mine1);
    for (int i = lane; i < C; i += 32) bj[i] = i < c ? h2f(bh[i]) : 0.0f;
}

// T = (I + L)^-1 (Th, and transposed Tt) and the decayed q.k matrix (hi, lo) of one chunk, by 256 threads. Shared memory:
// Kh, Qh [C][D + 8], Lh, Th, Tt [C][CP], xs [3][768]; Th, Tt and xs may lie on Kh and Qh, which are read up to the first
// barrier. Two neighbouring values of the q.k matrix, packed, go to put_qk(row, column, hi, lo). `stage3` is run beside the
// first products, before the first barrier; the matrices are complete when the function returns (the last barrier is behind them).
template <int D, class Stage3, class PutQK>
__device__ __forceinline__ void chunk_matrices(const uint16_t* Kh, const uint16_t* Qh, uint16_t* Lh, uint16_t* Th, uint16_t* Tt, uint16_t* xs,
                                               const float* G, const float* bj, float scale, Stage3 stage3, PutQK put_qk) {
    constexpr int DP = D + 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // ---- stage 1 (with 3 and 5 below): L[j][i] = f16(exp(G_j - G_i) (k_j . k_i) beta_j) for i < j, else 0
    // Only the 20 tiles of 16 x 8 that touch the lower triangle carry values (row block mi has 2 mi + 2 of them);
    // they are numbered 0..19 and dealt out to the warps in turn, the other 12 are zero and filled apart.
    auto lower_tile = [](int idx, int& mi, int& ni) { mi = idx < 2 ? 0 : idx < 6 ? 1 : idx < 12 ? 2 : 3; ni = idx - (mi * mi + mi); };
    constexpr int LOWER = 20;
    static_assert(C == 64, "the tile numbering above is that of a 64-row chunk");
    for (int idx = warp; idx < LOWER; idx += 8) {
        int mi, ni;
        lower_tile(idx, mi, ni);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_rows(acc, Kh + mi * 16 * DP, DP, Kh + ni * 8 * DP, DP, D, g, t);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int j = mi * 16 + g + (e >> 1) * 8, i = ni * 8 + 2 * t + (e & 1);
            Lh[j * CP + i] = i < j ? f2h(expf(G[j] - G[i]) * acc[e] * bj[j]) : (uint16_t)0;
        }
    }
    for (int e = tid; e < C * C / 2; e += 256) {      // the tiles above: L = 0, QK = 0
        const int r = e / (C / 2), i = e % (C / 2) * 2;
        if (i >= ((r >> 4) + 1) * 16) { *(uint32_t*)(Lh + r * CP + i) = 0; put_qk(r, i, 0u, 0u); }
    }
    // stages 3 and 5 need the operands only, not L or T: same phase, one barrier for the three
    stage3();
    // ---- stage 5: QK[t][i] = exp(G_t - G_i) (q_t . k_i) for i <= t, as hi + lo
    for (int idx = 7 - warp; idx < LOWER; idx += 8) {     // dealt out from the other end: a warp with 3 tiles of L gets 2 here
        int mi, ni;
        lower_tile(idx, mi, ni);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_rows(acc, Qh + mi * 16 * DP, DP, Kh + ni * 8 * DP, DP, D, g, t);
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int tt = mi * 16 + g + (e >> 1) * 8, i = ni * 8 + 2 * t;
            uint32_t hi = 0, lo = 0;
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const float x = i + b <= tt ? acc[e + b] * scale * expf(G[tt] - G[i + b]) : 0.0f;
                const uint16_t h = f2h(x);
                hi |= (uint32_t)h << (16 * b);
                lo |= (uint32_t)f2h(x - h2f(h)) << (16 * b);
            }
            put_qk(tt, i, hi, lo);
        }
    }
    __syncthreads();

    // ---- stage 2: T = (I + L)^-1 in fp16. Within a 16 x 16 diagonal block it is the forward substitution of the
    // reference, row by row with every entry rounded to fp16 before the next row uses it; column j depends on column j
    // only, so one lane owns a column and runs down the 16 rows (all four diagonal blocks at once, no block-wide
    // barrier). The blocks below the diagonal follow from (I + L) T = I block row by block row:
    //     T_ik = -T_ii (sum_{k <= m < i} L_im T_mk)
    // two small products per block on the tensor cores (the inner sum as hi + lo), rounded to fp16 once.
    {
        // One lane per column (64 lanes, two warps): the sum over i < r runs in i order, as the reference's
        // solve_tri_f16 forms it, with the column's earlier entries in registers; the entries of L of a row are the
        // same for all 16 columns of a block (broadcast reads that depend on nothing before them).
        if (tid < C) {
            const int j = tid, r0 = j & ~15, jl = j & 15;
            float tc[16];
#pragma unroll
            for (int rr = 0; rr < 16; rr++) {
                float s = 0.0f;
#pragma unroll
                for (int il = 0; il < rr; il++) {
                    const float l = h2f(Lh[(r0 + rr) * CP + r0 + il]);
                    if (il >= jl) s -= l * tc[il];
                }
                const uint16_t tv = jl <= rr ? f2h((rr == jl ? 1.0f : 0.0f) + s) : (uint16_t)0;
                Th[(r0 + rr) * CP + j] = tv;
                Tt[j * CP + r0 + rr] = tv;
                tc[rr] = h2f(tv);
            }
        }
        for (int e = tid; e < C * C; e += 256) {     // blocks above the block diagonal
            const int r = e / C, jj = e % C;
            if ((jj >> 4) > (r >> 4)) Th[r * CP + jj] = 0;
        }
    }
    __syncthreads();
    for (int bi = 1; bi < C / 16; bi++) {
        if (warp < bi) {
            const int bk = warp;
            uint16_t* xhi = xs + warp * 768;        // X transposed [16][24], hi and lo
            uint16_t* xlo = xhi + 384;
            for (int nt = 0; nt < 2; nt++) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                mma_rows(acc, Lh + bi * 16 * CP + bk * 16, CP, Tt + (bk * 16 + nt * 8) * CP + bk * 16, CP, 16 * (bi - bk), g, t);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int row = g + (e >> 1) * 8, n = nt * 8 + 2 * t + (e & 1);
                    split_store(xhi + n * 24 + row, xlo + n * 24 + row, acc[e]);
                }
            }
            __syncwarp();
            for (int nt = 0; nt < 2; nt++) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                mma_rows(acc, Th + bi * 16 * CP + bi * 16, CP, xhi + nt * 8 * 24, 24, 16, g, t);
                mma_rows(acc, Th + bi * 16 * CP + bi * 16, CP, xlo + nt * 8 * 24, 24, 16, g, t);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int row = bi * 16 + g + (e >> 1) * 8, col = bk * 16 + nt * 8 + 2 * t + (e & 1);
                    const uint16_t tv = f2h(-acc[e]);
                    Th[row * CP + col] = tv;
                    Tt[col * CP + row] = tv;
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace gdn
}  // namespace gehtp
