// The chunked gated delta rule over the chunks of a sequence, two launches for all of them (mma.sync m16n8k16, fp32
// accumulation, operands and roundings as in gdn_delta_mma.cu).
//
// Of a chunk's seven products only four touch the state: b = beta (v - e^G S k), u = T b, y and the new S. What does not -
// decays, T = (I + L)^-1 and the decayed q.k matrix - is made for all chunks side by side first:
//   delta_chunks_kernel  grid (head, chunk): T, q.k hi and lo (fp16) and the decays of one chunk into scratch
//   delta_scan_mma_kernel grid (head, 16 rows of S): walks the chunks with its rows of S in registers (fp32) and, as hi + lo
//                        fp16 operands, in shared memory; the next chunk's k, q, v, T and q.k come in by cp.async meanwhile
// One launch per chunk is bound by the chain of all seven stages (15 us, 32 times in 2048 tokens); the walk's own chain is
// three barriers a chunk. Its products are read from shared memory: k, q and S fragments are taken once for the two
// products and the hi and lo halves that use them.
#include <algorithm>
#include "gdn_delta.cuh"
#include "launchers.h"

namespace gehtp {

using namespace gdn;

namespace {

constexpr int DM = 16;                              // rows of S per CTA of the walk
constexpr int VP = DM + 8;
// scratch of one (head, chunk): T, q.k hi, q.k lo [C][C] fp16, then bj, eG, wd [C] fp32
constexpr size_t MAT = (size_t)C * C, ITEM_BYTES = 3 * MAT * 2 + 3 * C * 4;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int D>
__global__ void __launch_bounds__(256)
delta_chunks_kernel(const DeltaChunk* __restrict__ chunks, unsigned char* scratch, int ntok, int q_raw) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int DP = D + 8, STEPS = C * (D / 8) / 256;
    extern __shared__ __align__(16) unsigned char smem[];
    uint16_t* Kh = (uint16_t*)smem;                 // [C][DP]
    uint16_t* Qh = Kh + C * DP;
    uint16_t* Lh = Qh + C * DP;                     // [C][CP]
    uint16_t* xs = Lh + C * CP;                     // [3][768]
    // T over k and q, which have been read by then; q.k goes straight to scratch. Four CTAs fit an SM, and the 512 of 2048 tokens
    // and 16 heads are one round (19.1 us); with every matrix in a place of its own they were two (27.7).
    uint16_t *Th = Kh, *Tt = Th + C * CP;           // [C][CP] each
    float* G = (float*)(xs + 3 * 768);
    float* vec = G + C;                             // bj, eG, wd
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const DeltaChunk ck = chunks[blockIdx.y];
    const size_t off = (size_t)h * ntok * D;
#pragma unroll
    for (int u = 0; u < STEPS; u++) {
        const int e = tid + u * 256, r = e / (D / 8), n8 = (e % (D / 8)) * 8;
        cp_async16(Kh + r * DP + n8, ck.k + off + (size_t)r * D + n8);
        cp_async16(Qh + r * DP + n8, ck.q + off + (size_t)r * D + n8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (warp == 0) chunk_decays(ck.g + (size_t)h * ntok, ck.beta + (size_t)h * ntok, C, lane, G, vec, vec + C, vec + 2 * C);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    unsigned char* item = scratch + ((size_t)h * gridDim.y + blockIdx.y) * ITEM_BYTES;
    chunk_matrices<D>(Kh, Qh, Lh, Th, Tt, xs, G, vec, q_raw ? 1.0f : 1.0f / sqrtf((float)D), [] {}, [&](int r, int i, uint32_t hi, uint32_t lo) {
        uint32_t* at = (uint32_t*)(item + MAT * 2 + (r * C + i) * 2);
        at[0] = hi;
        at[MAT / 2] = lo;
    });
    for (int e = tid; e < C * C / 8; e += 256) *(uint4*)(item + (size_t)e * 16) = *(const uint4*)(Th + (e >> 3) * CP + (e & 7) * 8);
    if (tid < 3 * C) ((float*)(item + 3 * MAT * 2))[tid] = vec[tid];
}

__device__ __forceinline__ uint32_t smem_of(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// four 8 x 8 tiles of a row-major operand, one row address per lane
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

template <int D>
struct ScanBuf {
    static constexpr int DP = D + 8;
    uint16_t K[C * DP], Q[C * DP], T[C * CP], QKhi[C * CP], QKlo[C * CP], V[C * VP];
    float vec[3 * C];
};
template <int D>
struct ScanSmem {
    ScanBuf<D> buf[2];
    uint16_t Shi[DM * (D + 8)], Slo[DM * (D + 8)];
    uint16_t bThi[DM * CP], bTlo[DM * CP], uThi[DM * CP], uTlo[DM * CP], wuhi[DM * CP], wulo[DM * CP];
};

template <int D>
__global__ void __launch_bounds__(256, 1)
delta_scan_mma_kernel(const DeltaChunk* __restrict__ chunks, const unsigned char* scratch, float* __restrict__ Sg, int n, int ntok, int q_raw) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr int DP = D + 8, TPW = D / 64;         // 8-column tiles of S per warp
    extern __shared__ __align__(16) unsigned char smem[];
    ScanSmem<D>& sm = *(ScanSmem<D>*)smem;
    const int h = blockIdx.x, m0 = blockIdx.y * DM, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int mi = warp >> 1, ni = warp & 1;        // this warp's 16 tokens x 8 value rows of b, u and y
    const float scale = q_raw ? 1.0f : 1.0f / sqrtf((float)D);
    float* Sglob = Sg + ((size_t)h * D + m0) * D;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // The operands' addresses are read a chunk before they are used: read where they are needed, each chunk waited for them once
    // for its copies and once for its result (32 chunks of 16 heads: 97 -> 91 us).
    DeltaChunk ck = chunks[0];
    uint16_t* y_next = ck.y;
    auto fetch = [&](int ch) {
        ScanBuf<D>& b = sm.buf[ch & 1];
        const size_t off = (size_t)h * ntok * D;
#pragma unroll
        for (int u = 0; u < C * (D / 8) / 256; u++) {
            const int e = tid + u * 256, r = e / (D / 8), n8 = (e % (D / 8)) * 8;
            cp_async16(b.K + r * DP + n8, ck.k + off + (size_t)r * D + n8);
            cp_async16(b.Q + r * DP + n8, ck.q + off + (size_t)r * D + n8);
        }
        const unsigned char* item = scratch + ((size_t)h * n + ch) * ITEM_BYTES;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int e = tid + u * 256, d = (e >> 3) * CP + (e & 7) * 8;
            cp_async16(b.T + d, item + (size_t)e * 16);
            cp_async16(b.QKhi + d, item + MAT * 2 + (size_t)e * 16);
            cp_async16(b.QKlo + d, item + 2 * MAT * 2 + (size_t)e * 16);
        }
        if (tid < 128) cp_async16(b.V + (tid >> 1) * VP + (tid & 1) * 8, ck.v + off + (size_t)(tid >> 1) * D + m0 + (tid & 1) * 8);
        else if (tid < 128 + 3 * C / 4) cp_async16(b.vec + (tid - 128) * 4, item + 3 * MAT * 2 + (size_t)(tid - 128) * 16);
        asm volatile("cp.async.commit_group;" ::: "memory");
        ck = chunks[min(ch + 1, n - 1)];
    };
    fetch(0);
    // this warp's tiles of S: columns (warp + 8 j) * 8 + 2 t, + 1 of rows g and g + 8
    float S[TPW][4];
#pragma unroll
    for (int j = 0; j < TPW; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int m = g + (e >> 1) * 8, c = (warp + 8 * j) * 8 + 2 * t + (e & 1);
            S[j][e] = Sglob[(size_t)m * D + c];
            split_store(sm.Shi + m * DP + c, sm.Slo + m * DP + c, S[j][e]);
        }
    for (int ch = 0; ch < n; ch++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                            // chunk ch and S are in shared memory, the other buffer has been read
        uint16_t* yh = y_next + (size_t)h * ntok * D + m0;
        y_next = ck.y;
        if (ch + 1 < n) fetch(ch + 1);
        const ScanBuf<D>& b = sm.buf[ch & 1];
        const float *bj = b.vec, *eG = b.vec + C, *wd = b.vec + 2 * C;
        // ---- b and the state's part of y: S k and S q, hi and lo apart
        float kh[4] = {}, kl[4] = {}, qh[4] = {}, ql[4] = {};
        {
            // rows of an operand by ldmatrix: 16 rows x 16 columns of k and q, 8 rows x 32 columns of S
            const uint32_t arow = (mi * 16 + (lane & 15)) * DP + (lane >> 4) * 8, brow = (ni * 8 + (lane & 7)) * DP + (lane >> 3) * 8;
            const uint32_t pk = smem_of(b.K + arow), pq = smem_of(b.Q + arow), ph = smem_of(sm.Shi + brow), pl = smem_of(sm.Slo + brow);
#pragma unroll
            for (int k0 = 0; k0 < D; k0 += 32) {
                uint32_t bh[4], bl[4];
                ldsm(bh, ph + k0 * 2);
                ldsm(bl, pl + k0 * 2);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    uint32_t ak[4], aq[4];
                    ldsm(ak, pk + (k0 + 16 * i) * 2);
                    ldsm(aq, pq + (k0 + 16 * i) * 2);
                    mma16816(kh, ak, bh[2 * i], bh[2 * i + 1]);
                    mma16816(kl, ak, bl[2 * i], bl[2 * i + 1]);
                    mma16816(qh, aq, bh[2 * i], bh[2 * i + 1]);
                    mma16816(ql, aq, bl[2 * i], bl[2 * i + 1]);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int j = mi * 16 + g + (e >> 1) * 8, m = ni * 8 + 2 * t + (e & 1);
            split_store(sm.bThi + m * CP + j, sm.bTlo + m * CP + j, bj[j] * (h2f(b.V[j * VP + m]) - eG[j] * (kh[e] + kl[e])));
        }
        __syncthreads();
        // ---- u = T b, also weighted with the decay to the end of the chunk
        float uh[4] = {}, ul[4] = {};
        const uint32_t crow = (mi * 16 + (lane & 15)) * CP + (lane >> 4) * 8, drow = (ni * 8 + (lane & 7)) * CP + (lane >> 3) * 8;
        {
            const uint32_t pt = smem_of(b.T + crow), ph = smem_of(sm.bThi + drow), pl = smem_of(sm.bTlo + drow);
#pragma unroll
            for (int k0 = 0; k0 < C; k0 += 32) {
                uint32_t bh[4], bl[4], a0[4], a1[4];
                ldsm(bh, ph + k0 * 2);
                ldsm(bl, pl + k0 * 2);
                ldsm(a0, pt + k0 * 2);
                ldsm(a1, pt + k0 * 2 + 32);
                mma16816(uh, a0, bh[0], bh[1]);
                mma16816(ul, a0, bl[0], bl[1]);
                mma16816(uh, a1, bh[2], bh[3]);
                mma16816(ul, a1, bl[2], bl[3]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int j = mi * 16 + g + (e >> 1) * 8, m = ni * 8 + 2 * t + (e & 1);
            const float u = uh[e] + ul[e];
            split_store(sm.uThi + m * CP + j, sm.uTlo + m * CP + j, u);
            split_store(sm.wuhi + m * CP + j, sm.wulo + m * CP + j, wd[j] * u);
        }
        __syncthreads();
        // ---- y = e^G S q + QK u
        float y0[4] = {}, y1[4] = {}, y2[4] = {};
        {
            const uint32_t pa = smem_of(b.QKhi + crow), pb = smem_of(b.QKlo + crow), ph = smem_of(sm.uThi + drow), pl = smem_of(sm.uTlo + drow);
#pragma unroll
            for (int k0 = 0; k0 < C; k0 += 32) {
                uint32_t bh[4], bl[4];
                ldsm(bh, ph + k0 * 2);
                ldsm(bl, pl + k0 * 2);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    uint32_t ah[4], al[4];
                    ldsm(ah, pa + (k0 + 16 * i) * 2);
                    ldsm(al, pb + (k0 + 16 * i) * 2);
                    mma16816(y0, ah, bh[2 * i], bh[2 * i + 1]);
                    mma16816(y1, ah, bl[2 * i], bl[2 * i + 1]);
                    mma16816(y2, al, bh[2 * i], bh[2 * i + 1]);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int j = mi * 16 + g + (e >> 1) * 8, m = ni * 8 + 2 * t;
            const float w = eG[j] * scale;
            const uint32_t lo = f2h(w * (qh[e] + ql[e]) + (y0[e] + y1[e] + y2[e])), hi = f2h(w * (qh[e + 1] + ql[e + 1]) + (y0[e + 1] + y1[e + 1] + y2[e + 1]));
            *(uint32_t*)(yh + (size_t)j * D + m) = lo | (hi << 16);
        }
        // ---- S' = e^{G_last} S + (decayed u) k; a column of k over 32 tokens comes transposed out of its rows
        const float eC = eG[C - 1];
        float sh[TPW][4], sl[TPW][4];
#pragma unroll
        for (int j = 0; j < TPW; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) sh[j][e] = sl[j][e] = 0.0f;
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 32) {
            uint32_t a0[4], a1[4], l0[4], l1[4];
            const uint32_t wrow = ((lane & 15) * CP + (lane >> 4) * 8 + k0) * 2;
            ldsm(a0, smem_of(sm.wuhi) + wrow);
            ldsm(a1, smem_of(sm.wuhi) + wrow + 32);
            ldsm(l0, smem_of(sm.wulo) + wrow);
            ldsm(l1, smem_of(sm.wulo) + wrow + 32);
#pragma unroll
            for (int j = 0; j < TPW; j++) {
                uint32_t r[4];
                const uint32_t addr = (uint32_t)__cvta_generic_to_shared(b.K + (k0 + lane) * DP + (warp + 8 * j) * 8);
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
                mma16816(sh[j], a0, r[0], r[1]);
                mma16816(sl[j], l0, r[0], r[1]);
                mma16816(sh[j], a1, r[2], r[3]);
                mma16816(sl[j], l1, r[2], r[3]);
            }
        }
#pragma unroll
        for (int j = 0; j < TPW; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int m = g + (e >> 1) * 8, c = (warp + 8 * j) * 8 + 2 * t + (e & 1);
                S[j][e] = S[j][e] * eC + (sh[j][e] + sl[j][e]);
                split_store(sm.Shi + m * DP + c, sm.Slo + m * DP + c, S[j][e]);      // read last before the two barriers above
            }
    }
#pragma unroll
    for (int j = 0; j < TPW; j++)
#pragma unroll
        for (int e = 0; e < 4; e += 2)
            *(float2*)(Sglob + (size_t)(g + (e >> 1) * 8) * D + (warp + 8 * j) * 8 + 2 * t) = make_float2(S[j][e], S[j][e + 1]);
}

template <int D>
bool launch(cudaStream_t st, const DeltaChunk* chunks, unsigned char* scratch, float* S, uint32_t n, uint32_t ntok, uint32_t H, uint32_t q_raw) {
    static int have_a[64], have_b[64];
    // No more CTAs to an SM than an even spread needs: those that come up while the kernel before still holds SMs would pile up on
    // the ones it has left (256 tokens: 76 us a layer for 70). An SM has 228 KB.
    const uint32_t per_sm = (H * n + 147) / 148;
    const size_t need = (size_t)(2 * C * (D + 8) + C * CP + 3 * 768) * 2 + 4 * C * sizeof(float);
    const size_t sa = std::max(need, per_sm < 4 ? (size_t)228 * 1024 / (per_sm + 1) + 1024 : 0);
    if (!ensure_dyn_smem(delta_chunks_kernel<D>, sa, have_a) || !ensure_dyn_smem(delta_scan_mma_kernel<D>, sizeof(ScanSmem<D>), have_b)) return false;
    if (launch_pdl(delta_chunks_kernel<D>, dim3(H, n), dim3(256), sa, st, chunks, scratch, (int)ntok, (int)q_raw) != cudaSuccess ||
        launch_pdl(delta_scan_mma_kernel<D>, dim3(H, D / DM), dim3(256), sizeof(ScanSmem<D>), st, chunks, (const unsigned char*)scratch, S, (int)n, (int)ntok, (int)q_raw) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g_launches += 2;
    return true;
}

}  // namespace

size_t delta_scan_scratch_bytes(uint32_t n, uint32_t H) { return (size_t)n * H * ITEM_BYTES; }

bool k_delta_scan(cudaStream_t st, const DeltaChunk* chunks, void* scratch, float* S, uint32_t n, uint32_t ntok, uint32_t H, uint32_t D, uint32_t q_raw) {
    return D == 128 ? launch<128>(st, chunks, (unsigned char*)scratch, S, n, ntok, H, q_raw)
                    : D == 64 && launch<64>(st, chunks, (unsigned char*)scratch, S, n, ntok, H, q_raw);
}

}  // namespace gehtp
