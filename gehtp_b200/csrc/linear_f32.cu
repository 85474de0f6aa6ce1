// Projections of fp32 rows: y[M, N] = act(x[M, K] . w^T), w bf16 [N, K].
//
//   up to 16 rows   lin_f32_rows_kernel: weights streamed 16 bytes a lane, fp32 FMA
//   more rows       lin_f32_mma_kernel: an fp32 value is the exact sum of three bf16 values (8 + 8 + 8 bits of its 24), so three
//                   bf16 MMAs make the exact products of the fp32 ones; only the order of the sums differs from FMA tiles.
//                   An infinite weight has no such products (infinity times a middle part of 0): sums that come out as no
//                   number are made again in fp32 FMA
#include <cooperative_groups.h>
#include "linear_epi.cuh"
#include "mma_bf16.cuh"

namespace gehtp {

namespace {

// A warp owns 4 output columns and one of KS shares of K, cut in chunks of 256 (8 weights of each column a lane). Bound by
// the weight stream: 16-byte loads, 8 of them requested ahead of the dependency wait and 4 kept in flight in the loop
// (2-byte loads of one column pair a warp, in its place before: 38.7 us on average for 2048 x 1024 and 3072 x 1024 at one row, now
// 3.8; 1024 x 6144: 16.9, now 4.3). MR: rows of a pass.
template <int KS, int MR, class E>
__global__ void __launch_bounds__(256)
lin_f32_rows_kernel(const float* x, const uint16_t* __restrict__ w, const E epi, uint32_t M, uint32_t K, uint32_t N, uint32_t xs) {
    constexpr int CW = 4, NV = MR * CW, LPV = 32 / NV;
    __shared__ float part[8][NV];
    pdl_release();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ks = warp % KS, cg = warp / KS;
    const uint32_t n0 = (blockIdx.x * (8 / KS) + cg) * CW, m0 = blockIdx.y * MR, chunks = (K + 255) / 256;
    const uint16_t* wr[CW];
#pragma unroll
    for (int c = 0; c < CW; c++) wr[c] = w + (size_t)min(n0 + c, N - 1) * K + lane * 8;
    auto load = [&](uint32_t ch, uint4 (&q)[CW]) {
        const uint32_t k = ch * 256;
        const bool in = n0 < N && ch < chunks && k + lane * 8 < K;
#pragma unroll
        for (int c = 0; c < CW; c++) q[c] = in ? __ldcs((const uint4*)(wr[c] + k)) : make_uint4(0, 0, 0, 0);
    };
    uint4 q0[CW], q1[CW];
    load(ks, q0);
    load(ks + KS, q1);
    pdl_wait();
    float acc[MR][CW];
#pragma unroll
    for (int r = 0; r < MR; r++)
#pragma unroll
        for (int c = 0; c < CW; c++) acc[r][c] = 0.0f;
    auto use = [&](uint32_t ch, const uint4 (&q)[CW]) {
        const uint32_t k = ch * 256 + lane * 8;
        if (k >= K) return;
#pragma unroll
        for (int r = 0; r < MR; r++) {
            const float* xr = x + (size_t)min(m0 + r, M - 1) * xs + k;      // rows past the last repeat it; never stored
            const float4 a = *(const float4*)xr, b = *(const float4*)(xr + 4);
#pragma unroll
            for (int c = 0; c < CW; c++) {
                float s = acc[r][c];
                s = fmaf(a.x, __uint_as_float(q[c].x << 16), s); s = fmaf(a.y, __uint_as_float(q[c].x & 0xffff0000u), s);
                s = fmaf(a.z, __uint_as_float(q[c].y << 16), s); s = fmaf(a.w, __uint_as_float(q[c].y & 0xffff0000u), s);
                s = fmaf(b.x, __uint_as_float(q[c].z << 16), s); s = fmaf(b.y, __uint_as_float(q[c].z & 0xffff0000u), s);
                s = fmaf(b.z, __uint_as_float(q[c].w << 16), s); s = fmaf(b.w, __uint_as_float(q[c].w & 0xffff0000u), s);
                acc[r][c] = s;
            }
        }
    };
    for (uint32_t ch = ks; ch < chunks; ch += 2 * KS) {
        uint4 nx[CW];
        load(ch + 2 * KS, nx);
        use(ch, q0);
#pragma unroll
        for (int c = 0; c < CW; c++) q0[c] = nx[c];
        if (ch + KS >= chunks) break;
        load(ch + 3 * KS, nx);
        use(ch + KS, q1);
#pragma unroll
        for (int c = 0; c < CW; c++) q1[c] = nx[c];
    }
    float v[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] = acc[i / CW][i % CW];
    const float s = fold_sum(v);
    if (lane % LPV == 0) part[warp][lane / LPV] = s;
    __syncthreads();
    if (ks != 0 || lane >= NV / 2) return;
    const uint32_t i = 2 * lane, m = m0 + i / CW;
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int t = 0; t < KS; t++) { a += part[warp + t][i]; b += part[warp + t][i + 1]; }
    if (m < M) epi.pair(m, n0 + i % CW, a, b, N);
}

template <int KS, int MR, class E>
void launch_rows(cudaStream_t st, const LinearArgs& a, const E& epi, uint32_t M) {
    const uint32_t cols = 4 * (8 / KS);
    launch_pdl(lin_f32_rows_kernel<KS, MR, E>, dim3((a.N + cols - 1) / cols, (M + MR - 1) / MR), dim3(256), 0, st, (const float*)a.x, a.w, epi, M,
               a.K, a.N, a.xs);
    g_launches++;
}
template <int MR, class E>
void launch_rows_ks(cudaStream_t st, const LinearArgs& a, const E& epi, uint32_t M) {
    // shares of K until the chip has 16 warps an SM, each with a chunk at least
    const uint32_t groups = (a.N + 3) / 4 * ((M + MR - 1) / MR), chunks = (a.K + 255) / 256;
    if (groups >= 148 * 16 || chunks < 2) launch_rows<1, MR>(st, a, epi, M);
    else if (groups >= 148 * 8 || chunks < 4) launch_rows<2, MR>(st, a, epi, M);
    else if (groups >= 148 * 4 || chunks < 8) launch_rows<4, MR>(st, a, epi, M);
    else launch_rows<8, MR>(st, a, epi, M);
}

// ---- more rows
constexpr uint32_t BM = 64, BN = 64, BK = 32, ST = 4;          // CTA tile, k step, stages
constexpr uint32_t RA = 48, RB = 48;                           // floats of an A row, bf16 of a B row in shared memory: 64- and 128-bit
                                                               // fragment reads of 8 rows fall into different banks
constexpr uint32_t STAGE = BM * RA * 4 + BN * RB * 2, RC = BN + 4;
constexpr uint32_t MMA_SMEM = ST * STAGE;
static_assert(2 * BM * RC * 4 <= MMA_SMEM, "the sums of both k halves fit over the stages");

// hi + mid + lo of two fp32 values, packed in pairs: truncation leaves exactly 8 significant bits to each. Infinities stay
// in hi alone, so that a product is what the fp32 one would be.
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    const float ha = __uint_as_float(ua & 0xffff0000u), hb = __uint_as_float(ub & 0xffff0000u);
    const float ma = fabsf(a) == INFINITY ? 0.0f : a - ha, mb = fabsf(b) == INFINITY ? 0.0f : b - hb;
    const float la = ma - __uint_as_float(__float_as_uint(ma) & 0xffff0000u), lb = mb - __uint_as_float(__float_as_uint(mb) & 0xffff0000u);
    hi = __byte_perm(ua, ub, 0x7632);
    mid = __byte_perm(__float_as_uint(ma), __float_as_uint(mb), 0x7632);
    lo = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);
}

__device__ __noinline__ float dot_f32(const float* x, const uint16_t* w, uint32_t K) {
    float s = 0.0f;
    for (uint32_t k = 0; k < K; k++) s = fmaf(__ldcg(x + k), bf2f(__ldg(w + k)), s);
    return s;
}

// A CTA of 8 warps owns a 64 x 64 tile: 2 x 2 warp tiles of 32 x 32, and the two halves of every 32-deep k step. Lane (g, t)
// holds k = 4t .. 4t + 3 of a 16-deep step in the MMA's k slots 2t, 2t + 1, 2t + 8, 2t + 9 of both operands. The tensor core
// adds without rounding to nearest, so its sums run over 64 k of a warp at most and are added to fp32 registers. gridDim.z CTAs
// of a cluster share K; each adds and finishes its share of the tile's rows from all of them. Bound by the conversions and
// MMAs of the few tiles a prompt of some hundred rows has: 150 x 3072 x 1024 in 25 us, 150 x 1024 x 6144 in 36 (fp32 FMA tiles of
// 64 x 64, one element a load, in its place before: 392 and 172). Error against 64 bits over a 4-layer model: 3.2e-7, before 7.8e-7.
template <class E>
__global__ void __launch_bounds__(256)
lin_f32_mma_kernel(const float* x, const uint16_t* __restrict__ w, const E epi, uint32_t M, uint32_t K, uint32_t N, uint32_t xs) {
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_release();
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t wm = warp & 1, wn = (warp >> 1) & 1, kh = warp >> 2;
    const uint32_t n0 = blockIdx.x * BN, m0 = blockIdx.y * BM, KZ = gridDim.z;
    const uint32_t steps = (K + BK - 1) / BK, per = (steps + KZ - 1) / KZ, s0 = min(blockIdx.z * per, steps), s1 = min(s0 + per, steps);
    auto fetch_b = [&](uint32_t s) {
        if (s < s1) {
            const uint32_t n = tid >> 2, c = tid & 3, k = s * BK + c * 8;
            const bool in = n0 + n < N && k < K;
            cp16(smem_addr(smem + (s % ST) * STAGE + BM * RA * 4 + (n * RB + c * 8) * 2), w + (in ? (size_t)(n0 + n) * K + k : 0), in ? 16 : 0);
        }
    };
    auto fetch_a = [&](uint32_t s) {
        if (s < s1)
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) {
                const uint32_t m = (tid >> 3) + 32 * i, c = tid & 7, k = s * BK + c * 4;
                const bool in = m0 + m < M && k < K;
                cp16(smem_addr(smem + (s % ST) * STAGE + (m * RA + c * 4) * 4), x + (in ? (size_t)(m0 + m) * xs + k : 0), in ? 16 : 0);
            }
    };
#pragma unroll
    for (uint32_t i = 0; i < ST - 1; i++) fetch_b(s0 + i);      // weights: ahead of the dependency wait
    pdl_wait();
#pragma unroll
    for (uint32_t i = 0; i < ST - 1; i++) { fetch_a(s0 + i); cp_commit(); }
    float acc[2][4][4] = {}, run[2][4][4] = {};
    for (uint32_t s = s0; s < s1; s++) {
        cp_wait<ST - 2>();
        __syncthreads();
        fetch_b(s + ST - 1);
        fetch_a(s + ST - 1);
        cp_commit();
        const unsigned char* sa = smem + (s % ST) * STAGE;
        const float* A = (const float*)sa + (wm * 32 + g) * RA + kh * 16 + t * 4;
        const uint16_t* B = (const uint16_t*)(sa + BM * RA * 4) + (wn * 32 + g) * RB + kh * 16 + t * 4;
        uint2 b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = *(const uint2*)(B + j * 8 * RB);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float4 u = *(const float4*)(A + i * 16 * RA), v = *(const float4*)(A + (i * 16 + 8) * RA);
            uint32_t hi[4], mid[4], lo[4];
            split3(u.x, u.y, hi[0], mid[0], lo[0]);
            split3(v.x, v.y, hi[1], mid[1], lo[1]);
            split3(u.z, u.w, hi[2], mid[2], lo[2]);
            split3(v.z, v.w, hi[3], mid[3], lo[3]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                mma_bf16(run[i][j], lo, b[j].x, b[j].y);
                mma_bf16(run[i][j], mid, b[j].x, b[j].y);
                mma_bf16(run[i][j], hi, b[j].x, b[j].y);
            }
        }
        if (((s - s0) & 3) == 3 || s + 1 == s1) {
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) { acc[i][j][e] += run[i][j][e]; run[i][j][e] = 0.0f; }
        }
    }
    cp_wait<0>();
    __syncthreads();
    float* C = (float*)smem;                                    // [2][BM][RC]
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                *(float2*)(C + (kh * BM + wm * 32 + i * 16 + h * 8 + g) * RC + wn * 32 + j * 8 + 2 * t) = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
    if (KZ > 1) cluster.sync(); else __syncthreads();
    const uint32_t share = BM / KZ, r0 = blockIdx.z * share;
    for (uint32_t q = tid; q < share * (BN / 4); q += 256) {
        const uint32_t r = r0 + q / (BN / 4), c = q % (BN / 4) * 4;
        if (m0 + r >= M || n0 + c >= N) continue;
        float v[4] = {};
        for (uint32_t z = 0; z < KZ; z++) {
            const float* p = KZ > 1 ? cluster.map_shared_rank(C, z) : C;
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                const float4 f = *(const float4*)(p + (h * BM + r) * RC + c);
                v[0] += f.x; v[1] += f.y; v[2] += f.z; v[3] += f.w;
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; i++)
            if (isnan(v[i]) && n0 + c + i < N) v[i] = dot_f32(x + (size_t)(m0 + r) * xs, w + (size_t)(n0 + c + i) * K, K);
        epi.quad(m0 + r, n0 + c, v, N);
    }
    if (KZ > 1) cluster.sync();                                 // nobody leaves while its sums are being read
}

template <class E>
bool launch_mma(cudaStream_t st, const LinearArgs& a, const E& epi, uint32_t M) {
    static int have[64] = {};
    if (!ensure_dyn_smem(lin_f32_mma_kernel<E>, MMA_SMEM, have)) return false;
    const uint32_t nb = (a.N + BN - 1) / BN, mb = (M + BM - 1) / BM, steps = (a.K + BK - 1) / BK;
    uint32_t KZ = 1;                                            // CTAs for two an SM, at least 8 steps each
    while (KZ < 8 && nb * mb * KZ * 2 <= 296 && steps >= 16 * KZ) KZ *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb, mb, KZ); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = MMA_SMEM; cfg.stream = st;
    if (launch_pdl_cluster(lin_f32_mma_kernel<E>, cfg, dim3(1, 1, KZ), (const float*)a.x, a.w, epi, M, a.K, a.N, a.xs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g_launches++;
    return true;
}

}  // namespace

// Rows of 16-byte groups only. The rows kernel passes over the weights once per 4 rows: at 16 rows 4 passes of about 4 us meet
// the 21 us a column of MMA tiles takes whatever its rows.
bool k_linear_f32(cudaStream_t st, const LinearArgs& a, uint32_t M) {
    if (a.K % 8 || a.xs % 4 || (((uintptr_t)a.x | (uintptr_t)a.w) & 15u)) return false;
    bool done = true;
    with_epilogue<false>(a, [&](const auto& epi) {
        if (M > 16) { done = launch_mma(st, a, epi, M); return; }
        if (M == 1) launch_rows_ks<1>(st, a, epi, M);
        else if (M == 2) launch_rows_ks<2>(st, a, epi, M);
        else launch_rows_ks<4>(st, a, epi, M);
    });
    return done;
}

}  // namespace gehtp
