// The gated delta rule with one decay per head and key channel, sixteen tokens at a time (heads of 128 key channels).
//
// With g_t the decays, F_i = g_1 .. g_i of a chunk, u the corrections and S the state in front of the chunk:
//   u_i = b_i (v_i - (k_i F_i)^T S - sum_(j<i) M_ij u_j)      M_ij = sum_d k_i k_j g_(j+1) .. g_i
//   o_i = (q_i F_i)^T S + sum_(j<=i) N_ij u_j                 N_ij = sum_d q_i k_j g_(j+1) .. g_i
//   S'  = F_16 S + sum_j (k_j g_(j+1) .. g_16) u_j^T
// Solving the triangle for the two parts of u apart gives u = U - W S with W, U free of S. So
//   chunk_prep_kernel  grid (chunk, head): M, N, then W and U by substitution, the decayed q and k, into scratch; fp32 FMA.
//                      Decays of a range are running products of the g, never quotients or sums of logarithms: all factors
//                      are at most 1, and a product of n of them is off by n roundings
//   chunk_walk_kernel  grid (16 value columns, head): walks the chunks. S^T lies in registers as accumulator tiles of
//                      mma.sync m16n8k16, whose layout is that of the next product's A operand; warp w holds 16 of the 128
//                      key rows and leaves partial sums of W S and (qF) S that are added over the warps
// Operands of the tensor cores are three bf16 terms of an fp32 value (24 bits), six products each. Error of o and S against 64
// bits over 100 and 1024 tokens and decays from strong to none: 0.91 to 1.09 and 0.57 to 1.73 of that of the sums token by token
// (channel_delta.cu), 0.98 and 0.97 on average over 1024 tokens.
//
// Bound by the walk's chain: split of S, 24 MMAs of two warps a scheduler, sums over the warps, 12 MMAs, two barriers. 1024 tokens
// of 16 heads: walk 70 us in a prompt (MMAs 22 of them, sums over the warps 8), preparation 31; token by token 217 and 16. 32 heads
// (two CTAs an SM) 108 and 58; token by token 253 and 30. Copies by cp.async of every thread: 80; fp32 operands split in the walk: 80.
//
// Tokens are not kept apart inside a chunk: a value that is no number would reach rows in front of it. A CTA that has seen one
// goes back to the state it began with and takes its columns token by token.
#include <algorithm>
#include "launchers_rows.h"
#include "mma_bf16.cuh"
#include "sm100_umma.cuh"

namespace gehtp {

namespace {

constexpr int T = 16, D = 128, VC = 16;                       // tokens a chunk, key channels, value columns a CTA
// An item of scratch, in words. Operands of the walk's products lie as the three bf16 terms of four neighbouring values: the
// first two as one 16-byte load {hi, hi, mid, mid}, the third apart {lo, lo}. W | qF: [32 tokens][128 keys] (row strides 16 and
// 8 words apart modulo the banks), k: [128 keys in the order of the walk's columns][16 tokens].
constexpr int XS = 144, XL = 72;
constexpr int O_XL = 2 * T * XS, O_K = O_XL + 2 * T * XL, O_KL = O_K + D * T, O_N = O_KL + D * T / 2, O_F = O_N + T * T, SHARED = O_F + D;
constexpr int UV = 2 * T * VC, STAGE = SHARED + UV;                         // of which O_K words are W | qF
constexpr int RS = 36, US = 20;
constexpr int walk_words(int nb) { return nb * STAGE + 8 * VC * RS + VC * US; }
constexpr uint32_t WINDOW = 1024;                             // rows a pair of launches takes: the scratch of 16 heads (59 MB) stays in L2, that of 32 (118 MB) nearly fills it

__host__ __device__ inline size_t item_floats(uint32_t V) { return SHARED + (size_t)2 * T * V; }

// the three terms of four values, paired (x, y), (z, w); rounded ones, so that what the six products leave out has no sign
struct Terms { uint32_t v[3][2]; };
__device__ __forceinline__ Terms terms_of(float4 q) {
    Terms r;
    const float in[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int p = 0; p < 2; p++) {
        float a = in[2 * p], b = in[2 * p + 1];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            r.v[m][p] = pack_bf2(a, b);
            a -= __uint_as_float(r.v[m][p] << 16);
            b -= __uint_as_float(r.v[m][p] & 0xffff0000u);
        }
    }
    return r;
}
__device__ __forceinline__ void put_terms(float* two, float* third, const Terms& x) {
    *(uint4*)two = make_uint4(x.v[0][0], x.v[0][1], x.v[1][0], x.v[1][1]);
    *(uint2*)third = make_uint2(x.v[2][0], x.v[2][1]);
}
__device__ __forceinline__ Terms get_terms(const float* two, const float* third) {
    const uint4 a = *(const uint4*)two;
    const uint2 b = *(const uint2*)third;
    return {{{a.x, a.y}, {a.z, a.w}, {b.x, b.y}}};
}

__device__ __forceinline__ float softplus_of(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// What both forms read of the run: rows r0 .. r0 + rows of it
struct ChunkArgs {
    DeltaArgs a;
    uint32_t r0, rows;
};

// ---- what does not touch the state
template <class A>
__global__ void __launch_bounds__(256, 4)
chunk_prep_kernel(const ChunkArgs c) {
    pdl_release();
    __shared__ __align__(16) float sk[T][D + 4], sq[T][D + 4], sg[T][D + 4], sM[T][T + 4], sN[T][T], sb[T], sd[T];
    const DeltaArgs& a = c.a;
    const uint32_t h = blockIdx.y, t0 = blockIdx.x * T, H = a.heads, KH = a.kv_heads, kh = h / (H / KH), V = a.vdim, C = a.channels();
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float ea = expf(__ldg(a.a_log + h));
    const float4 db = __ldg((const float4*)(a.dt_bias + h * D) + lane);
    pdl_wait();
    // vectors of unit length and decays, a warp per token; tokens past the run change nothing
#pragma unroll
    for (int e = 0; e < T / 8; e++) {
        const uint32_t i = warp + 8 * e, r = c.r0 + t0 + i;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, g = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t0 + i < c.rows) {
            const float* qx = a.qkv + (size_t)r * C + kh * D;
            q = __ldcg((const float4*)qx + lane);
            k = __ldcg((const float4*)(qx + KH * D) + lane);
            const float4 z = __ldcg((const float4*)(a.a + ((size_t)r * H + h) * D) + lane);
            const float qq = warp_sum(fmaf(q.w, q.w, fmaf(q.z, q.z, fmaf(q.y, q.y, q.x * q.x))));
            const float kk = warp_sum(fmaf(k.w, k.w, fmaf(k.z, k.z, fmaf(k.y, k.y, k.x * k.x))));
            const float qk = warp_sum(fmaf(q.w, k.w, fmaf(q.z, k.z, fmaf(q.y, k.y, q.x * k.x))));
            const float iq = 1.0f / sqrtf((float)D) / sqrtf(qq + 1e-6f), ik = 1.0f / sqrtf(kk + 1e-6f);
            if (lane == 0) sd[i] = qk * iq * ik;              // N_ii of the vectors as they came: roundings of their 128 values left out
            q.x *= iq; q.y *= iq; q.z *= iq; q.w *= iq;
            k.x *= ik; k.y *= ik; k.z *= ik; k.w *= ik;
            g = make_float4(expf(-ea * softplus_of(z.x + db.x)), expf(-ea * softplus_of(z.y + db.y)),
                            expf(-ea * softplus_of(z.z + db.z)), expf(-ea * softplus_of(z.w + db.w)));
            if (lane == 0) sb[i] = sigmoid_f(A::ld((const typename A::T*)a.y + (size_t)r * a.ys + a.b_col + h));
        } else if (lane == 0) {
            sb[i] = sd[i] = 0.0f;
        }
        *(float4*)&sk[i][lane * 4] = k; *(float4*)&sq[i][lane * 4] = q; *(float4*)&sg[i][lane * 4] = g;
    }
    __syncthreads();
    // M and N: columns warp and 15 - warp, the key decayed from row to row, lanes along the channels
#pragma unroll 1
    for (int e = 0; e < 2; e++) {
        const int j = e ? T - 1 - (int)warp : (int)warp;
        float4 p = *(const float4*)&sk[j][lane * 4];
        float s[2 * T];
#pragma unroll
        for (int i = 0; i < T; i++) {
            s[i] = s[T + i] = 0.0f;
            if (i < j) continue;
            if (i > j) {
                const float4 g = *(const float4*)&sg[i][lane * 4], k = *(const float4*)&sk[i][lane * 4];
                p.x *= g.x; p.y *= g.y; p.z *= g.z; p.w *= g.w;
                s[i] = fmaf(p.w, k.w, fmaf(p.z, k.z, fmaf(p.y, k.y, p.x * k.x)));
            }
            const float4 q = *(const float4*)&sq[i][lane * 4];
            s[T + i] = fmaf(p.w, q.w, fmaf(p.z, q.z, fmaf(p.y, q.y, p.x * q.x)));
        }
        const float v = fold_sum(s);
        if (lane < T) sM[lane][j] = v;
        else sN[j][lane - T] = (int)lane - T == j ? sd[j] : v;
    }
    __syncthreads();
    float* item = a.work + ((size_t)h * gridDim.x + blockIdx.x) * item_floats(V);
    (item + O_N)[tid] = sN[tid % T][tid / T];
    // W and U: a column of the triangle's right-hand sides per thread
    auto solve = [&](float (&x)[T], float* rest) {
#pragma unroll
        for (int i = 0; i < T; i++) {
            float s = 0.0f;                                   // apart from x: sums of small terms keep their bits
#pragma unroll
            for (int j = 0; j < i; j += 4) {
                const float4 m = *(const float4*)&sM[i][j];
                s = fmaf(m.x, x[j], s);
                if (j + 1 < i) s = fmaf(m.y, x[j + 1], s);
                if (j + 2 < i) s = fmaf(m.z, x[j + 2], s);
                if (j + 3 < i) s = fmaf(m.w, x[j + 3], s);
            }
            const float d = x[i] - s;
            x[i] = sb[i] * d;
            if (rest) rest[i * VC] = fmaf(sb[i], d, -x[i]);       // what the product was rounded by
        }
    };
    if (tid < D) {
        const uint32_t d = tid;
        float x[T], f = 1.0f, b = 1.0f;
        // key d of the walk's warp d / 16: its order there is (column tile, column)
        const uint32_t row = (d & ~15u) + 8 * ((d >> 1) & 1) + 2 * ((d >> 2) & 3) + (d & 1);
#pragma unroll
        for (int i = T - 1; i >= 0; i--) { x[i] = sk[i][d] * b; b *= sg[i][d]; }
#pragma unroll
        for (int i = 0; i < T; i += 4)
            put_terms(item + O_K + row * T + i, item + O_KL + row * (T / 2) + i / 2, terms_of(make_float4(x[i], x[i + 1], x[i + 2], x[i + 3])));
#pragma unroll
        for (int i = 0; i < T; i++) {
            f *= sg[i][d];
            x[i] = sk[i][d] * f;
            sq[i][d] *= f;
        }
        (item + O_F)[d] = f;
        solve(x, nullptr);
#pragma unroll
        for (int i = 0; i < T; i++) sk[i][d] = x[i];
    }
    for (uint32_t col = tid - D; tid >= D && col < V; col += 256 - D) {
        float x[T];
#pragma unroll
        for (int i = 0; i < T; i++) x[i] = t0 + i < c.rows ? __ldcg(a.qkv + (size_t)(c.r0 + t0 + i) * C + 2 * KH * D + h * V + col) : 0.0f;
        float* out = item + SHARED + col / VC * UV + col % VC;
        solve(x, out + T * VC);
#pragma unroll
        for (int i = 0; i < T; i++) out[i * VC] = x[i];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2 * T / 8; e++) {
        const uint32_t i = warp + 8 * e;
        const float4 x = *(const float4*)(e < T / 8 ? &sk[i][lane * 4] : &sq[i - T][lane * 4]);
        put_terms(item + i * XS + lane * 4, item + O_XL + i * XL + lane * 2, terms_of(x));
    }
}

// ---- the walk
// c[n] = A B[n] over 16, the N sums side by side: the product of the first terms, whose sum of 16 loses next to nothing where the
// tensor core cuts it off, apart from the five below it, 2^-8 of its size; one rounded sum of the two. (All six into one
// accumulator: error of o against 64 bits 1.51e-7 where the sums token by token had 1.29e-7.)
template <int N>
__device__ __forceinline__ void mma_terms(float (&c)[N][4], const uint32_t (&a)[3][4], const Terms (&b)[N]) {
    constexpr int PA[5] = {2, 0, 1, 1, 0}, PB[5] = {0, 2, 1, 0, 1};
    float lo[N][4] = {};
#pragma unroll
    for (int n = 0; n < N; n++) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.0f;
#pragma unroll
    for (int m = 0; m < 5; m++)
#pragma unroll
        for (int n = 0; n < N; n++) mma_bf16(lo[n], a[PA[m]], b[n].v[PB[m]][0], b[n].v[PB[m]][1]);
#pragma unroll
    for (int n = 0; n < N; n++) mma_bf16(c[n], a[0], b[n].v[0][0], b[n].v[0][1]);
#pragma unroll
    for (int n = 0; n < N; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) c[n][e] += lo[n][e];
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// The columns c0 .. c0 + 15 of head h token by token: thread (d, half) holds eight columns of row d of S.
template <class A>
__device__ __noinline__ void walk_tokens(const ChunkArgs& c, float* sm, uint32_t h, uint32_t c0) {
    const DeltaArgs& a = c.a;
    const uint32_t tid = threadIdx.x, d = tid & (D - 1), half = tid / D, warp = tid >> 5, lane = tid & 31;
    const uint32_t H = a.heads, KH = a.kv_heads, kh = h / (H / KH), V = a.vdim, C = a.channels();
    float (*part)[16] = (float (*)[16])sm;                     // [8 warps][16 sums]
    float (*nrm)[4] = (float (*)[4])(sm + 128);
    float* Sg = a.S + ((size_t)h * D + d) * V + c0 + half * 8;
    const float ea = expf(__ldg(a.a_log + h)), db = __ldg(a.dt_bias + h * D + d);
    float S[8];
#pragma unroll
    for (int j = 0; j < 8; j++) S[j] = Sg[j];
    for (uint32_t t = 0; t < c.rows; t++) {
        const size_t r = c.r0 + t;
        const float *qx = a.qkv + r * C + kh * D, *vx = a.qkv + r * C + 2 * KH * D + h * V + c0 + half * 8;
        const float q = __ldcg(qx + d), k = __ldcg(qx + KH * D + d), g = expf(-ea * softplus_of(__ldcg(a.a + (r * H + h) * D + d) + db));
        const float qq = warp_sum(q * q), kk = warp_sum(k * k), qk = warp_sum(q * k);
        __syncthreads();
        if (lane == 0) { nrm[warp][0] = qq; nrm[warp][1] = kk; nrm[warp][2] = qk; }
        float s[16];
#pragma unroll
        for (int j = 0; j < 8; j++) { S[j] *= g; s[j] = S[j] * k; s[8 + j] = S[j] * q; }
        const float v = fold_sum(s);
        if ((lane & 1) == 0) part[warp][lane / 2] = v;
        __syncthreads();
        float n[3] = {};
#pragma unroll
        for (int w = 0; w < 4; w++)
#pragma unroll
            for (int m = 0; m < 3; m++) n[m] += nrm[half * 4 + w][m];
        const float iq = 1.0f / sqrtf((float)D) / sqrtf(n[0] + 1e-6f), ik = 1.0f / sqrtf(n[1] + 1e-6f);
        const float b = sigmoid_f(A::ld((const typename A::T*)a.y + r * a.ys + a.b_col + h));
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float sk = 0.0f, sq = 0.0f;
#pragma unroll
            for (int w = 0; w < 4; w++) { sk += part[half * 4 + w][j]; sq += part[half * 4 + w][8 + j]; }
            const float u = b * (__ldcg(vx + j) - sk * ik);
            S[j] = fmaf(k * ik, u, S[j]);
            if (d == 0) a.o[(r * H + h) * V + c0 + half * 8 + j] = fmaf(u, n[2] * iq * ik, sq * iq);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) Sg[j] = S[j];
}

template <class A, int NB>
__global__ void __launch_bounds__(256, NB == 2 ? 2 : 1)
chunk_walk_kernel(const ChunkArgs c) {
    extern __shared__ __align__(16) float sm[];
    __shared__ uint64_t full[2][NB];                          // copies of W | qF, of the rest
    // NB buffers of W | qF, NB of the rest of an item, then
    float* red = sm + NB * STAGE;                             // [8 warps][16 columns][RS]: parts of W S and (qF) S, 32 tokens
    float* us = red + 8 * VC * RS;                            // [16 columns][US]: u
    const DeltaArgs& a = c.a;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t h = blockIdx.y, c0 = blockIdx.x * VC, H = a.heads, V = a.vdim, n = (c.rows + T - 1) / T;
    const float* items = a.work + (size_t)h * n * item_floats(V);
    auto x_of = [&](uint32_t ch) { return sm + ch % NB * O_K; };
    auto rest_of = [&](uint32_t ch) { return sm + NB * O_K + ch % NB * (STAGE - O_K) - O_K; };     // indexed like an item
    constexpr int NEVER = 0x7FFFFFFF;
    int lost = NEVER;                                         // the chunk of the walk at which a wait ran out
    auto fetch_x = [&](uint32_t ch) {                         // one thread
        if (ch >= n || lost != NEVER) return;
        uint64_t* bar = &full[0][ch % NB];
        sm100::mbar_expect_tx(bar, O_K * 4);
        sm100::bulk_load(x_of(ch), items + ch * item_floats(V), O_K * 4, bar);
    };
    auto fetch_rest = [&](uint32_t ch) {
        if (ch >= n || lost != NEVER) return;
        const float* src = items + ch * item_floats(V);
        uint64_t* bar = &full[1][ch % NB];
        sm100::mbar_expect_tx(bar, (STAGE - O_K) * 4);
        sm100::bulk_load(rest_of(ch) + O_K, src + O_K, (SHARED - O_K) * 4, bar);
        sm100::bulk_load(rest_of(ch) + SHARED, src + SHARED + blockIdx.x * UV, UV * 4, bar);
    };
    auto arrived = [&](int part, uint32_t ch) {
        if (lost == NEVER && !sm100::mbar_wait(&full[part][ch % NB], ch / NB & 1)) { lost = (int)ch - (part == 0); raise_status(a.status, kStatusDeltaTimeout); }
    };
    if (tid == 0) {
        for (int i = 0; i < 2 * NB; i++) sm100::mbar_init(&full[i / NB][i % NB], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (uint32_t ch = 0; ch < NB; ch++) fetch_x(ch);
        for (uint32_t ch = 0; ch + 1 < NB; ch++) fetch_rest(ch);
    }
    // S^T: rows g and g + 8 (columns of S), tile m holds key rows key0 + 2 m and the one behind it. The k slots of a product
    // over 16 are numbered the same way: four neighbouring keys (tokens, for the update) are one 16-byte load
    const uint32_t key0 = 16 * warp + 4 * t;
    float* Sg = a.S + ((size_t)h * D + key0) * V + c0 + g;
    float S[2][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int e = 0; e < 4; e++) S[m][e] = Sg[(size_t)(2 * m + (e & 1)) * V + (e >> 1) * 8];
    // the sums this thread adds up: column v, tokens i and i + 1 of u (warps 0 - 3) or of o (4 - 7)
    const uint32_t v = tid & 15, i = (tid >> 4 & 7) * 2;
    const bool of_u = tid < 128;
    float* og = a.o + ((size_t)(c.r0 + i) * H + h) * V + c0 + v;
    bool bad = false;
    __syncthreads();
    Terms bx[4];
    auto load_x = [&](const float* st) {
#pragma unroll
        for (int j = 0; j < 4; j++) bx[j] = get_terms(st + (8 * j + g) * XS + key0, st + O_XL + (8 * j + g) * XL + key0 / 2);
    };
    arrived(0, 0);
    load_x(x_of(0));
    for (uint32_t ch = 0; ch < n; ch++) {
        const float* st = rest_of(ch);
        // ---- S^T (W | qF)^T over this warp's keys
        {
            uint32_t as[3][4];
            const Terms x = terms_of(make_float4(S[0][0], S[0][1], S[1][0], S[1][1])), y = terms_of(make_float4(S[0][2], S[0][3], S[1][2], S[1][3]));
#pragma unroll
            for (int m = 0; m < 3; m++) { as[m][0] = x.v[m][0]; as[m][1] = y.v[m][0]; as[m][2] = x.v[m][1]; as[m][3] = y.v[m][1]; }
            float p[4][4];
            mma_terms(p, as, bx);
            float* rw = red + warp * (VC * RS) + g * RS + 2 * t;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                *(float2*)(rw + 8 * j) = make_float2(p[j][0], p[j][1]);
                *(float2*)(rw + 8 * RS + 8 * j) = make_float2(p[j][2], p[j][3]);
            }
        }
        __syncthreads();
        if (tid == 0) { fetch_x(ch + NB); fetch_rest(ch + NB - 1); }      // into what was read before the barrier
        float2 s = make_float2(0.0f, 0.0f);
        {
            const float* r = red + v * RS + 2 * (tid >> 4);
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const float2 z = *(const float2*)(r + w * (VC * RS));
                s.x += z.x; s.y += z.y;
            }
        }
        arrived(1, ch);
        if (of_u) {
            const float* U = st + SHARED + i * VC + v;
            s.x = U[0] - (s.x - U[T * VC]);
            s.y = U[VC] - (s.y - U[T * VC + VC]);
            bad |= !finite(s.x) || !finite(s.y);
            *(float2*)(us + v * US + i) = s;
        }
        // operands of what follows, in the shadow of the barrier
        Terms bk[2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const uint32_t row = 16 * warp + 8 * m + g;
            bk[m] = get_terms(st + O_K + row * T + 4 * t, st + O_KL + row * (T / 2) + 2 * t);
        }
        const float4 f4 = *(const float4*)(st + O_F + key0);
        if (ch + 1 < n) { arrived(0, ch + 1); load_x(x_of(ch + 1)); }
        __syncthreads();
        // ---- S' = F S + (decayed k)^T u
        {
            uint32_t au[3][4];
            const Terms x = terms_of(*(const float4*)(us + g * US + 4 * t)), y = terms_of(*(const float4*)(us + (g + 8) * US + 4 * t));
#pragma unroll
            for (int m = 0; m < 3; m++) { au[m][0] = x.v[m][0]; au[m][1] = y.v[m][0]; au[m][2] = x.v[m][1]; au[m][3] = y.v[m][1]; }
            float d[2][4];
            mma_terms(d, au, bk);
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) S[m][e] = fmaf(S[m][e], m ? (e & 1 ? f4.w : f4.z) : (e & 1 ? f4.y : f4.x), d[m][e]);
        }
        if (!of_u) {
            float n0 = 0.0f, n1 = 0.0f;
#pragma unroll
            for (int j = 0; j < T; j += 4) {
                const float4 w = *(const float4*)(us + v * US + j), x = *(const float4*)(st + O_N + i * T + j), y = *(const float4*)(st + O_N + (i + 1) * T + j);
                n0 = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, n0))));
                n1 = fmaf(y.w, w.w, fmaf(y.z, w.z, fmaf(y.y, w.y, fmaf(y.x, w.x, n1))));
            }
            s.x += n0; s.y += n1;
            bad |= !finite(s.x) || !finite(s.y);
            float* out = og + (size_t)ch * T * H * V;
            if (ch * T + i < c.rows) out[0] = s.x;
            if (ch * T + i + 1 < c.rows) out[(size_t)H * V] = s.y;
        }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int e = 0; e < 4; e++) bad |= !finite(S[m][e]);
    if (__syncthreads_or(lost != NEVER)) {
        // Copies on their way land before the CTA's shared memory is another's. Thread 0 has requested what the walk asks for up to the
        // chunk at which it gave up (-1: the first), or all of it; the last copy of each buffer is behind all earlier ones.
        if (tid == 0)
            for (int part = 0; part < 2; part++) {
                const uint32_t asked = lost == NEVER ? n : min(n, (uint32_t)(lost + NB + 1 - part));
                for (uint32_t ch = asked > NB ? asked - NB : 0; ch < asked; ch++) sm100::mbar_wait(&full[part][ch % NB], ch / NB & 1);
            }
        __syncthreads();
        return;
    }
    if (__syncthreads_or(bad)) { walk_tokens<A>(c, sm, h, c0); return; }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int e = 0; e < 4; e++) Sg[(size_t)(2 * m + (e & 1)) * V + (e >> 1) * 8] = S[m][e];
}

template <class A, int NB>
void launch_walk(cudaStream_t st, const ChunkArgs& c) {
    constexpr size_t smem = (size_t)walk_words(NB) * 4;
    static int have[64] = {};
    ensure_dyn_smem(chunk_walk_kernel<A, NB>, smem, have);
    chunk_walk_kernel<A, NB><<<dim3(c.a.vdim / VC, c.a.heads), 256, smem, st>>>(c);
}
template <class A>
void launch(cudaStream_t st, const DeltaArgs& a, uint32_t rows) {
    for (uint32_t r0 = 0; r0 < rows; r0 += WINDOW) {
        const ChunkArgs c = {a, r0, std::min(WINDOW, rows - r0)};
        launch_pdl(chunk_prep_kernel<A>, dim3((c.rows + T - 1) / T, a.heads), dim3(256), 0, st, c);
        // three buffers while a CTA has an SM to itself (16 heads 76 us, two buffers 82), two CTAs an SM from there on
        if (a.vdim / VC * a.heads <= 148) launch_walk<A, 3>(st, c);
        else launch_walk<A, 2>(st, c);
        g_launches += 2;
    }
}

}  // namespace

// From two chunks on while a CTA has an SM to itself, from four where two share one and a chunk takes longer; below, what a chunk costs
// in the two launches is not made up for. A run of two such layers and two of latent attention without the head, token by token /
// in chunks, us: 16 heads, 32 tokens 314 / 308, 64 tokens 338 / 322, fp32 40 tokens 540 / 533; 32 heads, 33 tokens 438 / 450,
// 40 tokens 442 / 447, 56 tokens 466 / 471, 64 tokens 478 / 477, 80 tokens 500 / 494, 128 tokens 559 / 534.
bool delta_chunks_take(const DeltaArgs& a, uint32_t rows) {
    return a.dim == D && a.vdim % VC == 0 && rows >= (a.vdim / VC * a.heads <= 148 ? 2 : 4) * T && (((uintptr_t)a.qkv | (uintptr_t)a.a | (uintptr_t)a.dt_bias | (uintptr_t)a.work) & 15) == 0;
}

size_t delta_chunks_floats(const DeltaArgs& a, uint32_t max_rows) {
    return a.dim == D && a.vdim % VC == 0 ? (size_t)a.heads * ((std::min(max_rows, WINDOW) + T - 1) / T) * item_floats(a.vdim) : 0;
}

void k_delta_chunks(cudaStream_t st, const DeltaArgs& a, uint32_t rows) {
    if (a.bf16) launch<ActBf16>(st, a, rows);
    else launch<ActF32>(st, a, rows);
}

}  // namespace gehtp
