// Grouped-query attention of fp32 rows over a window of positions, fp32 FMA throughout (the arithmetic of
// window_exact_kernel; its sums in another order).
#include <cooperative_groups.h>
#include "launchers_rows.h"
#include "rows_common.cuh"

namespace gehtp {

namespace {

constexpr uint32_t FW = 8, FC = 8;            // warps of a CTA, CTAs of a cluster at most
constexpr int PB = 4;                         // positions a warp takes at a time

// A warp takes P (row, head) pairs of one key head - `hg` heads of P / hg neighbouring rows - against its share of the
// positions, PB at a time: a lane holds 4 * DI components of the queries, keys, values and sums, so keys and values are read
// once for all pairs in rows of 512 bytes; the P * PB dot products are folded over the warp until each lane has one score,
// one exponential and its part of the softmax. Warps meet in shared memory, CTAs of a cluster in distributed shared memory.
// Bound by the latency of one row's loads (one row), by its shuffles (many). 16 heads of 128 over
// 8 key heads: 4.8 us for one row behind 150 positions (8.4 with positions of earlier runs requested behind the wait and one trip
// to each CTA of the cluster after the other), 30 us for 150 rows (a thread per position walking its key alone, one CTA
// per head and row, in its place before: 89 us for both).
template <int P, int DI>
__global__ void __launch_bounds__(256)
window_f32_kernel(const WindowArgs a, uint32_t rows, uint32_t hg) {
    extern __shared__ __align__(16) float sm[];                   // [FW][P][vdim] values, combined into [P][vdim]
    __shared__ float wm[FW][P], wl[FW][P], cm[P], cl[P];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    constexpr int NV = P * PB, LPV = 32 / NV;
    pdl_release();
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, C = gridDim.x;
    const uint32_t rep = a.heads / a.kv_heads, parts = (rep + hg - 1) / hg, g = blockIdx.y / parts, hp = blockIdx.y % parts * hg;
    const uint32_t R = P / hg, r0 = blockIdx.z * R, row = a.row();
    auto pair_row = [&](uint32_t p) { return min(r0 + p / hg, rows - 1); };        // pairs past the last repeat it; never stored
    auto pair_head = [&](uint32_t p) { return g * rep + min(hp + p % hg, rep - 1); };
    // the counter moves at the end of a run only: it is read, and what earlier runs have left is requested, before the wait
    const uint32_t past = *(volatile const uint32_t*)a.counter;
    auto first_of = [&](uint32_t pos) { return pos + 1 > a.window ? pos + 1 - a.window : 0; };
    const uint32_t first = first_of(past + r0), last = past + pair_row(P - 1);
    const float *keys = (const float*)a.state + g * a.dim, *vals = (const float*)a.state + a.kv_heads * a.dim + g * a.vdim;
    float4 k[PB][DI], v[PB][DI];
    auto load = [&](uint32_t j0) {
#pragma unroll
        for (int b = 0; b < PB; b++) {
            const size_t at = (size_t)((j0 + b) % a.ring) * row;
#pragma unroll
            for (int i = 0; i < DI; i++) {
                const uint32_t d = lane * 4 + 128 * i;
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                k[b][i] = j0 + b <= last && d < a.dim ? __ldcg((const float4*)(keys + at + d)) : z;
                v[b][i] = j0 + b <= last && d < a.vdim ? __ldcg((const float4*)(vals + at + d)) : z;
            }
        }
    };
    const uint32_t step = PB * FW * C;
    uint32_t j0 = first + PB * (blockIdx.x * FW + warp);
    bool early = j0 + PB <= past;
    if (early) load(j0);
    pdl_wait();
    float4 q[P][DI], o[P][DI];
#pragma unroll
    for (int p = 0; p < P; p++)
#pragma unroll
        for (int i = 0; i < DI; i++) {
            const uint32_t d = lane * 4 + 128 * i;
            o[p][i] = make_float4(0.f, 0.f, 0.f, 0.f);
            q[p][i] = d < a.dim ? __ldcg((const float4*)((const float*)a.q + ((size_t)pair_row(p) * a.heads + pair_head(p)) * a.dim + d)) : o[p][i];
        }
    // this lane's pair and place among the PB positions
    const uint32_t mp = lane / LPV / PB, mb = lane / LPV % PB, mpos = past + pair_row(mp), mfirst = first_of(mpos);
    float m = -INFINITY, l = 0.0f;
    for (; j0 <= last; j0 += step) {
        if (!early) load(j0);                                     // past the last: zeros
        early = false;
        float s[NV];
#pragma unroll
        for (int p = 0; p < P; p++)
#pragma unroll
            for (int b = 0; b < PB; b++) {
                float x = 0.0f;
#pragma unroll
                for (int i = 0; i < DI; i++)
                    x = fmaf(q[p][i].x, k[b][i].x, fmaf(q[p][i].y, k[b][i].y, fmaf(q[p][i].z, k[b][i].z, fmaf(q[p][i].w, k[b][i].w, x))));
                s[p * PB + b] = x;
            }
        const float dot = fold_sum(s);
        const uint32_t j = j0 + mb;
        const bool seen = j >= mfirst && j <= mpos;
        const float sc = seen ? dot * a.scale : -INFINITY;
        float mn = fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, LPV));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2 * LPV));
        mn = fmaxf(m, mn);
        const float base = mn == -INFINITY ? 0.0f : mn;            // scores of -inf alone so far: weights of zero
        const float corr = expf(m - base), e = expf(sc - base);
        l = l * corr + e;
        m = mn;
        const uint32_t see = __ballot_sync(0xffffffffu, seen);
#pragma unroll
        for (int p = 0; p < P; p++) {
            const float f = __shfl_sync(0xffffffffu, corr, p * PB * LPV);
#pragma unroll
            for (int i = 0; i < DI; i++) { o[p][i].x *= f; o[p][i].y *= f; o[p][i].z *= f; o[p][i].w *= f; }
#pragma unroll
            for (int b = 0; b < PB; b++) {
                const float x = __shfl_sync(0xffffffffu, e, (p * PB + b) * LPV);
                if (see >> ((p * PB + b) * LPV) & 1u)             // a position this pair does not see is left out, whatever its values are
#pragma unroll
                    for (int i = 0; i < DI; i++) {
                        o[p][i].x = fmaf(x, v[b][i].x, o[p][i].x); o[p][i].y = fmaf(x, v[b][i].y, o[p][i].y);
                        o[p][i].z = fmaf(x, v[b][i].z, o[p][i].z); o[p][i].w = fmaf(x, v[b][i].w, o[p][i].w);
                    }
            }
        }
    }
    l += __shfl_xor_sync(0xffffffffu, l, LPV);
    l += __shfl_xor_sync(0xffffffffu, l, 2 * LPV);
    if (lane % (LPV * PB) == 0) { wm[warp][mp] = m; wl[warp][mp] = l; }
#pragma unroll
    for (int p = 0; p < P; p++)
#pragma unroll
        for (int i = 0; i < DI; i++) {
            const uint32_t d = lane * 4 + 128 * i;
            if (d < a.vdim) *(float4*)(sm + (warp * P + p) * a.vdim + d) = o[p][i];
        }
    __syncthreads();
    for (uint32_t i = tid; i < P * a.vdim; i += 256) {
        const uint32_t p = i / a.vdim;
        float mx = -INFINITY, sum = 0.0f, num = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < FW; w++) mx = fmaxf(mx, wm[w][p]);
#pragma unroll
        for (uint32_t w = 0; w < FW; w++) {
            const float f = wm[w][p] > -INFINITY ? expf(wm[w][p] - mx) : 0.0f;
            sum = fmaf(f, wl[w][p], sum);
            num = fmaf(f, sm[w * P * a.vdim + i], num);
        }
        sm[i] = num;                                              // only this thread reads element i of any warp
        if (i % a.vdim == 0) { cm[p] = mx; cl[p] = sum; }
    }
    const uint32_t per = (P * a.vdim + C - 1) / C, e0 = blockIdx.x * per, e1 = min(e0 + per, P * a.vdim);
    auto gate_of = [&](uint32_t i) {
        const uint32_t p = i / a.vdim;
        return a.gate_col == 0xFFFFFFFFu || i >= e1 ? 0.0f : __ldcg((const float*)a.y + (size_t)pair_row(p) * a.y_cols + a.gate_col + pair_head(p) * a.vdim + i % a.vdim);
    };
    const float gate0 = gate_of(e0 + tid);
    if (C > 1) cluster.sync(); else __syncthreads();
    for (uint32_t i = e0 + tid; i < e1; i += 256) {
        const uint32_t p = i / a.vdim, c = i % a.vdim;
        if (r0 + p / hg >= rows || hp + p % hg >= rep) continue;
        float num = 0.0f, den = 0.0f;
        if (C == 1) {
            num = sm[i]; den = cl[p];
        } else {
            // what the CTAs of the cluster have, requested together: one trip after the other cost 0.1 us each
            float mx = -INFINITY, pm[FC], pn[FC], pl[FC];
#pragma unroll
            for (uint32_t k = 0; k < FC; k++) {
                pm[k] = -INFINITY; pn[k] = pl[k] = 0.0f;
                if (k >= C) continue;
                pm[k] = *cluster.map_shared_rank(cm + p, k);
                pn[k] = *cluster.map_shared_rank(sm + i, k);
                pl[k] = *cluster.map_shared_rank(cl + p, k);
            }
#pragma unroll
            for (uint32_t k = 0; k < FC; k++) mx = fmaxf(mx, pm[k]);
#pragma unroll
            for (uint32_t k = 0; k < FC; k++) {
                const float f = pm[k] > -INFINITY ? expf(pm[k] - mx) : 0.0f;
                if (k >= C) continue;
                num = fmaf(f, pn[k], num);
                den = fmaf(f, pl[k], den);
            }
        }
        const uint32_t r = pair_row(p), h = pair_head(p);
        const float gate = a.gate_col == 0xFFFFFFFFu ? 1.0f : sigmoid_f(i == e0 + tid ? gate0 : gate_of(i));
        ((float*)a.out)[((size_t)r * a.heads + h) * a.vdim + c] = num / den * gate;
    }
    if (C > 1) cluster.sync();                                    // nobody leaves while its results are being read
}

template <int P, int DI>
bool launch(cudaStream_t st, const WindowArgs& a, uint32_t rows, uint32_t hg) {
    static int have[64] = {};
    const size_t smem = (size_t)FW * P * a.vdim * 4;
    if (smem > 40 * 1024 && !ensure_dyn_smem(window_f32_kernel<P, DI>, smem, have)) return false;
    const uint32_t rep = a.heads / a.kv_heads, R = P / hg;
    const dim3 grid(1, a.kv_heads * ((rep + hg - 1) / hg), (rows + R - 1) / R);
    const uint32_t most = a.window < a.ring ? a.window : a.ring;
    uint32_t C = 1;                                               // two rounds per warp before another CTA helps; two CTAs an SM
    while (C < FC && C * FW * PB * 2 < most && grid.y * grid.z * C * 2 <= 296) C *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C, grid.y, grid.z); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    if (launch_pdl_cluster(window_f32_kernel<P, DI>, cfg, dim3(C, 1, 1), a, rows, hg) != cudaSuccess) { cudaGetLastError(); return false; }
    g_launches++;
    return true;
}

}  // namespace

// Heads of 16-byte groups up to 256 components; false: sizes not taken, nothing launched.
bool k_window_f32(cudaStream_t st, const WindowArgs& a, uint32_t rows) {
    if (a.bf16 || a.dim % 4 || a.vdim % 4 || a.dim > 256 || a.vdim > 256 || a.row() % 4 || (((uintptr_t)a.q | (uintptr_t)a.state) & 15u)) return false;
    const uint32_t rep = a.heads / a.kv_heads;
    if ((rows + 7) / 8 > 65535u || rep > 65535u / a.kv_heads) return false;
    const bool wide = a.dim > 128 || a.vdim > 128;
    const uint32_t most = wide ? 4 : 8;
    uint32_t hg = 1, P;
    while (hg * 2 <= rep && hg * 2 <= most) hg *= 2;
    for (P = hg; P < most && P < hg * rows; P *= 2) {}
    if (wide) return P == 1 ? launch<1, 2>(st, a, rows, hg) : P == 2 ? launch<2, 2>(st, a, rows, hg) : launch<4, 2>(st, a, rows, hg);
    return P == 1 ? launch<1, 1>(st, a, rows, hg) : P == 2 ? launch<2, 1>(st, a, rows, hg) : P == 4 ? launch<4, 1>(st, a, rows, hg) : launch<8, 1>(st, a, rows, hg);
}

}  // namespace gehtp
