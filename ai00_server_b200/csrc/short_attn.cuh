// Softmax attention of prompt steps of many short sequences: the function of prompt_attn.cuh in f32 multiply-adds.  A CTA of prompt_attn.cuh has an SM to itself, whatever few of its
// 128 (token, head) rows are there; sequences of a few rows are better off with small CTAs, several of them on an SM.
//
// What bounds it: latency at the sizes it is for (a CTA's chain of loads, scores, softmax and values); at full rows f32 multiply-adds, 2 dk + 2 dv a (query head, key).  A CTA of four
// warps keeps 64 rows -- the query heads of ONE key / value head for 64 / rep consecutive tokens of one sequence -- and walks the keys in tiles of 32 that it stages once for all of them:
//   * scores   a thread owns 4 rows x 4 keys (rows and keys interleaved, so that the 16-byte reads of eight lanes fall into different banks): eight
//              reads for 64 products;
//   * softmax  running maximum and sum per row in the eight lanes that share it; the weights go through shared memory within the warp;
//   * values   a thread owns 8 rows x 8 entries of the output: 12 reads for 256 products;
//   * products run as packed pairs (fma.rn.f32x2), even and odd entries of a score summed apart;
//   * the next key tile arrives (cp.async) while the values are multiplied, the next value tile while the scores are.
// Measured (steps of four layers of attention, width 256, with prompt_attn.cuh and with this kernel): 64 sequences of 8 tokens, 32 query heads of 64 channels on as many key heads 944 and
// 777 us, of 32 tokens 1281 and 1199; 16 heads of 32 channels 554 and 480, 716 and 660; 16 query heads on 8 key heads, 32 channels, 8 tokens 425 and 384.  Longer ones: 40 tokens of 48
// sequences, 16 heads of 32 channels, 658 and 707.
#pragma once
#include "f32x2.cuh"
#include "prompt_attn.cuh"

namespace b200 {

constexpr int SH_ROWS = 64, SH_KT = 32, SH_THREADS = 128, SH_DMAX = 128;

__host__ __device__ inline size_t short_attn_smem(int dk, int dv) {
    return ((size_t)SH_ROWS * (dk + 4) + (size_t)SH_KT * (dk + 4) + (size_t)SH_KT * (dv + 4) + (size_t)SH_ROWS * (SH_KT + 4) + 2 * SH_ROWS) * sizeof(float);
}

__global__ void __launch_bounds__(SH_THREADS, 2) short_attn_kernel(const __grid_constant__ PromptAttnParams pp) {
    const SinkAttnParams& p = pp.a;
    extern __shared__ __align__(16) float sh_smem[];
    __shared__ int s_tile[2], s_again[SH_ROWS];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) step_token_run(p.meta, pp.qt, blockIdx.x, s_tile);
    __syncthreads();
    const int si = s_tile[0];
    if (si < 0) return;
    const int first = s_tile[1] * pp.qt, nq = min(pp.qt, p.meta.slot_count()[si] - first), t0 = p.meta.slot_start()[si] + first;
    const int slot = p.meta.slot_id()[si], pos0 = p.sm.tok_pos()[t0], pos1 = pos0 + nq - 1;
    const int dk = p.dk, dv = p.dv, rep = p.H / p.G, c = blockIdx.y, R = nq * rep, D = p.D;
    const int PK = dk + 4, PV = dv + 4, PP = SH_KT + 4;
    float* const sQ = sh_smem;                             // [64][dk + 4]
    float* const sK = sQ + SH_ROWS * PK;                   // [32][dk + 4]
    float* const sV = sK + SH_KT * PK;                     // [32][dv + 4]
    float* const sP = sV + SH_KT * PV;                     // [64][36]
    float* const sScl = sP + SH_ROWS * PP;                 // [64] rescaling of a row, later 1 / denominator
    const int* const tbl = p.table + (size_t)slot * p.stride;
    int nkeep, jlo;
    sa_segments(p, pos0, pos1, nkeep, jlo);
    const int nkeys = nkeep + pos1 - jlo + 1, ntiles = (nkeys + SH_KT - 1) / SH_KT;
    auto position = [&](int i) { return i < nkeep ? i : jlo + i - nkeep; };        // kept tokens first, then the window
    // a warp loads the rows 8 warp .. 8 warp + 7 of a tile; rows behind the last key hold the last one's values (their weights are zero)
    auto load = [&](float* dst, const int pitch, const int n4, const size_t off, const int ti) {
#pragma unroll 1
        for (int r = warp * (SH_KT / 4); r < (warp + 1) * (SH_KT / 4); ++r) {
            const float* src = p.cache + sa_token_row(tbl, p.page, position(min(ti * SH_KT + r, nkeys - 1))) * (size_t)D + off;
            for (int q = lane; q < n4; q += 32) cp_async16(dst + r * pitch + 4 * q, src + 4 * q);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const size_t koff = (size_t)p.koff + (size_t)c * dk, voff = (size_t)p.voff + (size_t)c * dv;
    load(sK, PK, dk / 4, koff, 0);
    load(sV, PV, dv / 4, voff, 0);
    for (int i = tid; i < SH_ROWS * (dk / 4); i += SH_THREADS) {
        const int r = i / (dk / 4), q = i - r * (dk / 4);
        *reinterpret_cast<float4*>(sQ + r * PK + 4 * q) =
            r < R ? *reinterpret_cast<const float4*>(p.q + (size_t)(t0 + r / rep) * p.ldq + (size_t)(c * rep + r % rep) * dk + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // scores: rows 16 i + 4 warp + rg (i < 4), keys 8 j + kg (j < 4)
    const int rg = lane >> 3, kg = lane & 7;
    float m[4], l[4];
    int pq[4];
    const float* bias[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 16 * i + 4 * warp + rg;
        m[i] = -CUDART_INF_F; l[i] = 0.f;
        pq[i] = r < R ? pos0 + r / rep : -1;               // rows beyond the last see nothing
        bias[i] = p.bias && r < R ? p.bias + (size_t)(c * rep + r % rep) * (p.nb + 1) : nullptr;
    }
    // values: the warp's rows in the same order, eight a half warp (local row 2 u + half of 16), entries 4 vl .. and 64 + 4 vl ..
    const int half = lane >> 4, vl = lane & 15;
    f32x2 acc[8][4];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[u][e] = 0ull;
    auto row_of = [&](int u) { const int w = 2 * u + half; return 16 * (w >> 2) + 4 * warp + (w & 3); };
    const bool v0 = 4 * vl < dv, v1 = 64 + 4 * vl < dv;
    for (int ti = 0; ti < ntiles; ++ti) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");        // the key tile
        __syncthreads();
        f32x2 s2[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
        {
            const float* qp = sQ + (4 * warp + rg) * PK;
            const float* kp = sK + kg * PK;
#pragma unroll 4
            for (int d = 0; d < dk; d += 4) {
                ulonglong2 q[4], k[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const ulonglong2*>(qp + i * 16 * PK + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(kp + j * 8 * PK + d);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        fma2(s2[i][j], q[i].x, k[j].x);
                        fma2(s2[i][j], q[i].y, k[j].y);
                    }
            }
        }
        __syncthreads();                                    // every warp is done with the key tile
        if (ti + 1 < ntiles) load(sK, PK, dk / 4, koff, ti + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int low = sa_low(p, pq[i]), r = 16 * i + 4 * warp + rg;
            float s[4], tmax = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int idx = ti * SH_KT + 8 * j + kg, at = position(idx);
                const float2 h = unpack2(s2[i][j]);
                const bool vis = idx < nkeys && at <= pq[i] && (at >= low || at < p.keep);
                s[j] = vis ? (h.x + h.y) * p.scale + (bias[i] ? bias[i][min(pq[i] - at, p.nb)] : 0.f) : -CUDART_INF_F;
                tmax = fmaxf(tmax, s[j]);
            }
            tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
            tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
            tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 4));
            const float mn = fmaxf(m[i], tmax);
            const float scl = m[i] > -CUDART_INF_F ? expf(m[i] - mn) : 0.f;
            float tsum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float w = s[j] > -CUDART_INF_F ? expf(s[j] - mn) : 0.f;
                sP[r * PP + 8 * j + kg] = w;
                tsum += w;
            }
            tsum += __shfl_xor_sync(0xffffffffu, tsum, 1);
            tsum += __shfl_xor_sync(0xffffffffu, tsum, 2);
            tsum += __shfl_xor_sync(0xffffffffu, tsum, 4);
            l[i] = l[i] * scl + tsum;
            m[i] = mn;
            if (kg == 0) sScl[r] = scl;
        }
        __syncwarp();                                       // rows of the weights belong to one warp
        asm volatile("cp.async.wait_group 1;" ::: "memory");        // the value tile
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float f = sScl[row_of(u)];
            const f32x2 f2 = pack2(f, f);
#pragma unroll
            for (int e = 0; e < 4; ++e) mul2(acc[u][e], f2);
        }
#pragma unroll 2
        for (int k = 0; k < SH_KT; k += 4) {
            ulonglong2 va[4], vb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                va[q] = v0 ? *reinterpret_cast<const ulonglong2*>(sV + (k + q) * PV + 4 * vl) : make_ulonglong2(0, 0);
                vb[q] = v1 ? *reinterpret_cast<const ulonglong2*>(sV + (k + q) * PV + 64 + 4 * vl) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float4 w = *reinterpret_cast<const float4*>(sP + row_of(u) * PP + k);
                const f32x2 w2[4] = {pack2(w.x, w.x), pack2(w.y, w.y), pack2(w.z, w.z), pack2(w.w, w.w)};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    fma2(acc[u][0], w2[q], va[q].x); fma2(acc[u][1], w2[q], va[q].y);
                    fma2(acc[u][2], w2[q], vb[q].x); fma2(acc[u][3], w2[q], vb[q].y);
                }
            }
        }
        __syncthreads();                                    // every warp is done with the value tile
        if (ti + 1 < ntiles) load(sV, PV, dv / 4, voff, ti + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // the sink joins the denominator
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 16 * i + 4 * warp + rg;
        if (kg == 0 && r < R) {
            const float sk = p.sink ? p.sink[c * rep + r % rep] : -CUDART_INF_F, mx = fmaxf(m[i], sk);
            const float f = m[i] > -CUDART_INF_F ? expf(m[i] - mx) : 0.f;
            sScl[r] = f / (l[i] * f + (p.sink ? expf(sk - mx) : 0.f));
        }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int r = row_of(u);
        float sum = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 a = unpack2(acc[u][e]); sum += a.x + a.y; }
        const bool again = (__ballot_sync(0xffffffffu, !(fabsf(sum) < CUDART_INF_F)) >> (16 * half) & 0xFFFFu) != 0;      // the 16 lanes of the row
        if (vl == 0) s_again[r] = again && r < R;
        if (r >= R || again) continue;
        const int t = t0 + r / rep, h = c * rep + r % rep;
        const float f = sScl[r];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int d = 64 * e + 4 * vl;
            if (d >= dv) continue;
            const float2 a = unpack2(acc[u][2 * e]), b = unpack2(acc[u][2 * e + 1]);
            float4 o = make_float4(a.x * f, a.y * f, b.x * f, b.y * f);
            if (p.gate) {
                const float* g = p.gate + (size_t)t * p.ldg + (p.gate_heads ? (size_t)h : (size_t)h * dv + d);
                const float g0 = lin_sigmoid(g[0]);
                o.x *= g0;
                o.y *= p.gate_heads ? g0 : lin_sigmoid(g[1]); o.z *= p.gate_heads ? g0 : lin_sigmoid(g[2]); o.w *= p.gate_heads ? g0 : lin_sigmoid(g[3]);
            }
            float* const dst = p.out + (size_t)t * p.ldo + (size_t)h * dv + d;
            dst[0] = o.x * p.out_mul; dst[1] = o.y * p.out_mul; dst[2] = o.z * p.out_mul; dst[3] = o.w * p.out_mul;
        }
    }
    __syncwarp();
    auto warp_row = [&](int w) { return 16 * (w >> 2) + 4 * warp + (w & 3); };
    for (unsigned left = __ballot_sync(0xffffffffu, lane < 16 && s_again[warp_row(lane & 15)]); left; left &= left - 1) {
        const int r = warp_row(__ffs(left) - 1);
        prompt_attn_row(p, sQ + r * PK, tbl, c, c * rep + r % rep, t0 + r / rep, pos0 + r / rep);
    }
}

}  // namespace b200
