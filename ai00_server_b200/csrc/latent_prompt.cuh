// Latent attention of prompt steps on the tensor cores (serving precision): the function of latent_attn_tc_kernel (latent_attn.cuh) with the same operands
// (TF32, rounded once, f32 sums and softmax), for steps whose keys are not split: many tokens, or contexts of fewer than four key tiles of 32 (kx_fill_step).
//
// What bounds it: the TF32 rate of mma.sync (about 125 multiply-adds a cycle and SM), if operands come cheaply.  All heads read the same latent row, so a CTA
// of eight warps keeps 64 rows -- up to 16 heads x 4 tokens, 8 x 8 and so on -- and reads each key tile once for them, where the 16-row form read it four
// times, waited for every tile and rounded its keys again in every product:
//   * keys arrive 16 at a time into two buffers (cp.async); the thread that asked for 16 bytes rounds them in place before the barrier;
//   * scores   a warp owns 16 rows x 8 keys, two accumulators;
//   * softmax  two rows a warp at a time;
//   * values   a warp owns all 64 rows of an eighth of the channels;
//   * the finished rows go out normalised: no partial results, no merging launch.
// Measured (eight documents of up to 700 tokens, 16 heads, rows of 576 floats, two steps, ncu): 2119 us and 124 of merging -> 1127.
// Where the line lies: short contexts leave it a quarter of the 16-row form's CTAs, but one launch instead of two.  Whole prompts of two layers with the 16-row form and with
// this one, width 2048: 1 x 20 tokens 342 and 342 us, 2 x 20 367 and 370, 1 x 64 426 and 422, 8 x 64 668 and 618, 16 x 32 606 and 571; width 1024: 1 x 96 361 and 358,
// 2 x 64 350 and 346, 16 x 32 377 and 374; width 512: 1 x 64 257 and 261, 2 x 20 212 and 215.
#pragma once
#include "latent_attn.cuh"

namespace b200 {

constexpr int LP_ROWS = 64, LP_KT = 16, LP_THREADS = 256, LP_MAX_NT = 8, LP_SP = LP_KT + 4;
constexpr size_t LATENT_PROMPT_SMEM = 227 * 1024 - 512;      // latent rows of up to 588 floats; longer ones stay with the 16-row form

struct LatentPromptParams {
    LatentAttnParams a;            // part and nsplit are not read
    float* out;                    // [T, H * rk]
    int hg, qt;                    // heads and tokens of a CTA: hg * qt <= LP_ROWS
};

__host__ __device__ inline size_t latent_prompt_smem(int D) {
    return ((size_t)(LP_ROWS + 2 * LP_KT) * la_stride(D) + LP_ROWS * LP_SP + LP_ROWS) * sizeof(float);
}

// One row (token t at position pos, head h) worked out again by the CTA's warps, key by key, each its channels from `c0` on: see prompt_attn_row.
__device__ __noinline__ void latent_prompt_row(const LatentPromptParams& pp, const int* tab, int h, int t, int pos, int c0, int cw) {
    const LatentAttnParams& p = pp.a;
    const int lane = threadIdx.x & 31, D = p.rk + p.dr;
    const float* q = p.q + (size_t)t * p.H * D + (size_t)h * D;
    float m = -CUDART_INF_F, l = 0.f, acc[2] = {0.f, 0.f};
    for (int kj = 0; kj <= pos; ++kj) {
        const float* row = p.cache + ((size_t)tab[kj / p.page] * p.page + kj % p.page) * D;
        float dot = 0.f;
        for (int d = lane; d < D; d += 32) dot = fmaf(__uint_as_float(to_tf32(q[d])), __uint_as_float(to_tf32(row[d])), dot);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float sc = dot * p.scale, mn = fmaxf(m, sc);
        float pj = 0.f, corr = 1.f;
        if (mn > -CUDART_INF_F) { pj = expf(sc - mn); corr = expf(m - mn); }
        l = l * corr + pj;
        m = mn;
        pj = __uint_as_float(to_tf32(pj));
        for (int e = 0; e < 2; ++e) {
            const int ch = c0 + lane + 32 * e;
            acc[e] = fmaf(pj, lane + 32 * e < cw && ch < p.rk ? __uint_as_float(to_tf32(row[ch])) : 0.f, acc[e] * corr);
        }
    }
    for (int e = 0; e < 2; ++e) {
        const int ch = c0 + lane + 32 * e;
        if (lane + 32 * e < cw && ch < p.rk) pp.out[(size_t)t * p.H * p.rk + (size_t)h * p.rk + ch] = acc[e] / l;
    }
}

__global__ void __launch_bounds__(LP_THREADS, 1) latent_prompt_kernel(const __grid_constant__ LatentPromptParams pp) {
    const LatentAttnParams& p = pp.a;
    extern __shared__ __align__(16) float lp_smem[];
    __shared__ int s_tile[2], s_again[LP_ROWS];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
    if (warp == 0) step_token_run(p.meta, pp.qt, blockIdx.x, s_tile);
    __syncthreads();
    const int si = s_tile[0];
    if (si < 0) return;
    const int first = s_tile[1] * pp.qt, nt = min(pp.qt, p.meta.slot_count()[si] - first), t0 = p.meta.slot_start()[si] + first;
    const int slot = p.meta.slot_id()[si], pos0 = p.sm.tok_pos()[t0], nkeys = pos0 + nt, ntiles = (nkeys + LP_KT - 1) / LP_KT;
    const int HG = pp.hg, h0 = blockIdx.y * HG, D = p.rk + p.dr, rk = p.rk, Dp = la_pad8(D), DS = la_stride(D);
    float* const sq = lp_smem;                             // [64][DS]
    float* const sk = sq + (size_t)LP_ROWS * DS;           // [2][16][DS]
    float* const ss = sk + (size_t)2 * LP_KT * DS;         // [64][20] scores, then probabilities
    float* const scorr = ss + LP_ROWS * LP_SP;             // [64] rescaling of a row, later 1 / denominator
    const int* const tab = p.table + (size_t)slot * p.stride;
    // warp w asks for the rows 2 w, 2 w + 1 of a tile
    auto load = [&](const int ti) {
        float* const buf = sk + (size_t)(ti & 1) * LP_KT * DS;
#pragma unroll
        for (int r = 2 * warp; r < 2 * warp + 2; ++r) {
            const int kj = ti * LP_KT + r;
            const float* src = kj < nkeys ? p.cache + ((size_t)tab[kj / p.page] * p.page + kj % p.page) * D : nullptr;
            for (int c = lane; c < D / 4; c += 32) {
                float* dst = buf + (size_t)r * DS + 4 * c;
                if (src) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src + 4 * c) : "memory");
                else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto round4 = [](float4 v) {
        return make_float4(__uint_as_float(to_tf32(v.x)), __uint_as_float(to_tf32(v.y)), __uint_as_float(to_tf32(v.z)), __uint_as_float(to_tf32(v.w)));
    };
    load(0);
    for (int i = tid; i < LP_ROWS * (D / 4); i += LP_THREADS) {
        const int r = i / (D / 4), c = i - r * (D / 4), qi = r / HG, h = h0 + r % HG;
        const bool in = qi < nt && h < p.H;
        *reinterpret_cast<float4*>(sq + (size_t)r * DS + 4 * c) =
            in ? round4(*reinterpret_cast<const float4*>(p.q + (size_t)(t0 + qi) * p.H * D + (size_t)h * D + 4 * c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int i = tid; i < (LP_ROWS + 2 * LP_KT) * (DS - D); i += LP_THREADS) {       // pad columns stay zero
        const int j = i / (DS - D);
        sq[(size_t)j * DS + D + (i - j * (DS - D))] = 0.f;
    }
    float m[4], l[4];                                      // rows 8 warp + 2 i + (lane >> 4)
#pragma unroll
    for (int i = 0; i < 4; ++i) { m[i] = -CUDART_INF_F; l[i] = 0.f; }
    const int cw = la_pad8((rk + 7) / 8);                  // latent channels per warp, a multiple of 8
    float o[4][LP_MAX_NT][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int n = 0; n < LP_MAX_NT; ++n) o[a][n][0] = o[a][n][1] = o[a][n][2] = o[a][n][3] = 0.f;
    for (int ti = 0; ti < ntiles; ++ti) {
        float* const kt = sk + (size_t)(ti & 1) * LP_KT * DS;
        if (ti + 1 < ntiles) {
            load(ti + 1);                                  // into the buffer of tile ti - 1: everyone left it at the barrier below
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
#pragma unroll
        for (int r = 2 * warp; r < 2 * warp + 2; ++r)      // this thread's own pieces
            for (int c = lane; c < D / 4; c += 32) {
                float4* const at = reinterpret_cast<float4*>(kt + (size_t)r * DS + 4 * c);
                *at = round4(*at);
            }
        __syncthreads();
        {
            const int rt = warp & 3, k8 = warp >> 2;
            float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
            const float* qa = sq + (size_t)(rt * 16 + gq) * DS + tq;
            const float* qb = qa + (size_t)8 * DS;
            const float* kb = kt + (size_t)(k8 * 8 + gq) * DS + tq;
            auto step = [&](float (&acc)[4], const int ks) {
                const uint32_t a[4] = {__float_as_uint(qa[ks]), __float_as_uint(qb[ks]), __float_as_uint(qa[ks + 4]), __float_as_uint(qb[ks + 4])};
                const uint32_t b[2] = {__float_as_uint(kb[ks]), __float_as_uint(kb[ks + 4])};
                mma_tf32_1688(acc, a, b);
            };
            int ks = 0;
#pragma unroll 4
            for (; ks + 16 <= Dp; ks += 16) { step(a0, ks); step(a1, ks + 8); }
            if (ks < Dp) step(a0, ks);
            *reinterpret_cast<float2*>(ss + (rt * 16 + gq) * LP_SP + k8 * 8 + tq * 2) = make_float2(a0[0] + a1[0], a0[1] + a1[1]);
            *reinterpret_cast<float2*>(ss + (rt * 16 + gq + 8) * LP_SP + k8 * 8 + tq * 2) = make_float2(a0[2] + a1[2], a0[3] + a1[3]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 8 * warp + 2 * i + (lane >> 4), key = lane & 15, qi = r / HG;
            const bool live = qi < nt && ti * LP_KT + key <= pos0 + qi;
            const float sc = live ? ss[r * LP_SP + key] * p.scale : -CUDART_INF_F;
            float mx = sc;
#pragma unroll
            for (int of = 8; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
            const float mn = fmaxf(m[i], mx);
            float pj = 0.f, corr = 1.f;
            if (mn > -CUDART_INF_F) {
                pj = live ? expf(sc - mn) : 0.f;
                corr = expf(m[i] - mn);
            }
            float ps = pj;
#pragma unroll
            for (int of = 8; of > 0; of >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, of);
            l[i] = l[i] * corr + ps;
            m[i] = mn;
            ss[r * LP_SP + key] = __uint_as_float(to_tf32(pj));
            if (key == 0) scorr[r] = corr;
        }
        __syncthreads();
        {
            uint32_t a[4][2][4];
#pragma unroll
            for (int rt = 0; rt < 4; ++rt) {
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const float* s0 = ss + (rt * 16 + gq) * LP_SP + ks * 8 + tq;
                    a[rt][ks][0] = __float_as_uint(s0[0]); a[rt][ks][1] = __float_as_uint(s0[8 * LP_SP]);
                    a[rt][ks][2] = __float_as_uint(s0[4]); a[rt][ks][3] = __float_as_uint(s0[8 * LP_SP + 4]);
                }
                const float c0 = scorr[rt * 16 + gq], c1 = scorr[rt * 16 + gq + 8];
#pragma unroll
                for (int n = 0; n < LP_MAX_NT; ++n) { o[rt][n][0] *= c0; o[rt][n][1] *= c0; o[rt][n][2] *= c1; o[rt][n][3] *= c1; }
            }
#pragma unroll
            for (int n = 0; n < LP_MAX_NT; ++n) {
                const int cb = warp * cw + n * 8;
                if (n * 8 >= cw || cb >= rk) break;
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const uint32_t b[2] = {__float_as_uint(kt[(size_t)(ks * 8 + tq) * DS + cb + gq]), __float_as_uint(kt[(size_t)(ks * 8 + tq + 4) * DS + cb + gq])};
#pragma unroll
                    for (int rt = 0; rt < 4; ++rt) mma_tf32_1688(o[rt][n], a[rt][ks], b);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((lane & 15) == 0) scorr[8 * warp + 2 * i + (lane >> 4)] = 1.f / l[i];
    if (tid < LP_ROWS) s_again[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int rt = 0; rt < 4; ++rt)
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < LP_MAX_NT; ++n) sum += o[rt][n][hrow * 2] + o[rt][n][hrow * 2 + 1];
            if (!(fabsf(sum) < CUDART_INF_F)) s_again[rt * 16 + gq + hrow * 8] = 1;
        }
    __syncthreads();
#pragma unroll
    for (int rt = 0; rt < 4; ++rt)
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            const int r = rt * 16 + gq + hrow * 8, qi = r / HG, h = h0 + r % HG;
            if (qi >= nt || h >= p.H || s_again[r]) continue;
            const float inv = scorr[r];
            float* const dst = pp.out + (size_t)(t0 + qi) * p.H * rk + (size_t)h * rk;
#pragma unroll
            for (int n = 0; n < LP_MAX_NT; ++n) {
                const int cb = warp * cw + n * 8;
                if (n * 8 >= cw || cb >= rk) break;
                const int d = cb + tq * 2;
                if (d < rk) dst[d] = o[rt][n][hrow * 2] * inv;
                if (d + 1 < rk) dst[d + 1] = o[rt][n][hrow * 2 + 1] * inv;
            }
        }
    unsigned long long left = __ballot_sync(0xffffffffu, s_again[lane]) | (unsigned long long)__ballot_sync(0xffffffffu, s_again[32 + lane]) << 32;
    for (; left; left &= left - 1) {
        const int r = __ffsll((long long)left) - 1;
        if (r / HG < nt && h0 + r % HG < p.H) latent_prompt_row(pp, tab, h0 + r % HG, t0 + r / HG, pos0 + r / HG, warp * cw, cw);
    }
}

}  // namespace b200
