// Routed mixture of experts around the grouped linear kernels (linear.cuh).
//   moe_route_kernel     one CTA per token: router logits (f32 products on the f32 row, in every precision), probabilities =
//                        softmax over all router outputs (real + identity experts);
//                        the `top` largest of (probability + selection bias) are chosen (ties: lower index), their weights
//                        are the un-biased probabilities, not renormalised
//   moe_group_kernel     one CTA: per-expert row counts, offsets and token lists in token order (deterministic), and for every
//                        (token, choice) its compact row, or -1 for an identity expert
//   moe_combine_kernel   x[t] += gate2[t] * ( sum_k w_k * (expert row | h[t] for an identity expert)
//                                              + sigmoid(sg . h[t]) * shared[t] )                     (residual accumulate, f32)
// The experts' matrices are stacked [E][...] so that one grouped launch covers all of them; rows are gathered by list.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include "common.cuh"

namespace b200 {

constexpr int MOE_MAX_TOP = 8;

struct MoeRouteParams {
    const float* h; int ldh;                  // [T, K] router input (f32)
    const __nv_bfloat16* Wr;                  // [NE, K] router matrix
    int K;
    const float* bias;                        // [NE] selection bias (nullptr: none)
    int NE, top;
    int* sel;                                 // [T][top] expert index
    float* wgt;                               // [T][top]
    MetaView meta;
    int mode = 0;                             // MOE_SOFTMAX_ALL | MOE_TOP_LOGITS | MOE_SIGMOID_GROUPS
    int groups = 0, keep = 0;                 // MOE_SIGMOID_GROUPS: equal groups of neighbouring experts, groups that stay eligible (0: no groups)
};

// MOE_SOFTMAX_ALL: probabilities over all outputs, choice by probability + bias, weights = the chosen probabilities as they are.
// MOE_TOP_LOGITS:  bias is part of the logits; the `top` largest logits are chosen, weights = softmax over the chosen logits only.
// MOE_SIGMOID_GROUPS: scores = sigmoid(logit); a group of neighbouring experts is judged by the sum of its two largest scores and
//                  only experts of the `keep` best groups are eligible; the `top` largest eligible scores are chosen, weights =
//                  the chosen scores over their sum.
enum MoeRouteMode { MOE_SOFTMAX_ALL = 0, MOE_TOP_LOGITS = 1, MOE_SIGMOID_GROUPS = 2 };

// Threads of a token's CTA.  Few tokens (decode): 32 warps, so that a warp has its outputs' rows requested in one or two turns (sixteen tokens, width 2048: 12.8 us of the step with
// eight, 8.5); many, or narrow rows: eight, the CTAs of other tokens cover the waits (2000 tokens: 46 us with 32, 38; a step of 64 tokens, four layers of width 128, 338 with 32, 321).
inline int moe_route_threads(int rows, int W) { return rows <= 128 && W >= 384 ? 1024 : 256; }
__host__ __device__ inline int moe_route_row(int K) { return (K + 255) & ~255; }
__host__ __device__ inline size_t moe_route_smem(int K, int NE) { return ((size_t)moe_route_row(K) + 3 * (size_t)NE) * sizeof(float); }

// warp-wide arg-max over a[0 .. n) in shared memory (ties: lower index); the winner's entry becomes -inf so that the next call
// finds the runner-up.  Every lane returns the same (index, value).
__device__ __forceinline__ int moe_warp_take_max(float* a, int n, float& val) {
    const int lane = threadIdx.x & 31;
    float best = -CUDART_INF_F; int bi = 0x7fffffff;
    for (int e = lane; e < n; e += 32) {
        const float c = a[e];
        if (c > best || (c == best && e < bi)) { best = c; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    __syncwarp();
    if (lane == 0 && bi < n) a[bi] = -CUDART_INF_F;
    __syncwarp();
    val = best;
    return bi;
}

// One CTA per token: router logits in f32 on the f32 row (every warp takes outputs warp, warp + NW, ...), then warp 0 turns them
// into the choice: softmax, + selection bias, `top` largest, weights = the unbiased probabilities.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) moe_route_kernel(const MoeRouteParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float moe_route_sm[];
    float* sh = moe_route_sm;                 // [K]
    float* z = sh + moe_route_row(p.K);       // [NE]
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = p.K;
    const bool vec = (K % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.Wr) & 15) == 0);
    // vec: the eight columns of a lane in two halves, so that a warp reads 512 bytes in a row (eight words of a lane side by side: every read of a word met eight lanes in a bank,
    // 50 us of a prompt step of 2000 tokens, 38 now)
#pragma unroll 4
    for (int k = threadIdx.x; k < K; k += blockDim.x) sh[vec ? (k & ~255) + (k & 4) * 32 + ((k >> 3) & 31) * 4 + (k & 3) : k] = p.h[(size_t)t * p.ldh + k];
    __syncthreads();
    constexpr int NW = THREADS / 32;
    for (int e0 = warp; e0 < p.NE; e0 += 2 * NW) {          // two outputs at a time
        const int e1 = min(e0 + NW, p.NE - 1);
        const __nv_bfloat16 *w0 = p.Wr + (size_t)e0 * K, *w1 = p.Wr + (size_t)e1 * K;
        float acc[2] = {0.f, 0.f};
        if (vec) {
#pragma unroll 4
            for (int k = lane * 8; k < K; k += 256) {
                const uint4 q[2] = {__ldg(reinterpret_cast<const uint4*>(w0 + k)), __ldg(reinterpret_cast<const uint4*>(w1 + k))};
                const float4 a = *reinterpret_cast<const float4*>(sh + (k & ~255) + 4 * lane), b = *reinterpret_cast<const float4*>(sh + (k & ~255) + 128 + 4 * lane);
                const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const __nv_bfloat162* hq = reinterpret_cast<const __nv_bfloat162*>(&q[i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __bfloat1622float2(hq[j]);
                        acc[i] = fmaf(f.x, x[2 * j], acc[i]);
                        acc[i] = fmaf(f.y, x[2 * j + 1], acc[i]);
                    }
                }
            }
        } else {
            for (int k = lane; k < K; k += 32) { acc[0] = fmaf(__bfloat162float(w0[k]), sh[k], acc[0]); acc[1] = fmaf(__bfloat162float(w1[k]), sh[k], acc[1]); }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o); acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o); }
        if (lane < 2 && e0 + lane * NW < p.NE) {
            const int e = e0 + lane * NW;
            z[e] = (lane ? acc[1] : acc[0]) + (p.mode == MOE_TOP_LOGITS && p.bias ? p.bias[e] : 0.f);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    if (p.mode == MOE_SIGMOID_GROUPS) {
        float* ms = z + p.NE;                 // [NE] scores still eligible (-inf: not, or already chosen)
        float* gs = ms + p.NE;                // [groups] group scores; a kept group's entry ends as -inf
        for (int e = lane; e < p.NE; e += 32) { const float s = 1.f / (1.f + expf(-z[e])); z[e] = s; ms[e] = s; }
        __syncwarp();
        if (p.groups > 0) {
            const int per = p.NE / p.groups;
            for (int g = lane; g < p.groups; g += 32) {
                float a = -CUDART_INF_F, b = -CUDART_INF_F;          // the two largest of the group
                for (int e = g * per; e < (g + 1) * per; ++e) {
                    const float s = z[e];
                    if (s > a) { b = a; a = s; } else if (s > b) b = s;
                }
                gs[g] = per > 1 ? a + b : a;
            }
            __syncwarp();
            for (int k = 0; k < p.keep; ++k) {             // taking a maximum leaves -inf in its place (every score is finite)
                float v;
                (void)moe_warp_take_max(gs, p.groups, v);
            }
            for (int e = lane; e < p.NE; e += 32)
                if (gs[e / per] != -CUDART_INF_F) ms[e] = -CUDART_INF_F;   // its group was not kept
            __syncwarp();
        }
        int idx[MOE_MAX_TOP];
        float sc[MOE_MAX_TOP], sum = 0.f;
        for (int k = 0; k < p.top; ++k) {
            float v;
            idx[k] = moe_warp_take_max(ms, p.NE, v);
            sc[k] = z[min(idx[k], p.NE - 1)];
            sum += sc[k];
        }
        if (lane == 0)
            for (int k = 0; k < p.top; ++k) {
                p.sel[(size_t)t * p.top + k] = idx[k];
                p.wgt[(size_t)t * p.top + k] = sc[k] / (sum + 1e-20f);
            }
        return;
    }
    if (p.mode == MOE_TOP_LOGITS) {
        unsigned long long taken = 0ull;
        float zs[MOE_MAX_TOP];
        float top_max = -CUDART_INF_F;
        for (int k = 0; k < p.top; ++k) {
            float best = -CUDART_INF_F; int bi = 0x7fffffff;
            for (int e = lane, i = 0; e < p.NE; e += 32, ++i) {
                if ((taken >> i) & 1ull) continue;
                const float c = z[e];
                if (c > best || (c == best && e < bi)) { best = c; bi = e; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            if ((bi & 31) == lane) taken |= 1ull << (bi >> 5);
            if (lane == 0) p.sel[(size_t)t * p.top + k] = bi;
            zs[k] = best;
            if (k == 0) top_max = best;
        }
        float sum = 0.f;
        for (int k = 0; k < p.top; ++k) sum += expf(zs[k] - top_max);
        if (lane == 0)
            for (int k = 0; k < p.top; ++k) p.wgt[(size_t)t * p.top + k] = expf(zs[k] - top_max) / sum;
        return;
    }
    float mx = -CUDART_INF_F;
    for (int e = lane; e < p.NE; e += 32) mx = fmaxf(mx, z[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
    for (int e = lane; e < p.NE; e += 32) sum += expf(z[e] - mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = 1.f / sum;
    unsigned long long taken_lo = 0ull;       // lanes keep their own "already chosen" marks: expert e = lane + 32 * i -> bit i
    for (int k = 0; k < p.top; ++k) {
        float best = -CUDART_INF_F; int bi = 0x7fffffff;
        for (int e = lane, i = 0; e < p.NE; e += 32, ++i) {
            if ((taken_lo >> i) & 1ull) continue;
            const float c = expf(z[e] - mx) * inv + (p.bias ? p.bias[e] : 0.f);
            if (c > best || (c == best && e < bi)) { best = c; bi = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if ((bi & 31) == lane) taken_lo |= 1ull << (bi >> 5);
        if (lane == 0) {
            p.sel[(size_t)t * p.top + k] = bi;
            p.wgt[(size_t)t * p.top + k] = expf(z[bi] - mx) * inv;
        }
    }
}

struct MoeGroupParams {
    const int* sel; int top, E;               // real experts are 0 .. E-1
    int* cnt; int* off; int* list;            // [E], [E], [T * top]
    int* row_of;                              // [T][top] compact row or -1
    MetaView meta;
};

__global__ void __launch_bounds__(256) moe_group_kernel(const MoeGroupParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ int moe_smem[];         // [E] counts, [E] offsets, [T * top] choices
    int* s_cnt = moe_smem;
    int* s_off = s_cnt + p.E;
    int* s_sel = s_off + p.E;
    const int T = p.meta.T(), n = T * p.top;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s_sel[i] = p.sel[i];
    __syncthreads();
    // a warp per expert: ballots over 32 choices at a time keep the token order without a serial scan
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int e = warp; e < p.E; e += nw) {
        int c = 0;
        for (int i0 = 0; i0 < n; i0 += 32) c += __popc(__ballot_sync(0xffffffffu, i0 + lane < n && s_sel[i0 + lane] == e));
        if (lane == 0) s_cnt[e] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int e = 0; e < p.E; ++e) { s_off[e] = acc; acc += s_cnt[e]; }
    }
    __syncthreads();
    for (int e = warp; e < p.E; e += nw) {
        if (lane == 0) { p.cnt[e] = s_cnt[e]; p.off[e] = s_off[e]; }
        int w = s_off[e];
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool hit = i < n && s_sel[i] == e;
            const unsigned mask = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                const int pos = w + __popc(mask & ((1u << lane) - 1u));
                p.list[pos] = i / p.top;
                p.row_of[i] = pos;
            }
            w += __popc(mask);
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (s_sel[i] >= p.E) p.row_of[i] = -1;
}

// The same for steps of more than 128 tokens and up to 256 experts: a warp walks every choice once per expert above (60 us for 2048 tokens with four choices each); here
// every warp takes its own 1 / 32 of the choices, lanes that chose the same expert find one another (match), and counts per warp become first places.
constexpr int MOE_GROUP_THREADS = 1024, MOE_GROUP_MAX_E = 256;
__host__ __device__ inline size_t moe_group_wide_smem(int E) { return (size_t)(MOE_GROUP_THREADS / 32 + 1) * E * sizeof(int); }

__global__ void __launch_bounds__(MOE_GROUP_THREADS) moe_group_wide_kernel(const MoeGroupParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ int moe_smem[];         // [32 warps][E] counts, then first places; [E] totals
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = p.meta.T() * p.top, E = p.E;
    const int seg = ((n + 31) / 32 + 31) & ~31, i0 = min(n, warp * seg), i1 = min(n, i0 + seg);
    int* const mine = moe_smem + warp * E;
    int* const total = moe_smem + 32 * E;
    for (int e = lane; e < E; e += 32) mine[e] = 0;
    __syncwarp();
    auto walk = [&](auto&& each) {
        for (int b = i0; b < i1; b += 32) {
            const int i = b + lane, c = i < i1 ? p.sel[i] : -1, e = c < E ? c : -1;
            const unsigned same = __match_any_sync(0xffffffffu, e);
            each(i, e, same);
            __syncwarp();
            if (e >= 0 && lane == __ffs(same) - 1) mine[e] += __popc(same);
            __syncwarp();
        }
    };
    walk([](int, int, unsigned) {});
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += MOE_GROUP_THREADS) {
        int s = 0;
        for (int w = 0; w < 32; ++w) { const int c = moe_smem[w * E + e]; moe_smem[w * E + e] = s; s += c; }
        total[e] = s;
        p.cnt[e] = s;
    }
    __syncthreads();
    if (warp == 0) {
        int acc = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int c = e0 + lane < E ? total[e0 + lane] : 0;
            int upto = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (e0 + lane < E) { total[e0 + lane] = acc + upto - c; p.off[e0 + lane] = acc + upto - c; }
            acc += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    __syncthreads();
    walk([&](int i, int e, unsigned same) {
        if (i >= i1) return;
        const int pos = e >= 0 ? total[e] + mine[e] + __popc(same & ((1u << lane) - 1u)) : -1;
        p.row_of[i] = pos;
        if (e >= 0) p.list[pos] = i / p.top;
    });
}

struct MoeCombineParams {
    float* x;                                 // [T, W] residual, accumulated in place
    const float* h;                           // [T, W] the feed-forward's input
    const float* gate;  int ldg;              // [T, W] residual gate of the feed-forward
    const float* rows;                        // [T * top, W] expert outputs, compact rows
    const int* row_of; const float* wgt; int top;
    const float* shared;                      // [T, W] shared expert output (nullptr: none)
    const __nv_bfloat16* sg;                  // [W] shared-expert gate vector
    int W;
    MetaView meta;
};

// A thread takes four neighbouring columns and requests all that they need at once, the experts' rows among it (column after column, a round trip to memory each: 20 us of a decode step
// of sixteen tokens, width 2048, four experts, and 76 of a prompt step of 2000, now 3 and 39).  Widths that are no multiple of four, or wider than the CTA: column after column.
constexpr int MOE_COMBINE_MAX = 1024;
inline int moe_combine_threads(int W) { return W % 4 == 0 && W / 4 <= MOE_COMBINE_MAX ? std::max(64, (W / 4 + 31) / 32 * 32) : 256; }

__global__ void __launch_bounds__(MOE_COMBINE_MAX) moe_combine_kernel(const MoeCombineParams p) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[32];
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    const int W = p.W;
    float sgate = 0.f;
    if (W % 4 == 0 && W / 4 <= (int)blockDim.x && p.ldg % 4 == 0 && row_whole(p.x) && row_whole(p.h) && row_whole(p.gate) && row_whole(p.rows) && row_whole(p.shared) && row_whole(p.sg, 8)) {
        const int c = 4 * threadIdx.x;
        const bool in = c < W;
        const size_t at = (size_t)t * W + c;
        int rows[MOE_MAX_TOP]; float wg[MOE_MAX_TOP];
#pragma unroll
        for (int k = 0; k < MOE_MAX_TOP; ++k)
            if (k < p.top) { rows[k] = p.row_of[(size_t)t * p.top + k]; wg[k] = p.wgt[(size_t)t * p.top + k]; }
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 h = in ? *reinterpret_cast<const float4*>(p.h + at) : none;
        const float4 g = in ? *reinterpret_cast<const float4*>(p.gate + (size_t)t * p.ldg + c) : none;
        const float4 sh = in && p.shared ? *reinterpret_cast<const float4*>(p.shared + at) : none;
        const float4 sg = in && p.shared ? row_bf16(__ldg(reinterpret_cast<const uint2*>(p.sg + c))) : none;
        float4 x = in ? *reinterpret_cast<const float4*>(p.x + at) : none, e[MOE_MAX_TOP];
#pragma unroll
        for (int k = 0; k < MOE_MAX_TOP; ++k)
            if (k < p.top && in) e[k] = rows[k] >= 0 ? *reinterpret_cast<const float4*>(p.rows + (size_t)rows[k] * W + c) : h;
        if (p.shared) sgate = 1.f / (1.f + expf(-rms_block_sum(row_dot(sg, h, 0.f), red)));
        if (!in) return;
        float4 f = none;
#pragma unroll
        for (int k = 0; k < MOE_MAX_TOP; ++k)
            if (k < p.top) { f.x = fmaf(wg[k], e[k].x, f.x); f.y = fmaf(wg[k], e[k].y, f.y); f.z = fmaf(wg[k], e[k].z, f.z); f.w = fmaf(wg[k], e[k].w, f.w); }
        if (p.shared) { f.x = fmaf(sgate, sh.x, f.x); f.y = fmaf(sgate, sh.y, f.y); f.z = fmaf(sgate, sh.z, f.z); f.w = fmaf(sgate, sh.w, f.w); }
        x.x += g.x * f.x; x.y += g.y * f.y; x.z += g.z * f.z; x.w += g.w * f.w;
        *reinterpret_cast<float4*>(p.x + at) = x;
        return;
    }
    if (p.shared) {
        float d = 0.f;
        for (int c = threadIdx.x; c < W; c += blockDim.x) d = fmaf(__bfloat162float(p.sg[c]), p.h[(size_t)t * W + c], d);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = d;
        __syncthreads();
        d = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) d += red[w];
        sgate = 1.f / (1.f + expf(-d));
    }
    int rows[MOE_MAX_TOP]; float wg[MOE_MAX_TOP];
#pragma unroll
    for (int k = 0; k < MOE_MAX_TOP; ++k)
        if (k < p.top) { rows[k] = p.row_of[(size_t)t * p.top + k]; wg[k] = p.wgt[(size_t)t * p.top + k]; }
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        float f = 0.f;
#pragma unroll
        for (int k = 0; k < MOE_MAX_TOP; ++k)
            if (k < p.top) f = fmaf(wg[k], rows[k] >= 0 ? p.rows[(size_t)rows[k] * W + c] : p.h[(size_t)t * W + c], f);
        if (p.shared) f = fmaf(sgate, p.shared[(size_t)t * W + c], f);
        p.x[(size_t)t * W + c] += p.gate[(size_t)t * p.ldg + c] * f;
    }
}

}  // namespace b200
