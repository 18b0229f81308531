// Residual update + LayerNorm + token shift + static lerps, one 256-thread group per token.
//
// Replaces web-rwkv's `layer_norm`, `token_shift` and `add` WGSL dispatches on the path
// `Runtime::infer` (reference run.rs:1143).  Fused so the
// residual stream makes one HBM/L2 round trip per half-layer:
//     x_out = x_in + gate (.) sum_p part[p]            (projection results of the previous
//                                                       half-layer, one partial per TP rank)
//     xx    = LN(x_out)                                 eps 1e-5
//     prev  = first token of its slot ? shift_state[slot] : LN(x_out[t-1])   (recomputed)
//     sx    = prev - xx
//     mix_j = f16(xx + sx * mu_j)  -> A16 operand buffers of the following projections
// The shift state of the PREVIOUS LN stage is committed here (dst <- last token's xx), which
// keeps every state write strictly after all reads of the old value with no extra launch.
//
// Code shape: only a handful of CTAs run these rows and everything they touch sits at L2 latency
// (~0.5 us per dependent round trip), so the row lives in registers and every batch of loads is
// issued together; parameters that do not depend on the phase are requested before the reductions.
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int LN_THREADS = 256;
constexpr int LN_MAXC = 8192;       // largest row the stand-alone kernels buffer
constexpr float LN_EPS = 1e-5f;

struct LnMixParams {
    const float* x_in;      // [T, C]
    float* x_out;           // [T, C] (may alias x_in only when n_parts == 0)
    int C;
    MetaView meta;
    int n_parts;
    const float* parts[8];  // [T, C] each
    int n_gate;             // 0 = no gate; else column-blocked gate, one block per TP rank
    int gate_cl;            // columns per gate block (C / n_gate)
    const float* gates[8];  // [T, gate_cl] each
    const float* ln_w;
    const float* ln_b;
    const float* shift_state;   // [S, C] rows of this layer / kind
    int n_mix;
    const float* mu[6];
    __half* mix_out[6];
    int kq_tile;            // th: token rows of this step's A16 operands (16 x token tiles; 32 with split operands)
    float* xx_out;          // [T, C]
    float* sx_out;          // [T, C] or null
    float* commit_dst;      // [S, C] or null
    const float* commit_src;    // [T, C]
    unsigned long long* trace;  // profiling aid (null in production)
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void add4(float4& a, const float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

// residual source shared by the LN stages: x_in + gate (.) sum_p parts[p]
struct ResidualSrc {     // held by value: pointers into kernel-parameter space would turn into slow generic loads
    const float* x_in;
    int C, n_parts, n_gate, gate_cl;
    const float* parts[8];
    const float* gates[8];
};
template <typename P>
__device__ __forceinline__ ResidualSrc make_residual_src(const P& p) {
    ResidualSrc r;
    r.x_in = p.x_in; r.C = p.C; r.n_parts = p.n_parts; r.n_gate = p.n_gate; r.gate_cl = p.gate_cl;
#pragma unroll
    for (int i = 0; i < 8; ++i) { r.parts[i] = p.parts[i]; r.gates[i] = p.gates[i]; }
    return r;
}

// Row t of the updated residual into a[NV] (thread owns columns 4*(tid + 256 j)).  Memory-level
// parallelism is what matters here (a handful of CTAs, everything L2-latency bound): all loads of
// a batch (x + 4 partials, then 4 more partials + gate) are in flight together.
template <int NV>
__device__ __forceinline__ void residual_row(const ResidualSrc& r, const int t, float4 (&a)[NV]) {
    const int C = r.C;
    const size_t base = (size_t)t * C;
    float4 s[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        a[j] = (c < C) ? ld4(r.x_in + base + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        s[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (r.n_parts == 0) return;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (half * 4 >= r.n_parts) break;
        float4 v[4][NV];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const int c = 4 * (threadIdx.x + LN_THREADS * j);
                v[q][j] = (half * 4 + q < r.n_parts && c < C) ? ld4(r.parts[half * 4 + q] + base + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
        for (int q = 0; q < 4; ++q)        // fixed order: deterministic, identical on all ranks
#pragma unroll
            for (int j = 0; j < NV; ++j) add4(s[j], v[q][j]);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        if (r.n_gate > 0 && c < C) {
            const int gb = c / r.gate_cl;
            const float4 gt = ld4(r.gates[gb] + (size_t)t * r.gate_cl + (c - gb * r.gate_cl));
            s[j].x *= gt.x; s[j].y *= gt.y; s[j].z *= gt.z; s[j].w *= gt.w;
        }
        add4(a[j], s[j]);
    }
}

// two-pass mean / rstd of a row held in registers
template <int NV>
__device__ __forceinline__ void row_stats(const int C, const float4 (&a)[NV], float* red, float& mean, float& rstd) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) s += (a[j].x + a[j].y) + (a[j].z + a[j].w);
    mean = block_sum(s, red) / (float)C;
    float s2 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        if (c < C) {
            const float dx = a[j].x - mean, dy = a[j].y - mean, dz = a[j].z - mean, dw = a[j].w - mean;
            s2 += (dx * dx + dy * dy) + (dz * dz + dw * dw);
        }
    }
    const float var = block_sum(s2, red) / (float)C;
    rstd = 1.0f / sqrtf(var + LN_EPS);
}

__device__ __forceinline__ float4 ln_apply(const float4 a, const float mean, const float rstd, const float4 w, const float4 b) {
    float4 o;
    o.x = (a.x - mean) * rstd * w.x + b.x;
    o.y = (a.y - mean) * rstd * w.y + b.y;
    o.z = (a.z - mean) * rstd * w.z + b.z;
    o.w = (a.w - mean) * rstd * w.w + b.w;
    return o;
}

template <int NV>
__device__ __forceinline__ void ln_mix_row_nv(const LnMixParams& p, const int t, float* red, unsigned long long* stamps = nullptr) {
    auto stamp = [&](int i) { if (stamps && threadIdx.x == 0) stamps[i] = globaltimer_ns(); };
    stamp(0);
    const int C = p.C;
    const int slot = p.meta.tok_slot()[t];
    const int prev_t = p.meta.tok_prev()[t];
    const bool last = p.meta.tok_last()[t] != 0;
    const ResidualSrc r = make_residual_src(p);
    float4 a[NV], w[NV], b[NV], pv[NV];
    stamp(1);
    residual_row<NV>(r, t, a);
    stamp(2);
    // LN parameters and the shift state do not depend on this phase: request them before the
    // reductions so their latency hides behind the two block sums
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        const bool ok = c < C;
        w[j] = ok ? ld4(p.ln_w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        b[j] = ok ? ld4(p.ln_b + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        pv[j] = (ok && prev_t < 0) ? ld4(p.shift_state + (size_t)slot * C + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (p.x_out != p.x_in || p.n_parts > 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (threadIdx.x + LN_THREADS * j);
            if (c < C) *reinterpret_cast<float4*>(p.x_out + (size_t)t * C + c) = a[j];
        }
    }
    float mean, rstd;
    stamp(3);
    row_stats<NV>(C, a, red, mean, rstd);
    stamp(4);
    if (prev_t >= 0) {          // multi-token slot (prefill): previous token's LN output, recomputed
        float pmean, prstd;
        residual_row<NV>(r, prev_t, pv);
        row_stats<NV>(C, pv, red, pmean, prstd);
#pragma unroll
        for (int j = 0; j < NV; ++j) pv[j] = ln_apply(pv[j], pmean, prstd, w[j], b[j]);
    }
    float4 sx[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        a[j] = ln_apply(a[j], mean, rstd, w[j], b[j]);       // xx
        sx[j].x = pv[j].x - a[j].x; sx[j].y = pv[j].y - a[j].y; sx[j].z = pv[j].z - a[j].z; sx[j].w = pv[j].w - a[j].w;
        if (c < C) {
            *reinterpret_cast<float4*>(p.xx_out + (size_t)t * C + c) = a[j];
            if (p.sx_out) *reinterpret_cast<float4*>(p.sx_out + (size_t)t * C + c) = sx[j];
            if (last && p.commit_dst)
                *reinterpret_cast<float4*>(p.commit_dst + (size_t)slot * C + c) = ld4(p.commit_src + (size_t)t * C + c);
        }
    }
    stamp(5);
#pragma unroll 1
    for (int m = 0; m < p.n_mix; ++m) {
        const float* mup = p.mu[m];
        __half* outp = p.mix_out[m];
        float4 mu[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (threadIdx.x + LN_THREADS * j);
            mu[j] = (c < C) ? ld4(mup + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (threadIdx.x + LN_THREADS * j);
            if (c < C) {
                uint2 o;
                o.x = pack_h2(a[j].x + sx[j].x * mu[j].x, a[j].y + sx[j].y * mu[j].y);
                o.y = pack_h2(a[j].z + sx[j].z * mu[j].z, a[j].w + sx[j].w * mu[j].w);
                *reinterpret_cast<uint2*>(outp + a16_index(t, c, p.kq_tile)) = o;
            }
        }
    }
}

__device__ __forceinline__ void ln_mix_row(const LnMixParams& p, const int t, float* red, unsigned long long* stamps = nullptr) {
    const int nv = (p.C + 4 * LN_THREADS - 1) / (4 * LN_THREADS);
    if (nv <= 1) ln_mix_row_nv<1>(p, t, red);
    else if (nv == 2) ln_mix_row_nv<2>(p, t, red);
    else if (nv <= 4) ln_mix_row_nv<4>(p, t, red, stamps);
    else ln_mix_row_nv<8>(p, t, red);
    if (stamps && threadIdx.x == 0) stamps[6] = globaltimer_ns();
}

__global__ void __launch_bounds__(LN_THREADS) ln_mix_kernel(const __grid_constant__ LnMixParams p) {
    __shared__ float red[32];
    trace_stamp(p.trace, 0);
    pdl_launch_dependents();
    pdl_wait();
    trace_stamp(p.trace, 1);
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    ln_mix_row(p, t, red);
    trace_stamp(p.trace, 7);
}

// Steps of more than 16 tokens: LN_ROWS neighbouring tokens to a CTA, a group of LN_THREADS threads per row and one for the row before
// them.  A token's shift partner is the normed row of the token before it: ln_mix_kernel computes it a second time, after its own row, so a
// launch was two dependent chains of loads and reductions and read every partial sum twice (18-23 us for 256 rows of 2560 with 5-7
// partial sums); here the rows' chains run side by side and the partner is in shared memory.  Same sums in the same order.
constexpr int LN_ROWS = 2, LN_ROWS_THREADS = (LN_ROWS + 1) * LN_THREADS;

template <int NV>
__device__ __forceinline__ void ln_mix_rows_nv(const LnMixParams& p, const int t0, float* rows, float* red) {
    const int C = p.C, T = p.meta.T(), g = threadIdx.x / LN_THREADS, tid = threadIdx.x % LN_THREADS, lane = tid & 31, warp = tid >> 5;
    const int t = t0 - 1 + g;                                  // group 0: the row before
    const bool live = t >= 0 && t < T && (g > 0 || (t0 < T && p.meta.tok_prev()[t0] >= 0));
    auto group_sum = [&](float v) {                            // block_sum of the group's LN_THREADS threads
        v = warp_sum(v);
        named_bar_sync(1 + g, LN_THREADS);
        if (lane == 0) red[g * 8 + warp] = v;
        named_bar_sync(1 + g, LN_THREADS);
        return warp_sum(lane < LN_THREADS / 32 ? red[g * 8 + lane] : 0.f);
    };
    float4 a[NV];
    if (live) {
        const size_t base = (size_t)t * C;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (tid + LN_THREADS * j);
            a[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c >= C) continue;
            a[j] = ld4(p.x_in + base + c);
            if (p.n_parts == 0) continue;
            float4 v[8], s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = q < p.n_parts ? ld4(p.parts[q] + base + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) add4(s, v[q]);         // fixed order, identical on all ranks
            if (p.n_gate > 0) {
                const int gb = c / p.gate_cl;
                const float4 gt = ld4(p.gates[gb] + (size_t)t * p.gate_cl + (c - gb * p.gate_cl));
                s.x *= gt.x; s.y *= gt.y; s.z *= gt.z; s.w *= gt.w;
            }
            add4(a[j], s);
        }
        if (g > 0 && (p.x_out != p.x_in || p.n_parts > 0)) {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const int c = 4 * (tid + LN_THREADS * j);
                if (c < C) *reinterpret_cast<float4*>(p.x_out + base + c) = a[j];
            }
        }
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) s1 += (a[j].x + a[j].y) + (a[j].z + a[j].w);
        const float mean = group_sum(s1) / (float)C;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (4 * (tid + LN_THREADS * j) >= C) continue;
            const float dx = a[j].x - mean, dy = a[j].y - mean, dz = a[j].z - mean, dw = a[j].w - mean;
            s2 += (dx * dx + dy * dy) + (dz * dz + dw * dw);
        }
        const float rstd = 1.0f / sqrtf(group_sum(s2) / (float)C + LN_EPS);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (tid + LN_THREADS * j);
            if (c >= C) continue;
            a[j] = ln_apply(a[j], mean, rstd, ld4(p.ln_w + c), ld4(p.ln_b + c));
            *reinterpret_cast<float4*>(rows + (size_t)g * C + c) = a[j];
        }
    }
    __syncthreads();
    if (!live || g == 0) return;
    const int slot = p.meta.tok_slot()[t];
    const bool shared = p.meta.tok_prev()[t] >= 0, commit = p.meta.tok_last()[t] != 0 && p.commit_dst;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (tid + LN_THREADS * j);
        if (c >= C) continue;
        const float4 pv = shared ? *reinterpret_cast<const float4*>(rows + (size_t)(g - 1) * C + c) : ld4(p.shift_state + (size_t)slot * C + c);
        const float4 sx = make_float4(pv.x - a[j].x, pv.y - a[j].y, pv.z - a[j].z, pv.w - a[j].w);
        *reinterpret_cast<float4*>(p.xx_out + (size_t)t * C + c) = a[j];
        if (p.sx_out) *reinterpret_cast<float4*>(p.sx_out + (size_t)t * C + c) = sx;
        if (commit) *reinterpret_cast<float4*>(p.commit_dst + (size_t)slot * C + c) = ld4(p.commit_src + (size_t)t * C + c);
#pragma unroll 2
        for (int m = 0; m < p.n_mix; ++m) {
            const float4 mu = ld4(p.mu[m] + c);
            *reinterpret_cast<uint2*>(p.mix_out[m] + a16_index(t, c, p.kq_tile)) =
                make_uint2(pack_h2(a[j].x + sx.x * mu.x, a[j].y + sx.y * mu.y), pack_h2(a[j].z + sx.z * mu.z, a[j].w + sx.w * mu.w));
        }
    }
}

__global__ void __launch_bounds__(LN_ROWS_THREADS) ln_mix_rows_kernel(const __grid_constant__ LnMixParams p) {
    extern __shared__ __align__(16) float ln_rows[];
    __shared__ float red[(LN_ROWS + 1) * 8];
    trace_stamp(p.trace, 0);
    pdl_launch_dependents();
    pdl_wait();
    trace_stamp(p.trace, 1);
    const int t0 = blockIdx.x * LN_ROWS, nv = (p.C + 4 * LN_THREADS - 1) / (4 * LN_THREADS);
    if (t0 >= p.meta.T()) return;
    if (nv <= 1) ln_mix_rows_nv<1>(p, t0, ln_rows, red);
    else if (nv == 2) ln_mix_rows_nv<2>(p, t0, ln_rows, red);
    else if (nv <= 3) ln_mix_rows_nv<3>(p, t0, ln_rows, red);
    else if (nv <= 4) ln_mix_rows_nv<4>(p, t0, ln_rows, red);
    else ln_mix_rows_nv<8>(p, t0, ln_rows, red);
    trace_stamp(p.trace, 7);
}

// Long prompt steps: TALL_ROWS tokens to a CTA and the one before them, 64 threads a row, rows in shared memory (so that few registers are held and two CTAs of 2560 columns
// share an SM: sixteen rows' loads in flight).  The row before is read again by one token in seven instead of one in two, and the f16 operands leave eight channels of
// eight tokens at a time: runs of 112 bytes where a thread of the form above leaves 8.
// Bytes bound it: 2048 rows of 2560 with one partial sum and a gate, 120 to 140 MB: in place 46 -> 29 us.
constexpr int TALL_ROWS = 7, TALL_GROUP = 64, TALL_THREADS = (TALL_ROWS + 1) * TALL_GROUP, TALL_PAD = 4;      // pad: eight rows' 16 bytes lie in different banks
__host__ __device__ inline size_t ln_tall_smem(int C) { return (size_t)(TALL_ROWS + 1) * (C + TALL_PAD) * 4; }

// the updated residual of row t, 64 threads: put(c, four entries) for every four columns
template <typename F>
__device__ __forceinline__ void tall_residual(const ResidualSrc& r, const int t, const int l, F&& put) {
    constexpr int U = 3;
    const size_t base = (size_t)t * r.C;
    for (int c0 = 4 * l; c0 < r.C; c0 += 4 * TALL_GROUP * U) {
        float4 a[U], s[U], v[2][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + 4 * TALL_GROUP * u;
            a[u] = c < r.C ? ld4(r.x_in + base + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            s[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (r.n_parts > 0) {
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                if (q >= r.n_parts) break;
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int c = c0 + 4 * TALL_GROUP * u;
                        v[e][u] = q + e < r.n_parts && c < r.C ? ld4(r.parts[q + e] + base + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                for (int e = 0; e < 2; ++e)        // fixed order, identical on all ranks
#pragma unroll
                    for (int u = 0; u < U; ++u) add4(s[u], v[e][u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int c = c0 + 4 * TALL_GROUP * u;
                if (r.n_gate > 0 && c < r.C) {
                    const int gb = r.n_gate > 1 ? c / r.gate_cl : 0;
                    const float* gp = r.gates[0];
#pragma unroll
                    for (int i = 1; i < 8; ++i) gp = (gb == i) ? r.gates[i] : gp;
                    const float4 gt = ld4(gp + (size_t)t * r.gate_cl + (c - gb * r.gate_cl));
                    s[u].x *= gt.x; s[u].y *= gt.y; s[u].z *= gt.z; s[u].w *= gt.w;
                }
                add4(a[u], s[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + 4 * TALL_GROUP * u < r.C) put(c0 + 4 * TALL_GROUP * u, a[u]);
    }
}

// mean and 1 / deviation of a row in shared memory; `bar`: the group's barrier, s1: this thread's sum
__device__ __forceinline__ void tall_stats(const float* row, const int C, const int l, const int bar, float s1, float* red, float& mean, float& rstd) {
    auto sum = [&](float v) {
        v = warp_sum(v);
        named_bar_sync(bar, TALL_GROUP);
        if ((l & 31) == 0) red[l >> 5] = v;
        named_bar_sync(bar, TALL_GROUP);
        return red[0] + red[1];
    };
    mean = sum(s1) / (float)C;
    float s2 = 0.f;
    for (int c = 4 * l; c < C; c += 4 * TALL_GROUP) {
        const float4 a = ld4(row + c);
        const float dx = a.x - mean, dy = a.y - mean, dz = a.z - mean, dw = a.w - mean;
        s2 += (dx * dx + dy * dy) + (dz * dz + dw * dw);
    }
    rstd = 1.0f / sqrtf(sum(s2) / (float)C + LN_EPS);
}

__global__ void __launch_bounds__(TALL_THREADS, 2) ln_mix_tall_kernel(const __grid_constant__ LnMixParams p) {
    extern __shared__ __align__(16) float ln_tall[];
    __shared__ float red[TALL_ROWS + 1][2];
    trace_stamp(p.trace, 0);
    pdl_launch_dependents();
    const int C = p.C, pitch = C + TALL_PAD, T = p.meta.T(), t0 = blockIdx.x * TALL_ROWS, g = threadIdx.x / TALL_GROUP, l = threadIdx.x % TALL_GROUP;
    const int t = t0 - 1 + g;                                  // group 0: the row before
    const bool live = t >= 0 && t < T && (g > 0 || (t0 < T && p.meta.tok_prev()[t0] >= 0));
    pdl_wait();
    trace_stamp(p.trace, 1);
    if (t0 >= T) return;
    if (live) {
        const ResidualSrc r = make_residual_src(p);
        float* const row = ln_tall + (size_t)g * pitch;
        const bool keep = g > 0 && (p.x_out != p.x_in || p.n_parts > 0);
        float s1 = 0.f, mean, rstd;
        tall_residual(r, t, l, [&](const int c, const float4 a) {
            s1 += (a.x + a.y) + (a.z + a.w);
            *reinterpret_cast<float4*>(row + c) = a;
            if (keep) *reinterpret_cast<float4*>(p.x_out + (size_t)t * C + c) = a;
        });
        tall_stats(row, C, l, 1 + g, s1, red[g], mean, rstd);
        for (int c = 4 * l; c < C; c += 4 * TALL_GROUP) *reinterpret_cast<float4*>(row + c) = ln_apply(ld4(row + c), mean, rstd, ld4(p.ln_w + c), ld4(p.ln_b + c));
    }
    __syncthreads();
    // eight channels of a row a thread: rows in neighbouring lanes
    const int rr = threadIdx.x & 7, to = t0 + rr;
    if (rr == TALL_ROWS || to >= T) return;
    const float* const row = ln_tall + (size_t)(rr + 1) * pitch;
    const bool shared = p.meta.tok_prev()[to] >= 0, commit = p.meta.tok_last()[to] != 0 && p.commit_dst;
    const int slot = p.meta.tok_slot()[to];
    const float* const before = shared ? row - pitch : p.shift_state + (size_t)slot * C;
    for (int c = 8 * (threadIdx.x >> 3); c < C; c += TALL_THREADS) {
        float4 a[2], sx[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const bool ok = c + 4 * e < C;
            const float4 pv = ok ? ld4(before + c + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
            a[e] = ok ? ld4(row + c + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
            sx[e] = make_float4(pv.x - a[e].x, pv.y - a[e].y, pv.z - a[e].z, pv.w - a[e].w);
            if (!ok) continue;
            *reinterpret_cast<float4*>(p.xx_out + (size_t)to * C + c + 4 * e) = a[e];
            if (p.sx_out) *reinterpret_cast<float4*>(p.sx_out + (size_t)to * C + c + 4 * e) = sx[e];
            if (commit) *reinterpret_cast<float4*>(p.commit_dst + (size_t)slot * C + c + 4 * e) = ld4(p.commit_src + (size_t)to * C + c + 4 * e);
        }
        for (int m = 0; m < p.n_mix; ++m) {
            uint2 h[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float4 mu = c + 4 * e < C ? ld4(p.mu[m] + c + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
                h[e] = make_uint2(pack_h2(a[e].x + sx[e].x * mu.x, a[e].y + sx[e].y * mu.y), pack_h2(a[e].z + sx[e].z * mu.z, a[e].w + sx[e].w * mu.w));
            }
            __half* const o = p.mix_out[m] + a16_index(to, c, p.kq_tile);
            if (c + 4 < C) *reinterpret_cast<uint4*>(o) = make_uint4(h[0].x, h[0].y, h[1].x, h[1].y);
            else *reinterpret_cast<uint2*>(o) = h[0];
        }
    }
    trace_stamp(p.trace, 7);
}

// ---------------------------------------------------------------------------------------
// Embedding gather + LN0 (reference: web-rwkv embeds on the CPU and runs ln0 on the device,
// here the f16 table lives in HBM and both are one kernel).
// ---------------------------------------------------------------------------------------
struct EmbedParams {
    const __half* emb;     // [V, C]
    int C, V;
    MetaView meta;
    const float* ln_w;
    const float* ln_b;
    float* x_out;          // [T, C]
};

template <int NV>
__device__ __forceinline__ void embed_row_nv(const EmbedParams& p, const int t, float* red) {
    const int C = p.C;
    int tok = p.meta.tok()[t];
    tok = min(max(tok, 0), p.V - 1);
    float4 a[NV], w[NV], b[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        if (c < C) {
            const uint2 raw = *reinterpret_cast<const uint2*>(p.emb + (size_t)tok * C + c);
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
            const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
            a[j] = make_float4(lo.x, lo.y, hi.x, hi.y);
            w[j] = ld4(p.ln_w + c);
            b[j] = ld4(p.ln_b + c);
        } else {
            a[j] = w[j] = b[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    float mean, rstd;
    row_stats<NV>(C, a, red, mean, rstd);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        if (c < C) *reinterpret_cast<float4*>(p.x_out + (size_t)t * C + c) = ln_apply(a[j], mean, rstd, w[j], b[j]);
    }
}

__device__ __forceinline__ void embed_row(const EmbedParams& p, const int t, float* red) {
    const int nv = (p.C + 4 * LN_THREADS - 1) / (4 * LN_THREADS);
    if (nv <= 1) embed_row_nv<1>(p, t, red);
    else if (nv == 2) embed_row_nv<2>(p, t, red);
    else if (nv <= 4) embed_row_nv<4>(p, t, red);
    else embed_row_nv<8>(p, t, red);
}

__global__ void __launch_bounds__(LN_THREADS) embed_ln0_kernel(const __grid_constant__ EmbedParams p) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    embed_row(p, t, red);
}

// ---------------------------------------------------------------------------------------
// Final residual update + ln_out for the rows that need logits (RnnOption::Last -> last token
// of the slot, Full -> every token; reference run.rs:812-822, 710-724), gathered into the A16
// operand of the head GEMM.  Also commits the last layer's channel-mix shift state.
// ---------------------------------------------------------------------------------------
struct LnOutParams {
    const float* x_in;      // [T, C]
    int C;
    MetaView meta;
    int n_parts;
    const float* parts[8];
    int n_gate;
    int gate_cl;
    const float* gates[8];
    const float* ln_w;
    const float* ln_b;
    __half* head_in;        // A16 [R rows, C]
    int kq_tile;
    float* commit_dst;
    const float* commit_src;
    float* hidden_out;      // optional [T, C]: updated residual (hidden states of the embeddings route)
};

template <int NV>
__device__ __forceinline__ void ln_out_row_nv(const LnOutParams& p, const int t, float* red) {
    const int C = p.C;
    const int slot = p.meta.tok_slot()[t];
    const bool last = p.meta.tok_last()[t] != 0;
    const int row = p.meta.tok_outrow()[t];
    if (last && p.commit_dst) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int c = 4 * (threadIdx.x + LN_THREADS * j);
            if (c < C) *reinterpret_cast<float4*>(p.commit_dst + (size_t)slot * C + c) = ld4(p.commit_src + (size_t)t * C + c);
        }
    }
    if (row < 0 && !p.hidden_out) return;
    const ResidualSrc r = make_residual_src(p);
    float4 a[NV], w[NV], b[NV];
    residual_row<NV>(r, t, a);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        const bool ok = c < C;
        w[j] = ok ? ld4(p.ln_w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        b[j] = ok ? ld4(p.ln_b + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (ok && p.hidden_out) *reinterpret_cast<float4*>(p.hidden_out + (size_t)t * C + c) = a[j];
    }
    if (row < 0) return;
    float mean, rstd;
    row_stats<NV>(C, a, red, mean, rstd);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int c = 4 * (threadIdx.x + LN_THREADS * j);
        if (c < C) {
            const float4 y = ln_apply(a[j], mean, rstd, w[j], b[j]);
            uint2 o;
            o.x = pack_h2(y.x, y.y);
            o.y = pack_h2(y.z, y.w);
            *reinterpret_cast<uint2*>(p.head_in + a16_index(row, c, p.kq_tile)) = o;
        }
    }
}

__device__ __forceinline__ void ln_out_row(const LnOutParams& p, const int t, float* red) {
    const int nv = (p.C + 4 * LN_THREADS - 1) / (4 * LN_THREADS);
    if (nv <= 1) ln_out_row_nv<1>(p, t, red);
    else if (nv == 2) ln_out_row_nv<2>(p, t, red);
    else if (nv <= 4) ln_out_row_nv<4>(p, t, red);
    else ln_out_row_nv<8>(p, t, red);
}

__global__ void __launch_bounds__(LN_THREADS) ln_out_kernel(const __grid_constant__ LnOutParams p) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    ln_out_row(p, t, red);
}

// Long prompt steps: a row to 64 threads, eight rows a CTA; few rows have logits, and the others stop at their residual.
// (One row to a CTA whose 256 threads hold eight partial sums each left an SM one row: 54 us for 2048 rows of 2560; now 21.)
__global__ void __launch_bounds__(TALL_THREADS, 2) ln_out_tall_kernel(const __grid_constant__ LnOutParams p) {
    extern __shared__ __align__(16) float ln_tall[];
    __shared__ float red[TALL_ROWS + 1][2];
    pdl_launch_dependents();
    const int C = p.C, g = threadIdx.x / TALL_GROUP, l = threadIdx.x % TALL_GROUP, t = blockIdx.x * (TALL_ROWS + 1) + g;
    const bool live = t < p.meta.T();
    const int slot = live ? p.meta.tok_slot()[t] : 0, out = live ? p.meta.tok_outrow()[t] : -1;
    const bool commit = live && p.meta.tok_last()[t] != 0 && p.commit_dst;
    pdl_wait();
    if (!live) return;
    if (commit)
        for (int c = 4 * l; c < C; c += 4 * TALL_GROUP) *reinterpret_cast<float4*>(p.commit_dst + (size_t)slot * C + c) = ld4(p.commit_src + (size_t)t * C + c);
    if (out < 0 && !p.hidden_out) return;
    const ResidualSrc r = make_residual_src(p);
    float* const row = ln_tall + (size_t)g * (C + TALL_PAD);
    float s1 = 0.f, mean, rstd;
    tall_residual(r, t, l, [&](const int c, const float4 a) {
        s1 += (a.x + a.y) + (a.z + a.w);
        if (out >= 0) *reinterpret_cast<float4*>(row + c) = a;
        if (p.hidden_out) *reinterpret_cast<float4*>(p.hidden_out + (size_t)t * C + c) = a;
    });
    if (out < 0) return;
    tall_stats(row, C, l, 1 + g, s1, red[g], mean, rstd);
    for (int c = 4 * l; c < C; c += 4 * TALL_GROUP) {
        const float4 y = ln_apply(ld4(row + c), mean, rstd, ld4(p.ln_w + c), ld4(p.ln_b + c));
        *reinterpret_cast<uint2*>(p.head_in + a16_index(out, c, p.kq_tile)) = make_uint2(pack_h2(y.x, y.y), pack_h2(y.z, y.w));
    }
}

}  // namespace b200
