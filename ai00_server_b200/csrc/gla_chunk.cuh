// Gated linear attention of prompt steps, sixteen tokens at a time: the recurrence of gla.cuh
//     S_t = diag(alpha_t) S_{t-1} + k_t v_t^T,    o_t = q_scale S_t^T q_t
// over a run of n <= 16 tokens, with b_t the sum of the run's log alpha up to t and S' = diag(e^{b_n}) S_0:
//     q'_t = q_t e^{b_t - b_n},   k'_s = k_s e^{b_n - b_s},   A[t, s] = q'_t . k'_s (s <= t)
//     o_t = q_scale (S'^T q'_t + sum_{s <= t} A[t, s] v_s),    S_n = S' + sum_s k'_s v_s^T
// A run ends before a channel's decays come to less than e^-12, so every factor is a number and its exponent's rounding stays small, and before a decay that is no number, which
// would be a factor of the tokens before it; where that leaves fewer than four tokens (decays of e^-4 a token) the CTA goes token by token instead.
//
// What bounds the token-by-token form (gla.cuh): a chain of products, exchanges and reads a token, about 1400 cycles of an SM for half a head (39 % of the issue slots, no unit busy).
// Here the state's products are MMAs of full height, every f32 number in three bf16 parts (24 bits; six products of parts), sums in f32:
//   * eight warps keep the state in registers (a row of the key dimension in two threads), leave its parts in shared memory, read both products from tensor memory and add
//     the second to the state; the products within a run (A v) are f32 multiply-adds;
//   * eight warps prepare the next run meanwhile: decays, their sums, q', k', A, and the operands' parts.
// Parts of the queries lie side by side, so that a part of the state meets all it needs in one MMA: S_high [q_high, q_mid, q_low], S_mid [q_high, q_mid], S_low [q_high].
// Measured (heads of 128 x 128, sixteen a layer): 256 tokens of eight sequences 256 -> 70 us, 128 of sixteen 184 -> 78, 1000 of one 618 -> 240 (6500 cycles a run of a head; the split of
// the state and its exchange with the tensor core hold it).  Distance from 64 bits (2-norm): read-outs 2.6e-7 -> 1.4e-7, states 2.7e-7 -> 8.8e-8.
#pragma once
#include <math_constants.h>
#include "bf16_parts.cuh"
#include "gla.cuh"
#include "linear_umma.cuh"
#include "mix.cuh"

namespace b200 {

constexpr int GC_RUN = 16, GC_DMAX = 128, GC_THREADS = 512, GC_HALF = GC_THREADS / 2;
constexpr float GC_LEAST = -12.f;
constexpr int GC_SHORT = 4;                                  // runs of fewer tokens go token by token
constexpr int GC_ROWS = 97;                                  // operand rows: three parts of sixteen queries, three of sixteen keys; one more, so that 16 bytes of eight runs lie in different banks
constexpr int GC_PITCH = GC_DMAX + 8;                        // (rows two apart half a turn of the banks apart)
constexpr uint32_t GC_TD1 = 0, GC_TD2 = 128, GC_TMEM_COLS = 256;      // tensor memory: read-outs [2 halves of the channels][3 parts of the queries][16 tokens], the run's addition to the state
// shared memory: state parts [3][16 runs of eight columns][128][16 bytes] | two of {operands [16 runs of eight channels][97][16 bytes] (token by token: q, k, decays [3][16][128]),
// values [16][136], A [16][20], decays [128]} | value parts [3][16 runs][16][16 bytes] | sums of A [8][16][16] | logarithms [16][128]
constexpr int GC_STATE = 3 * 16 * 128 * 16, GC_OPS = 16 * GC_ROWS * 16, GC_VAL = GC_RUN * GC_PITCH * 4, GC_A = GC_RUN * 20 * 4, GC_BUF = GC_OPS + GC_VAL + GC_A + 512, GC_VPARTS = 3 * 16 * 16 * 16;
constexpr int GC_LOGS = GC_RUN * GC_DMAX * 4;
constexpr size_t GC_SMEM = GC_STATE + 2 * GC_BUF + GC_VPARTS + 8 * GC_RUN * GC_RUN * 4 + GC_LOGS + 128;
static_assert(GC_OPS >= 3 * GC_LOGS && GC_BUF % 128 == 0, "token by token the operands' memory holds q, k and the decays");

__device__ __forceinline__ void gc_mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the smaller of two numbers, not a number if either is none (fminf leaves those out)
__device__ __forceinline__ float gc_min(const float a, const float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__global__ void __launch_bounds__(GC_THREADS, 1) gla_chunk_kernel(const __grid_constant__ GlaParams p) {
    extern __shared__ __align__(16) uint8_t gc_smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[6];
    __shared__ uint32_t s_tmem;
    __shared__ int s_n[2];                                   // tokens of the run; negative: token by token
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = smem_u32(s_bar), b_full = bar, b_free = bar + 16, b_d1 = bar + 32, b_d2 = bar + 40;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { mbar_init(b_full + 8 * i, GC_HALF / 32); mbar_init(b_free + 8 * i, 1); }
        mbar_init(b_d1, 1); mbar_init(b_d2, 1);
        mbar_fence_init();
    }
    if (warp == 0) tc_alloc(smem_u32(&s_tmem), GC_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&s_tmem);
    pdl_launch_dependents();                                // behind the allocation: see linear_umma.cuh
    pdl_wait();
    const MetaView& meta = p.norm.meta;
    const int h = blockIdx.x, si = blockIdx.y;
    if (si < meta.nslots()) {
        const int slot = meta.slot_id()[si], t0 = meta.slot_start()[si], nt = meta.slot_count()[si], dk = p.dk, dv = p.dv;
        const uint32_t raw = smem_u32(gc_smem_raw), base = (raw + 127u) & ~127u;
        uint8_t* const g0 = gc_smem_raw + (base - raw);
        uint8_t* const gbuf = g0 + GC_STATE;
        uint8_t* const gvp = gbuf + 2 * GC_BUF;
        float* const sums = reinterpret_cast<float*>(gvp + GC_VPARTS);       // the warps' parts of A
        float* const logs = sums + 8 * GC_RUN * GC_RUN;
        if (warp >= 8) {
            // ===================== the next run's operands: a warp takes two tokens, a lane four channels =====================
            const int w = warp - 8, c4 = 4 * lane;
            auto whole = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
            const float* const kp = p.k + (size_t)t0 * p.ld + (size_t)h * dk + c4;
            const float* const qp = p.q + (size_t)t0 * p.ld + (size_t)h * dk + c4;
            const float* const vp = p.v + (size_t)t0 * p.ld + (size_t)h * dv + c4;
            const float* const zp = p.z + (size_t)t0 * p.ldz + (size_t)h * dk + c4;
            const bool vec = (dk | dv | p.ld | p.ldz) % 4 == 0 && whole(p.k) && whole(p.q) && whole(p.v) && whole(p.z);
            auto load4 = [&](const float* x, const int left) {
                float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
                if (vec) {
                    if (left > 0) r = *reinterpret_cast<const float4*>(x);
                } else {
                    if (left > 0) r.x = x[0];
                    if (left > 1) r.y = x[1];
                    if (left > 2) r.z = x[2];
                    if (left > 3) r.w = x[3];
                }
                return r;
            };
            float4 z[2], q[2], k[2], v[2];
            auto request = [&](const int pos) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = pos + 2 * w + u, lk = t < nt ? dk - c4 : 0, lv = t < nt ? dv - c4 : 0;
                    z[u] = load4(zp + (size_t)t * p.ldz, lk);
                    q[u] = load4(qp + (size_t)t * p.ld, lk);
                    k[u] = load4(kp + (size_t)t * p.ld, lk);
                    v[u] = load4(vp + (size_t)t * p.ld, lv);
                }
            };
            request(0);
            int c = 0;
            for (int pos = 0; pos < nt; ++c) {
                const int b = c & 1, left = nt - pos;
                uint8_t* const ops = gbuf + b * GC_BUF;
                float* const val = reinterpret_cast<float*>(ops + GC_OPS);
                float* const A = val + GC_RUN * GC_PITCH;
                float* const dec = A + GC_RUN * 20;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const bool in = pos + 2 * w + u < nt;
                    auto log_decay = [&](const float x, const int e) {
                        const float g = (fminf(x, 0.f) - log1pf(expf(-fabsf(x)))) * p.inv_tau;
                        return in && c4 + e < dk ? g : 0.f;
                    };
                    *reinterpret_cast<float4*>(logs + (2 * w + u) * GC_DMAX + c4) = make_float4(log_decay(z[u].x, 0), log_decay(z[u].y, 1), log_decay(z[u].z, 2), log_decay(z[u].w, 3));
                }
                named_bar_sync(2, GC_HALF);
                // sums up to every token, and how many tokens the run holds: every warp works it out for all channels
                float4 own[2], sum = make_float4(0.f, 0.f, 0.f, 0.f), g[GC_RUN];
                own[0] = own[1] = sum;
#pragma unroll
                for (int t = 0; t < GC_RUN; ++t) g[t] = *reinterpret_cast<const float4*>(logs + t * GC_DMAX + c4);
                int most = 0;                                // tokens until a sum is too small (sums only fall)
#pragma unroll
                for (int t = 0; t < GC_RUN; ++t) {
                    add4(sum, g[t]);
                    if (t == 2 * w) own[0] = sum;
                    if (t == 2 * w + 1) own[1] = sum;
                    most += gc_min(gc_min(sum.x, sum.y), gc_min(sum.z, sum.w)) >= GC_LEAST;      // (a sum that is no number counts as too small)
                }
                most = __reduce_min_sync(0xffffffffu, most);
                const bool few = most < min(GC_SHORT, left);
                const int n = few ? min(left, GC_RUN) : min(most, left);
                if (n < GC_RUN) {
                    sum = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int t = 0; t < n; ++t) add4(sum, *reinterpret_cast<const float4*>(logs + t * GC_DMAX + c4));
                }
                if (c > 1) mbar_wait(b_free + 8 * b, ((c >> 1) - 1) & 1, 61);
                if (tid == GC_HALF) s_n[b] = few ? -n : n;
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = 2 * w + u;
                    const bool in = t < n;
                    *reinterpret_cast<float4*>(val + t * GC_PITCH + c4) = in ? v[u] : zero;
                    if (few) {
                        const float4 g = *reinterpret_cast<const float4*>(logs + t * GC_DMAX + c4);
                        float* const x = reinterpret_cast<float*>(ops) + t * GC_DMAX + c4;
                        *reinterpret_cast<float4*>(x) = q[u];
                        *reinterpret_cast<float4*>(x + GC_RUN * GC_DMAX) = k[u];
                        *reinterpret_cast<float4*>(x + 2 * GC_RUN * GC_DMAX) = make_float4(expf(g.x), expf(g.y), expf(g.z), expf(g.w));
                        continue;
                    }
                    auto up_to = [&](const float x, const float bt, const float bn) {
                        const float f = x * expf(bt - bn);
                        return in ? f : 0.f;
                    };
                    float4 x[2] = {make_float4(up_to(q[u].x, own[u].x, sum.x), up_to(q[u].y, own[u].y, sum.y), up_to(q[u].z, own[u].z, sum.z), up_to(q[u].w, own[u].w, sum.w)),
                                   make_float4(up_to(k[u].x, sum.x, own[u].x), up_to(k[u].y, sum.y, own[u].y), up_to(k[u].z, sum.z, own[u].z), up_to(k[u].w, sum.w, own[u].w))};
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int part = 0; part < 3; ++part) {
                            uint2 r;
                            r.x = pt_take(x[e].x, x[e].y);
                            r.y = pt_take(x[e].z, x[e].w);
                            *reinterpret_cast<uint2*>(ops + ((lane >> 1) * GC_ROWS + (3 * e + part) * GC_RUN + t) * 16 + (lane & 1) * 8) = r;
                        }
                    }
                }
                if (w == 0 && !few) *reinterpret_cast<float4*>(dec + c4) = make_float4(expf(sum.x), expf(sum.y), expf(sum.z), expf(sum.w));
                pos += n;
                request(pos);
                named_bar_sync(2, GC_HALF);
                if (few) {
                    if (lane == 0) mbar_arrive(b_full + 8 * b);
                    continue;
                }
                {                                            // A: sixteen channels a warp (mma.sync on the operands' parts), the warps' sums added up
                    const int grp = lane >> 2, tig = lane & 3;
                    float a[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                    auto word = [&](const int run, const int row) { return *reinterpret_cast<const uint32_t*>(ops + (run * GC_ROWS + row) * 16 + 4 * tig); };
                    uint32_t qa[3][4], kb[3][4];             // kb: tokens 0 .. 7 and 8 .. 15, lower and upper eight channels
#pragma unroll
                    for (int part = 0; part < 3; ++part)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            qa[part][e] = word(2 * w + (e >> 1), part * GC_RUN + grp + 8 * (e & 1));
                            kb[part][e] = word(2 * w + (e & 1), (3 + part) * GC_RUN + grp + 8 * (e >> 1));
                        }
                    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // the smallest first
#pragma unroll
                    for (int e = 0; e < 6; ++e)
#pragma unroll
                        for (int y = 0; y < 2; ++y) gc_mma_bf16(a[y], qa[PA[e]], kb[PB[e]][2 * y], kb[PB[e]][2 * y + 1]);
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int e = 0; e < 2; ++e) *reinterpret_cast<float2*>(sums + (w * GC_RUN + grp + 8 * e) * 16 + 8 * y + 2 * tig) = make_float2(a[y][2 * e], a[y][2 * e + 1]);
                }
                named_bar_sync(2, GC_HALF);
                {
                    const int x = tid - GC_HALF, t = x >> 4, s_ = x & 15;
                    float a = 0.f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) a += sums[e * 256 + x];
                    A[t * 20 + s_] = s_ <= t ? a : 0.f;
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_full + 8 * b);
            }
        } else {
            // ===================== the state: thread = (row i of the key dimension, half of the columns) and later (column i, half of the tokens) =====================
            const int i = tid & 127, half = tid >> 7;
            const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            const bool one = elect_one();
            float S[64];
            const int ks = p.s.ks, rt = p.s.rt;
            float* const rec = p.state + ((size_t)slot * p.H + h) * ((size_t)ks * rt * dv) + (size_t)((i % rt) >> 2) * dv * ks * 4 + (i / rt) * 4 + (i & 3);      // entry (i, j) at 4 ks j
#pragma unroll
            for (int j = 0; j < 64; ++j) S[j] = i < dk && 64 * half + j < dv ? rec[(size_t)(64 * half + j) * ks * 4] : 0.f;
            const uint32_t I48 = umma_idesc_bf16(128, 48) | (1u << 15), I32 = umma_idesc_bf16(128, 32) | (1u << 15), I16 = umma_idesc_bf16(128, 16) | (1u << 15);
            const uint32_t I2 = umma_idesc_bf16(128, 128) | (3u << 15);
            const uint64_t ds = umma_desc(base, 128, 2048), dvp = umma_desc(base + GC_STATE + 2 * GC_BUF, 128, 256);
            uint32_t c = 0, products = 0;                    // runs, and those multiplied by the tensor core
            for (int pos = 0; pos < nt; ++c) {
                const uint32_t b = c & 1;
                const uint8_t* const ops = gbuf + b * GC_BUF;
                const float* const val = reinterpret_cast<const float*>(ops + GC_OPS);
                const float* const A = val + GC_RUN * GC_PITCH;
                mbar_wait(b_full + 8 * b, (c >> 1) & 1, 62);
                const int n = s_n[b];
                if (n < 0) {                                 // token by token: S <- alpha S + k v, read-outs summed over the rows in halves of 32 columns
                    const float* const x = reinterpret_cast<const float*>(ops) + i;
                    float* const red = reinterpret_cast<float*>(g0);      // [2 tokens][4 warps of rows][128 columns]
                    for (int t = 0; t < -n; ++t) {
                        const float q = x[t * GC_DMAX], k = x[(GC_RUN + t) * GC_DMAX], a = x[(2 * GC_RUN + t) * GC_DMAX];
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            float o[32];
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                float& e = S[32 * g + j];
                                e = fmaf(k, val[t * GC_PITCH + 64 * half + 32 * g + j], e * a);
                                o[j] = q * e;
                            }
#pragma unroll
                            for (int d = 16; d > 0; d >>= 1) {      // lanes with the bit set keep the upper half
                                const bool hi = lane & d;
#pragma unroll
                                for (int j = 0; j < d; ++j) {
                                    const float mine = hi ? o[d + j] : o[j], other = hi ? o[j] : o[d + j];
                                    o[j] = mine + __shfl_xor_sync(0xffffffffu, other, d);
                                }
                            }
                            red[((t & 1) * 4 + (warp & 3)) * 128 + 64 * half + 32 * g + lane] = o[0];
                        }
                        named_bar_sync(1, GC_HALF);
                        if (half == (t & 1) && i < dv) {
                            const float* const r = red + (t & 1) * 512 + i;
                            p.norm.x[(size_t)(t0 + pos + t) * p.norm.ldx + (size_t)h * dv + i] = ((r[0] + r[128]) + (r[256] + r[384])) * p.q_scale;
                        }
                    }
                    named_bar_sync(1, GC_HALF);              // all have read the run
                    if (tid == 0) mbar_arrive(b_free + 8 * b);
                    pos -= n;
                    continue;
                }
                const uint32_t turn = products++ & 1;
                {
                    const float f = A[GC_RUN * 20 + i];      // the run's decay
#pragma unroll
                    for (int j = 0; j < 64; ++j) S[j] *= f;
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) {                // parts of the state
                    float x[8];
                    uint4 part[3];
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = S[8 * r + e];
                    pt_split8(x, part);
#pragma unroll
                    for (int w = 0; w < 3; ++w) *reinterpret_cast<uint4*>(g0 + ((w * 16 + 8 * half + r) * 128 + i) * 16) = part[w];
                }
                {                                            // parts of the values: a token and eight columns a thread
                    const int t = i & 15, run = (i >> 4) + 8 * half;
                    float x[8];
                    uint4 part[3];
                    *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(val + t * GC_PITCH + 8 * run);
                    *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(val + t * GC_PITCH + 8 * run + 4);
                    pt_split8(x, part);
#pragma unroll
                    for (int w = 0; w < 3; ++w) *reinterpret_cast<uint4*>(gvp + ((w * 16 + run) * 16 + t) * 16) = part[w];
                }
                fence_proxy_async_smem();
                tc_fence_before();
                named_bar_sync(1, GC_HALF);
                if (warp == 0) {
                    tc_fence_after();
                    const uint64_t dq = umma_desc(base + GC_STATE + b * GC_BUF, GC_ROWS * 16, 128), dk_ = umma_desc(base + GC_STATE + b * GC_BUF + 48 * 16, 128, GC_ROWS * 16);
                    constexpr uint32_t KS = 16, KQ = 2 * GC_ROWS, PS = 16 * 128, PV = 16 * 16;      // steps of 16 channels, parts (in 16 bytes)
                    // Small products first, each half of the channels in columns of its own: four additions at full size, which the tensor core rounds towards zero, then one that
                    // rounds to nearest (in one sum with the products as they come, read-outs were 4.2e-7 from 64 bits where the token-by-token form is 2.6e-7)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint32_t d = tmem + GC_TD1 + 48 * e;
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + PS + k * KS, dq + k * KQ, k == 4 * e ? I48 : I32, k > 4 * e);      // (the first sets all columns)
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + 2 * PS + k * KS, dq + k * KQ, I16, 1);
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + k * KS, dq + k * KQ, I48, 1);
                    }
                    if (one) tc_commit(b_d1);
                    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // the smallest first
#pragma unroll
                    for (int e = 0; e < 6; ++e)
                        if (one) tc_mma_f16(tmem + GC_TD2, dk_ + PA[e] * 16, dvp + PB[e] * PV, I2, e > 0);
                    if (one) tc_commit(b_d2);
                    __syncwarp();
                }
                // products within the run while the MMAs run: column i, tokens 8 half ..
                float o[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) o[u] = 0.f;
#pragma unroll
                for (int s0 = 0; s0 < GC_RUN; s0 += 4) {
                    if (s0 > 8 * half + 7) break;
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = val[(s0 + e) * GC_PITCH + i];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const float4 a = *reinterpret_cast<const float4*>(A + (8 * half + u) * 20 + s0);
                        o[u] = fmaf(a.x, v[0], fmaf(a.y, v[1], fmaf(a.z, v[2], fmaf(a.w, v[3], o[u]))));
                    }
                }
                {
                    float sum = 0.f;
#pragma unroll
                    for (int u = 0; u < 8; ++u) sum += o[u];
                    if (!(fabsf(sum) < CUDART_INF_F))        // zero times a later token's value that is no number: those tokens left out one by one
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            o[u] = 0.f;
                            for (int s0 = 0; s0 <= 8 * half + u; ++s0) o[u] = fmaf(A[(8 * half + u) * 20 + s0], val[s0 * GC_PITCH + i], o[u]);
                        }
                }
                mbar_wait(b_d1, turn, 63);
                tc_fence_after();
                {
                    float r[8];
#pragma unroll
                    for (int e = 5; e >= 0; --e) {           // the smallest first: parts of the queries, halves of the channels
                        float x[8];
                        tc_ld8(tm + GC_TD1 + 48 * (e & 1) + 16 * (e >> 1) + 8 * half, x);
#pragma unroll
                        for (int u = 0; u < 8; ++u) r[u] = e == 5 ? x[u] : r[u] + x[u];
                    }
                    float* const out = p.norm.x + (size_t)(t0 + pos) * p.norm.ldx + (size_t)h * dv + i;
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (8 * half + u < n && i < dv) out[(size_t)(8 * half + u) * p.norm.ldx] = (r[u] + o[u]) * p.q_scale;
                    }
                }
                mbar_wait(b_d2, turn, 64);
                tc_fence_after();
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    float x[16];
                    tc_ld16(tm + GC_TD2 + 64 * half + 16 * g, x);
#pragma unroll
                    for (int j = 0; j < 16; ++j) S[16 * g + j] += x[j];
                }
                named_bar_sync(1, GC_HALF);                  // all have read the run's values
                if (tid == 0) mbar_arrive(b_free + 8 * b);
                pos += n;
            }
#pragma unroll
            for (int j = 0; j < 64; ++j)
                if (i < dk && 64 * half + j < dv) rec[(size_t)(64 * half + j) * ks * 4] = S[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, GC_TMEM_COLS);
}

}  // namespace b200
