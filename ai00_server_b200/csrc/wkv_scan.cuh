// WKV recurrences of prompt steps: the recurrence, GroupNorm, v7 bonus and gate of wkv.cuh (same operands, same state layout
// M[value][key], reference run.rs:1143) for steps in which a sequence holds more than WKV_STAGE_TOK tokens.
//
// What bounds it: the chain of tokens of one (head, sequence), 64-odd CTAs for one prompt.  The decode kernel spends four barriers, a
// round trip to memory and the norm of one warp on every token (2.6 us a token at 7B widths, the decay LoRA evaluated in place); here
// the loop over tokens has NO barrier and no memory latency:
//   * the vectors of the next TC tokens are requested while TC tokens run.  RWKV-5 / 6 copy them to their places as they are (cp.async, no registers: 94 instead of 162, so that
//     five CTAs of an SM run instead of three); RWKV-7 works out what does not depend on the state (unit key, removal / write vectors, value residual, bonus) per group, a warp per token;
//   * a thread holds 4 values x 8 neighbouring keys of the state; key-indexed vectors lie in shared memory with each run of eight split into
//     two half rows, so that the eight lanes of a value row read 128 contiguous bytes and the other three rows of the warp share them;
//   * products run as packed pairs of neighbouring keys (half the instructions of a loop that is bound by them); RWKV-5 / 6: the bonus of the current
//     token, (sum_c r u k) v, is one number a token, worked out with the group and added behind the sums;
//   * the loop over tokens leaves the four read-outs of a thread as they are; the eight lanes' parts are summed with the norms and outputs, per group, a
//     warp per token (exchanges between lanes in the loop were a chain of four, some 25 cycles each, on every token).  Sums over keys run even and odd
//     keys apart: results agree with wkv.cuh's to f32 rounding.
// Decays come from the decay projection's own launch in these steps (lora2.cuh: 6 us beside the scan's own time below).  Where the decode kernel
// evaluates that low-rank stage itself (RWKV-6), its sums run in another order: decays, and with them states, agree to f32 rounding and not to the bit.
// Measured, RWKV-6 (vectors through registers and three CTAs an SM before, copied and five now): 64 tokens of 32 sequences, 40 heads, 93 -> 78 us, 128 of sixteen, 64 heads, 141 -> 119, 61 of six
// 25 -> 25, one prompt of 100, 64 heads, 29 -> 27 (263 in the decode kernel).  At five CTAs the path to shared memory is busy 73 % of the time, issue slots 53 %, multiply-adds 46 %;
// eight values a thread halve its reads but leave two warps a head (97 us at the first of these).
#pragma once
#include "f32x2.cuh"
#include "wkv.cuh"

namespace b200 {

constexpr int WKS_THREADS = 128;
// TC_: tokens per group.  RWKV-5 / 6: eight, of which an SM holds five CTAs, or sixteen, three CTAs, where three an SM are all there are (one prompt of 100 tokens, 64 heads, 29 and 27 us;
// 64 tokens of 32 sequences, 40 heads, 78 and 87)
template <int VER, int TC_> struct WksCfg {
    static constexpr int TC = TC_;
    static constexpr int CTAS = VER == 7 || TC_ == 16 ? 3 : 5;      // of an SM
    static constexpr int UNROLL = CTAS == 3 ? 2 : 1;        // (five CTAs: two tokens at a time are 80 us instead of 78 in the step above)
    static constexpr int NA = VER == 7 ? 6 : 4;             // staged vectors: r, k, v, w (, -kk, kk a)
    static constexpr int BUF = NA * TC * WKV_N;             // floats of one group
    static constexpr int OUT_ROW = WKV_N + 4, OUT = 8 * OUT_ROW;      // a token's read-outs: eight partial sums of every value (padded: conflict-free)
    static constexpr int SMEM_BYTES = (2 * BUF + 2 * TC + TC * OUT) * 4;
};
// place of key c in a staged vector: keys 8 j .. 8 j + 3 at 4 j, 8 j + 4 .. 8 j + 7 at 32 + 4 j
__device__ __forceinline__ int wks_place(int c) { return (c >> 3) * 4 + (c & 3) + ((c >> 2) & 1) * 32; }

template <int VER, int TC_>
__global__ void __launch_bounds__(WKS_THREADS, WksCfg<VER, TC_>::CTAS) wkv_scan_kernel(const __grid_constant__ WkvParams p) {
    using Cfg = WksCfg<VER, TC_>;
    constexpr int TC = Cfg::TC, TW = TC / 4;                // tokens per warp in the per-group phases
    extern __shared__ __align__(16) float wks[];
    float* const sc = wks + 2 * Cfg::BUF;                   // [2][TC] bonus of the token
    float* const so = sc + 2 * TC;                          // [TC][8][64] partial read-outs
    pdl_launch_dependents();
    const int h = blockIdx.x, si = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ig = tid >> 3, j = tid & 7, ch = h * WKV_N;
    if (si >= p.meta.nslots()) return;
    const int slot = p.meta.slot_id()[si], t0 = p.meta.slot_start()[si], nt = p.meta.slot_count()[si];
    float* const M = p.state + ((size_t)slot * p.H + h) * (WKV_N * WKV_N);
    f32x2 m[4][4];                                          // pairs of keys
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float4 v4 = __ldcs(reinterpret_cast<const float4*>(M + (ig * 4 + e) * WKV_N + 8 * j + 4 * q));
            m[e][2 * q] = pack2(v4.x, v4.y); m[e][2 * q + 1] = pack2(v4.z, v4.w);
        }
    const int c2 = ch + lane;                               // the per-group phases give a lane the channels lane and lane + 32
    auto ld2 = [](const float* q) { return make_float2(q[0], q[32]); };
    const float2 lw = ld2(p.lnx_w + c2), lb = ld2(p.lnx_b + c2);
    float2 kk_ = make_float2(0.f, 0.f), ka_ = kk_, rk_ = kk_, u2 = kk_;
    if (VER == 7) { kk_ = ld2(p.k_k + c2); ka_ = ld2(p.k_a + c2); rk_ = ld2(p.r_k + c2); }
    if (VER != 7) u2 = make_float2(p.u[ch + (lane >> 2) * 8 + (lane & 3)], p.u[ch + (lane >> 2) * 8 + 4 + (lane & 3)]);      // the keys at places lane and lane + 32
    pdl_wait();

    // RWKV-5 / 6: the vectors go to their places as they are, sixteen bytes a copy
    auto copy = [&](const int g0, const int b) {
        constexpr int ARR = VER == 6 ? 4 : 3;
#pragma unroll
        for (int x = tid; x < ARR * TC * 16; x += WKS_THREADS) {
            const int arr = x / (TC * 16), tt = x / 16 % TC, c = x & 15;
            const float* const src = arr == 0 ? p.r : (arr == 1 ? p.k : (arr == 2 ? p.v : p.w));
            float* const d = wks + b * Cfg::BUF + (arr * TC + tt) * WKV_N + (arr == 2 ? 4 * c : (c >> 1) * 4 + (c & 1) * 32);
            if (g0 + tt < nt) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_u32(d)), "l"(src + (size_t)(t0 + g0 + tt) * p.ld + ch + 4 * c) : "memory");
        }
    };
    auto landed = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
    struct Row { float2 r, k, v, w, a, nu, vf; };
    Row row[VER == 7 ? TW : 1];
    auto request = [&](const int g0) {                      // the group's vectors -> registers
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int t = g0 + warp + 4 * i;
            if (t >= nt) continue;
            const size_t at = (size_t)(t0 + t) * p.ld + c2;
            row[i].r = ld2(p.r + at); row[i].k = ld2(p.k + at); row[i].v = ld2(p.v + at);
            row[i].w = ld2(p.w + at);
            row[i].a = ld2(p.a + at);
            if (!p.layer0) { row[i].nu = ld2(p.nu + at); row[i].vf = ld2(p.v_first + at); }
        }
    };
    auto prepare = [&](const int g0, const int b) {         // registers -> shared memory, with all that the state does not enter
        float* const buf = wks + b * Cfg::BUF;
        auto st2 = [&](const int arr, const int tt, const float2 x) {      // by key
            float* const d = buf + (arr * TC + tt) * WKV_N;
            d[wks_place(lane)] = x.x;
            d[wks_place(lane + 32)] = x.y;
        };
        auto sum2 = [&](const float2 x) { return warp_sum(x.x) + warp_sum(x.y); };
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int tt = warp + 4 * i, t = g0 + tt;
            if (t >= nt) continue;                          // warp-uniform
            const float2 r = row[i].r;
            float2 k = row[i].k, v = row[i].v;
            const float2 a = row[i].a;
            float2 kk = make_float2(k.x * kk_.x, k.y * kk_.y);
            const float norm = fmaxf(sqrtf(sum2(make_float2(kk.x * kk.x, kk.y * kk.y))), 1e-12f);
            kk.x /= norm; kk.y /= norm;
            k.x *= 1.f + (a.x - 1.f) * ka_.x; k.y *= 1.f + (a.y - 1.f) * ka_.y;
            if (p.layer0) {
                float* const d = p.v_first + (size_t)(t0 + t) * p.ld + c2;
                d[0] = v.x; d[32] = v.y;
            } else { v.x += (row[i].vf.x - v.x) * row[i].nu.x; v.y += (row[i].vf.y - v.y) * row[i].nu.y; }
            const float bonus = sum2(make_float2(r.x * k.x * rk_.x, r.y * k.y * rk_.y));
            if (lane == 0) sc[b * TC + tt] = bonus;
            st2(4, tt, make_float2(-kk.x, -kk.y));
            st2(5, tt, make_float2(kk.x * a.x, kk.y * a.y));
            st2(0, tt, r); st2(1, tt, k);
            buf[(2 * TC + tt) * WKV_N + lane] = v.x;        // by value
            buf[(2 * TC + tt) * WKV_N + lane + 32] = v.y;
            st2(3, tt, row[i].w);
        }
    };
    if (VER == 7) { request(0); prepare(0, 0); }
    else {
        copy(0, 0);
        if (VER == 5)
            for (int x = tid; x < 2 * TC * WKV_N; x += WKS_THREADS) wks[(x / (TC * WKV_N)) * Cfg::BUF + (3 * TC + x / WKV_N % TC) * WKV_N + wks_place(x % WKV_N)] = p.w_static[ch + x % WKV_N];
        landed();
    }
    __syncthreads();
    for (int g0 = 0, b = 0; g0 < nt; g0 += TC, b ^= 1) {
        const int n = min(TC, nt - g0);
        if (VER == 7) request(g0 + TC);
        else copy(g0 + TC, b ^ 1);
        float2 gate[TW];
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int t = g0 + warp + 4 * i;
            gate[i] = t < nt ? ld2(p.g + (size_t)(t0 + t) * p.ld + c2) : make_float2(0.f, 0.f);
        }
        const float* const buf = wks + b * Cfg::BUF;
#pragma unroll (Cfg::UNROLL)
        for (int tt = 0; tt < n; ++tt) {
            auto ld8 = [&](const int arr, f32x2 (&x)[4]) {
                const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(buf + (arr * TC + tt) * WKV_N + 4 * j);
                const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(buf + (arr * TC + tt) * WKV_N + 32 + 4 * j);
                x[0] = lo.x; x[1] = lo.y; x[2] = hi.x; x[3] = hi.y;
            };
            f32x2 r[4], k[4], w[4];
            float o[4];
            ld8(0, r); ld8(1, k); ld8(3, w);
            const float4 v4 = *reinterpret_cast<const float4*>(buf + (2 * TC + tt) * WKV_N + 4 * ig);
            const f32x2 v[4] = {pack2(v4.x, v4.x), pack2(v4.y, v4.y), pack2(v4.z, v4.z), pack2(v4.w, v4.w)};
            if (VER != 7) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    f32x2 acc = 0ull;
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        fma2(acc, r[f], m[e][f]);
                        m[e][f] = fmadd2(w[f], m[e][f], prod2(k[f], v[e]));
                    }
                    const float2 a2 = unpack2(acc);
                    o[e] = a2.x + a2.y;
                }
            } else {
                f32x2 nk[4], ka[4];
                float sa[4];
                ld8(4, nk); ld8(5, ka);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    f32x2 s = prod2(m[e][0], nk[0]);
#pragma unroll
                    for (int f = 1; f < 4; ++f) fma2(s, m[e][f], nk[f]);
                    const float2 a2 = unpack2(s);
                    sa[e] = a2.x + a2.y;
                }
#pragma unroll
                for (int off = 4; off > 0; off >>= 1)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sa[e] += __shfl_xor_sync(0xffffffffu, sa[e], off);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const f32x2 s2 = pack2(sa[e], sa[e]);
                    f32x2 acc = 0ull;
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        m[e][f] = fmadd2(v[e], k[f], fmadd2(m[e][f], w[f], prod2(s2, ka[f])));      // the state, the largest term, is not rounded apart
                        fma2(acc, m[e][f], r[f]);
                    }
                    const float2 a2 = unpack2(acc);
                    o[e] = a2.x + a2.y;
                }
            }
            *reinterpret_cast<float4*>(so + tt * Cfg::OUT + j * Cfg::OUT_ROW + ig * 4) = make_float4(o[0], o[1], o[2], o[3]);
        }
        if (VER == 7) prepare(g0 + TC, b ^ 1);
        else landed();
        __syncthreads();
        // GroupNorm over the head (+ bonus) * gate -> operand of the output projection, a warp per token
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int tt = warp + 4 * i;
            if (tt >= n) continue;
            float2 x = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float2 y = ld2(so + tt * Cfg::OUT + q * Cfg::OUT_ROW + lane);
                x.x += y.x; x.y += y.y;
            }
            float s;
            if (VER == 7) s = sc[b * TC + tt];
            else {
                const float2 r = ld2(buf + tt * WKV_N + lane), k = ld2(buf + (TC + tt) * WKV_N + lane);      // by place
                s = warp_sum(r.x * (u2.x * k.x)) + warp_sum(r.y * (u2.y * k.y));
            }
            const float2 v = ld2(buf + (2 * TC + tt) * WKV_N + lane);
            if (VER != 7) { x.x = fmaf(s, v.x, x.x); x.y = fmaf(s, v.y, x.y); }
            const float mean = warp_sum(x.x + x.y) * (1.f / WKV_N);
            const float d0 = x.x - mean, d1 = x.y - mean;
            const float rstd = 1.0f / sqrtf(warp_sum(d0 * d0 + d1 * d1) * (1.f / WKV_N) + GN_EPS);
            float y0 = d0 * rstd * lw.x + lb.x, y1 = d1 * rstd * lw.y + lb.y;
            if (VER == 7) {
                y0 += s * v.x; y1 += s * v.y;
            }
            y0 *= gate[i].x; y1 *= gate[i].y;
            p.out[a16_index(t0 + g0 + tt, c2, p.kq_tile)] = f2h_sat(y0);
            p.out[a16_index(t0 + g0 + tt, c2 + 32, p.kq_tile)] = f2h_sat(y1);
        }
        __syncthreads();                                    // the group's buffers are refilled next
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            const float2 lo = unpack2(m[e][2 * q]), hi = unpack2(m[e][2 * q + 1]);
            __stcs(reinterpret_cast<float4*>(M + (ig * 4 + e) * WKV_N + 8 * j + 4 * q), make_float4(lo.x, lo.y, hi.x, hi.y));
        }
}

}  // namespace b200
