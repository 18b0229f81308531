// Recurrences with one decay a head, sixteen tokens of a prompt step at a time (the construction of gla_chunk.cuh):
//   DELTA   the gated delta rule of delta_rule.cuh with a decay per head:   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q      (k, q of unit length)
//   else    the matrix memory of matrix_memory.cuh:                         S <- e^(f + m - m') S + e^(i - m') k v^T;  o = S^T q, and the normaliser's factor
// Over a run of n <= 16 tokens, b_t the sum of the logarithms of the decays up to t (never positive):
//     u_t = beta_t (v_t - e^{b_t} S_0^T k_t - sum_{s < t} e^{b_t - b_s} (k_s . k_t) u_s)      or  e^(i - m') v_t
//     o_t = e^{b_t} S_0^T q_t + sum_{s <= t} e^{b_t - b_s} (k_s . q_t) u_s,      S_n = e^{b_n} S_0 + sum_s e^{b_n - b_s} k_s u_s^T
// Decays are factors of sums here and never of operands, so that no run has to end early.  A logarithm below DC_LEAST, -inf among them, counts as DC_LEAST: its factor is zero in f32
// either way (e^-104 is), and sums with the parts they lost need finite terms.
//
// What bounds the token-by-token forms: a chain of two reductions and exchanges a token (1.6 us a token of a sequence on an SM).  Here eight warps keep the state in registers, as in
// gla_chunk.cuh; the triangular system for u is solved by the thread of a column in registers, a row of it a step; eight warps prepare the next run: unit lengths and gates within a
// warp, the 16 x 16 products by mma.sync on the operands' parts.  Every f32 number is three bf16 parts in an operand, sums are f32.  The matrix memory writes its state by f32
// multiply-adds: the tensor core cuts its sums, which a state of so few roundings shows (7.9e-8 from 64 bits token by token and so, 8.9e-8 with it; 66 and 52 us).
// Measured, heads of 128 x 128: delta rule, sixteen heads, 128 tokens of sixteen sequences 208 -> 103 us, 1000 of one 580 -> 323; matrix memory, eight heads, 128 of sixteen 124 -> 66,
// sixteen heads, 1000 of one 577 -> 428.  Distance from 64 bits (2-norm): delta rule, read-outs 1.69e-7 -> 1.42e-7, states 1.49e-7 -> 1.36e-7; matrix memory, read-outs 1.13e-7 ->
// 1.14e-7, the factor they are taken with 4.2e-7 -> 3.1e-7, states 7.9e-8 -> 7.8e-8.
#pragma once
#include "delta_rule.cuh"
#include "gla_chunk.cuh"
#include "matrix_memory.cuh"

namespace b200 {

struct RunChunkParams {
    const float* q; const float* k; const float* v; int ld;      // q, k of key head h / rep
    int rep;
    const float* z; int ldz;                      // decay pre-activation / forget gate [T, H]
    const float* b; int ldb;                      // write-strength logits / input gate [T, H]
    const float* a_log;                           // DELTA: [H]
    float* state;
    float* n; float* m; float* fac;               // matrix memory: [S][H][dk], [S][H][dv], [T][H]
    int H, dk, dv;
    float q_scale, eps, cap;                      // eps: of the unit length / of the denominator
    ScanShape s;
    HeadNormParams norm;
};

constexpr int DC_KEYS = GC_RUN * GC_DMAX * 4, DC_BUF = GC_OPS + GC_VAL + 2 * GC_A + 512 + DC_KEYS;
constexpr size_t DC_SMEM = GC_STATE + 2 * DC_BUF + GC_VPARTS + 2 * 8 * GC_RUN * GC_RUN * 4 + 128;
constexpr float DC_LEAST = -1e4f;
constexpr uint32_t DC_TD1 = 0, DC_TD2 = 192, DC_TMEM_COLS = 512;      // tensor memory: read-outs [2 halves of the channels][3 parts][16 queries, 16 keys], the run's addition to the state

template <bool DELTA>
__global__ void __launch_bounds__(GC_THREADS, 1) run_chunk_kernel(const __grid_constant__ RunChunkParams p) {
    extern __shared__ __align__(16) uint8_t gc_smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[6];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = smem_u32(s_bar), b_full = bar, b_free = bar + 16, b_d1 = bar + 32, b_d2 = bar + 40;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { mbar_init(b_full + 8 * i, GC_HALF / 32); mbar_init(b_free + 8 * i, 1); }
        mbar_init(b_d1, 1); mbar_init(b_d2, 1);
        mbar_fence_init();
    }
    if (warp == 0) tc_alloc(smem_u32(&s_tmem), DC_TMEM_COLS);
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
        const size_t hs = (size_t)slot * p.H + h;
        const uint32_t raw = smem_u32(gc_smem_raw), base = (raw + 127u) & ~127u;
        uint8_t* const g0 = gc_smem_raw + (base - raw);
        uint8_t* const gbuf = g0 + GC_STATE;
        uint8_t* const gvp = gbuf + 2 * DC_BUF;
        float* const writes = reinterpret_cast<float*>(gvp);                 // matrix memory: what the run's keys write [16][128]
        float* const sums = reinterpret_cast<float*>(gvp + GC_VPARTS);       // the warps' parts of q . k and k . k
        if (warp >= 8) {
            // ===================== the next run's operands: a warp takes two tokens, a lane four channels =====================
            const int w = warp - 8, c4 = 4 * lane, hk = h / p.rep;
            auto whole = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
            const float* const kp = p.k + (size_t)t0 * p.ld + (size_t)hk * dk + c4;
            const float* const qp = p.q + (size_t)t0 * p.ld + (size_t)hk * dk + c4;
            const float* const vp = p.v + (size_t)t0 * p.ld + (size_t)h * dv + c4;
            const bool vec = (dk | dv | p.ld) % 4 == 0 && whole(p.k) && whole(p.q) && whole(p.v);
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
            float4 q[2], k[2], v[2];
            float z = 0.f, g = 0.f;
            auto request = [&](const int pos) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = pos + 2 * w + u, lk = t < nt ? dk - c4 : 0, lv = t < nt ? dv - c4 : 0;
                    q[u] = load4(qp + (size_t)t * p.ld, lk);
                    k[u] = load4(kp + (size_t)t * p.ld, lk);
                    v[u] = load4(vp + (size_t)t * p.ld, lv);
                }
                const int t = pos + (lane & 15);             // gates of the run, in every warp
                z = t < nt ? p.z[(size_t)(t0 + t) * p.ldz + h] : 0.f;
                g = t < nt ? p.b[(size_t)(t0 + t) * p.ldb + h] : 0.f;
            };
            request(0);
            const float rate = DELTA ? expf(p.a_log[h]) : 0.f;
            float m_run = DELTA ? 0.f : p.m[hs * dv];
            float4 nrm = make_float4(0.f, 0.f, 0.f, 0.f);    // the normaliser, in every warp
            if (!DELTA) {
                const float* const np = p.n + hs * dk + c4;
                if (c4 < dk) nrm.x = np[0];
                if (c4 + 1 < dk) nrm.y = np[1];
                if (c4 + 2 < dk) nrm.z = np[2];
                if (c4 + 3 < dk) nrm.w = np[3];
            }
            int c = 0;
            for (int pos = 0; pos < nt; pos += GC_RUN, ++c) {
                const int b = c & 1, n = min(nt - pos, GC_RUN);
                uint8_t* const ops = gbuf + b * DC_BUF;
                float* const val = reinterpret_cast<float*>(ops + GC_OPS);
                float* const A = val + GC_RUN * GC_PITCH;
                float* const L = A + GC_RUN * 20;
                float* const sc = L + GC_RUN * 20;           // [16] (e^{b_t}, beta_t e^{b_t}, e^{b_n - b_t}, -), then e^{b_n}
                float* const keys = sc + 128;                // matrix memory: [16][128]
                // lane t: gates of token t, sums of the logarithms
                const int tt = lane & 15;
                const bool in = tt < n;
                float bt, write = 0.f, least = 0.f;          // b_t, what a value is written with, e^-m
                if (DELTA) {
                    bt = in ? -rate * (fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)))) : 0.f;
                    if (bt < DC_LEAST) bt = DC_LEAST;        // (not fmaxf: what is no number stays so)
                    write = in ? 1.f / (1.f + expf(-g)) : 0.f;
                } else {
                    const float ig = p.cap * tanhf(g / p.cap), zc = p.cap * tanhf(z / p.cap);
                    const float fg = fminf(zc, 0.f) - log1pf(expf(-fabsf(zc)));
                    float m_prev = 0.f, m_new = 0.f;
#pragma unroll
                    for (int u = 0; u < GC_RUN; ++u) {
                        const float f = __shfl_sync(0xffffffffu, fg, u), i = __shfl_sync(0xffffffffu, ig, u), next = u < n ? fmaxf(f + m_run, i) : m_run;
                        if (tt == u) { m_prev = m_run; m_new = next; }
                        m_run = next;
                    }
                    bt = in ? fg + m_prev - m_new : 0.f;
                    write = in ? expf(ig - m_new) : 0.f;
                    least = expf(-m_new);
                }
                // sums with what their roundings lost: differences of large sums are factors of neighbouring tokens
                float lost = 0.f;
                {
                    const float mine = bt;
                    bt = 0.f;
#pragma unroll
                    for (int u = 0; u < GC_RUN; ++u) {
                        const float x = __shfl_sync(0xffffffffu, mine, u), next = bt + x, grown = next - bt, gone = (bt - (next - grown)) + (x - grown);
                        if (u <= tt) { bt = next; lost += gone; }
                    }
                }
                const float end = __shfl_sync(0xffffffffu, bt, 15), end_lost = __shfl_sync(0xffffffffu, lost, 15);
                const float after = expf(bt == end ? end_lost - lost : (end - bt) + (end_lost - lost));      // e^{b_n - b_t}
                if (c > 1) mbar_wait(b_free + 8 * b, ((c >> 1) - 1) & 1, 71);
                const float e_t = expf(bt), before = fmaf(e_t, lost, e_t), e_n = expf(end), whole_run = fmaf(e_n, end_lost, e_n);      // e^{b_t}, e^{b_n}
                if (w == 0 && lane < GC_RUN) reinterpret_cast<float4*>(sc)[lane] = make_float4(before, write * before, after, 0.f);
                if (w == 0 && lane == 0) sc[4 * GC_RUN] = whole_run;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = 2 * w + u;
                    if (DELTA) {                             // unit lengths
                        const float kk = warp_sum(fmaf(k[u].x, k[u].x, fmaf(k[u].y, k[u].y, fmaf(k[u].z, k[u].z, k[u].w * k[u].w))));
                        const float qq = warp_sum(fmaf(q[u].x, q[u].x, fmaf(q[u].y, q[u].y, fmaf(q[u].z, q[u].z, q[u].w * q[u].w))));
                        const float fk = 1.f / sqrtf(kk + p.eps), fq = p.q_scale / sqrtf(qq + p.eps);
                        k[u].x *= fk; k[u].y *= fk; k[u].z *= fk; k[u].w *= fk;
                        q[u].x *= fq; q[u].y *= fq; q[u].z *= fq; q[u].w *= fq;
                    }
                    const float wv = __shfl_sync(0xffffffffu, write, t);
                    *reinterpret_cast<float4*>(val + t * GC_PITCH + c4) = t < n ? make_float4(v[u].x * wv, v[u].y * wv, v[u].z * wv, v[u].w * wv) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (!DELTA) *reinterpret_cast<float4*>(keys + t * GC_DMAX + c4) = k[u];
                    float4 x[2] = {q[u], k[u]};
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int part = 0; part < 3; ++part) {
                            uint2 r;
                            r.x = pt_take(x[e].x, x[e].y);
                            r.y = pt_take(x[e].z, x[e].w);
                            *reinterpret_cast<uint2*>(ops + ((lane >> 1) * GC_ROWS + (2 * part + e) * GC_RUN + t) * 16 + (lane & 1) * 8) = r;
                        }
                }
                // the normaliser's products with this warp's queries, of the state before the run
                float nq[2] = {0.f, 0.f};
                if (!DELTA)
#pragma unroll
                    for (int u = 0; u < 2; ++u) nq[u] = warp_sum(fmaf(nrm.x, q[u].x, fmaf(nrm.y, q[u].y, fmaf(nrm.z, q[u].z, nrm.w * q[u].w))));
                request(pos + GC_RUN);
                named_bar_sync(2, GC_HALF);
                {                                            // q . k and k . k: sixteen channels a warp (mma.sync on the operands' parts)
                    const int grp = lane >> 2, tig = lane & 3;
                    auto word = [&](const int run, const int row) { return *reinterpret_cast<const uint32_t*>(ops + (run * GC_ROWS + row) * 16 + 4 * tig); };
                    uint32_t kb[3][4];                       // tokens 0 .. 7 and 8 .. 15, lower and upper eight channels
#pragma unroll
                    for (int part = 0; part < 3; ++part)
#pragma unroll
                        for (int e = 0; e < 4; ++e) kb[part][e] = word(2 * w + (e & 1), (2 * part + 1) * GC_RUN + grp + 8 * (e >> 1));
#pragma unroll
                    for (int which = 0; which < (DELTA ? 2 : 1); ++which) {
                        float a[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                        uint32_t qa[3][4];
#pragma unroll
                        for (int part = 0; part < 3; ++part)
#pragma unroll
                            for (int e = 0; e < 4; ++e) qa[part][e] = word(2 * w + (e >> 1), (2 * part + which) * GC_RUN + grp + 8 * (e & 1));
                        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // the smallest first
#pragma unroll
                        for (int e = 0; e < 6; ++e)
#pragma unroll
                            for (int y = 0; y < 2; ++y) gc_mma_bf16(a[y], qa[PA[e]], kb[PB[e]][2 * y], kb[PB[e]][2 * y + 1]);
#pragma unroll
                        for (int y = 0; y < 2; ++y)
#pragma unroll
                            for (int e = 0; e < 2; ++e)
                                *reinterpret_cast<float2*>(sums + ((which * 8 + w) * GC_RUN + grp + 8 * e) * 16 + 8 * y + 2 * tig) = make_float2(a[y][2 * e], a[y][2 * e + 1]);
                    }
                }
                if (!DELTA) {                                // the normaliser behind the run
                    nrm.x *= whole_run; nrm.y *= whole_run; nrm.z *= whole_run; nrm.w *= whole_run;
                    const float mine = write * after;
#pragma unroll
                    for (int t = 0; t < GC_RUN; ++t) {
                        const float a = __shfl_sync(0xffffffffu, mine, t);
                        const float4 x = *reinterpret_cast<const float4*>(keys + t * GC_DMAX + c4);
                        nrm.x = fmaf(a, x.x, nrm.x); nrm.y = fmaf(a, x.y, nrm.y); nrm.z = fmaf(a, x.z, nrm.z); nrm.w = fmaf(a, x.w, nrm.w);
                    }
                }
                named_bar_sync(2, GC_HALF);
                {                                            // thread = (t, s); lanes 0 .. 15 hold row 2 w, 16 .. 31 row 2 w + 1
                    const int x = tid - GC_HALF, t = x >> 4, s_ = x & 15;
                    const float b_t = __shfl_sync(0xffffffffu, bt, t), l_t = __shfl_sync(0xffffffffu, lost, t), w_t = __shfl_sync(0xffffffffu, write, t);
                    const float f = s_ < t ? expf((b_t - bt) + (l_t - lost)) : (s_ == t ? 1.f : 0.f);      // (lane & 15 is s)
                    float a = 0.f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) a += sums[e * 256 + x];
                    a = s_ <= t ? a * f : 0.f;
                    A[t * 20 + s_] = a;
                    if (DELTA) {
                        float l = 0.f;
#pragma unroll
                        for (int e = 0; e < 8; ++e) l += sums[(8 + e) * 256 + x];
                        L[s_ * 20 + t] = s_ < t ? l * f * w_t : 0.f;      // column after column
                    } else {
                        float row = s_ <= t ? a * write : 0.f;      // n . q: the tokens of the run
#pragma unroll
                        for (int o = 1; o < 16; o <<= 1) row += __shfl_xor_sync(0xffffffffu, row, o);
                        const float before_t = __shfl_sync(0xffffffffu, before, t), e_m = __shfl_sync(0xffffffffu, least, t);
                        const float all = row + (t & 1 ? nq[1] : nq[0]) * before_t;
                        if (s_ == 0 && t < n) p.fac[(size_t)(t0 + pos + t) * p.H + h] = p.q_scale / (fmaxf(fabsf(all * p.q_scale), e_m) + p.eps);
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_full + 8 * b);
            }
            if (!DELTA && w == 0) {
                float* const np = p.n + hs * dk + c4;
                if (c4 < dk) np[0] = nrm.x;
                if (c4 + 1 < dk) np[1] = nrm.y;
                if (c4 + 2 < dk) np[2] = nrm.z;
                if (c4 + 3 < dk) np[3] = nrm.w;
                for (int i = lane; i < dv; i += 32) p.m[hs * dv + i] = m_run;
            }
        } else {
            // ===================== the state: thread = (row i of the key dimension, half of the columns) and later (column i, half of the tokens) =====================
            const int i = tid & 127, half = tid >> 7;
            const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            const bool one = elect_one();
            float S[64];
            const int ks = p.s.ks, rt = p.s.rt;
            float* const rec = p.state + hs * ((size_t)ks * rt * dv) + (size_t)((i % rt) >> 2) * dv * ks * 4 + (i / rt) * 4 + (i & 3);      // entry (i, j) at 4 ks j
#pragma unroll
            for (int j = 0; j < 64; ++j) S[j] = i < dk && 64 * half + j < dv ? rec[(size_t)(64 * half + j) * ks * 4] : 0.f;
            const uint32_t I96 = umma_idesc_bf16(128, 96) | (1u << 15), I64 = umma_idesc_bf16(128, 64) | (1u << 15), I32 = umma_idesc_bf16(128, 32) | (1u << 15);
            const uint32_t I2 = umma_idesc_bf16(128, 128) | (3u << 15);
            const uint64_t ds = umma_desc(base, 128, 2048), dvp = umma_desc(base + GC_STATE + 2 * DC_BUF, 128, 256);
            uint32_t c = 0;
            for (int pos = 0; pos < nt; pos += GC_RUN, ++c) {
                const uint32_t b = c & 1;
                const int n = min(nt - pos, GC_RUN);
                const uint8_t* const ops = gbuf + b * DC_BUF;
                const float* const val = reinterpret_cast<const float*>(ops + GC_OPS);
                const float* const A = val + GC_RUN * GC_PITCH;
                const float* const L = A + GC_RUN * 20;
                const float4* const sc = reinterpret_cast<const float4*>(L + GC_RUN * 20);
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
                fence_proxy_async_smem();
                tc_fence_before();
                mbar_wait(b_full + 8 * b, (c >> 1) & 1, 72);
                named_bar_sync(1, GC_HALF);
                if (warp == 0) {
                    tc_fence_after();
                    const uint64_t dq = umma_desc(base + GC_STATE + b * DC_BUF, GC_ROWS * 16, 128);
                    constexpr uint32_t KS = 16, KQ = 2 * GC_ROWS, PS = 16 * 128;      // steps of 16 channels, parts (in 16 bytes)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {            // small products first, each half of the channels in columns of its own: see gla_chunk.cuh
                        const uint32_t d = tmem + DC_TD1 + 96 * e;
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + PS + k * KS, dq + k * KQ, k == 4 * e ? I96 : I64, k > 4 * e);      // (the first sets all columns)
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + 2 * PS + k * KS, dq + k * KQ, I32, 1);
#pragma unroll
                        for (int k = 4 * e; k < 4 * e + 4; ++k)
                            if (one) tc_mma_f16(d, ds + k * KS, dq + k * KQ, I96, 1);
                    }
                    if (one) tc_commit(b_d1);
                    __syncwarp();
                }
                float u[GC_RUN];                             // column i
                if (DELTA)
#pragma unroll
                    for (int t = 0; t < GC_RUN; ++t) u[t] = val[t * GC_PITCH + i];
                auto written = [&](const int t) { return DELTA ? u[t] : val[t * GC_PITCH + i]; };
                mbar_wait(b_d1, c & 1, 73);
                tc_fence_after();
                if (DELTA) {
                    float x[GC_RUN];
#pragma unroll
                    for (int e = 5; e >= 0; --e) {           // the smallest first: parts, halves of the channels
                        float y[16];
                        tc_ld16(tm + DC_TD1 + 96 * (e & 1) + 32 * (e >> 1) + 16, y);
#pragma unroll
                        for (int t = 0; t < GC_RUN; ++t) x[t] = e == 5 ? y[t] : x[t] + y[t];
                    }
#pragma unroll
                    for (int t = 0; t < GC_RUN; ++t) u[t] = fmaf(-sc[t].y, x[t], u[t]);
#pragma unroll
                    for (int s0 = 0; s0 < GC_RUN - 1; ++s0)  // u of token s0 is known: the tokens behind it
#pragma unroll
                        for (int t4 = s0 / 4 * 4; t4 < GC_RUN; t4 += 4) {
                            const float4 l = *reinterpret_cast<const float4*>(L + s0 * 20 + t4);
                            if (t4 > s0) u[t4] = fmaf(-l.x, u[s0], u[t4]);
                            if (t4 + 1 > s0) u[t4 + 1] = fmaf(-l.y, u[s0], u[t4 + 1]);
                            if (t4 + 2 > s0) u[t4 + 2] = fmaf(-l.z, u[s0], u[t4 + 2]);
                            if (t4 + 3 > s0) u[t4 + 3] = fmaf(-l.w, u[s0], u[t4 + 3]);
                        }
                }
                if (DELTA) {                                 // the run's writes, with the decays behind them: parts [3][16 runs of columns][16 tokens][16 bytes]
#pragma unroll
                    for (int t = 0; t < 8; t += 2) {
                        const int at = 8 * half + t;
                        float x = (half ? u[8 + t] : u[t]) * sc[at].z, y = (half ? u[9 + t] : u[t + 1]) * sc[at + 1].z;
#pragma unroll
                        for (int w = 0; w < 3; ++w) {
                            const uint32_t r = pt_take(x, y);
                            uint16_t* const o = reinterpret_cast<uint16_t*>(gvp + ((w * 16 + (i >> 3)) * 16 + at) * 16) + (i & 7);
                            o[0] = (uint16_t)r;
                            o[8] = (uint16_t)(r >> 16);
                        }
                    }
                    fence_proxy_async_smem();
                    tc_fence_before();
                } else {
#pragma unroll
                    for (int t = 0; t < 8; ++t) writes[(8 * half + t) * GC_DMAX + i] = val[(8 * half + t) * GC_PITCH + i] * sc[8 * half + t].z;
                }
                named_bar_sync(1, GC_HALF);
                if (DELTA && warp == 0) {
                    tc_fence_after();
                    const uint64_t dk_ = umma_desc(base + GC_STATE + b * DC_BUF + GC_RUN * 16, 128, GC_ROWS * 16);
                    constexpr uint32_t PV = 16 * 16;
                    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // the smallest first
#pragma unroll
                    for (int e = 0; e < 6; ++e)
                        if (one) tc_mma_f16(tmem + DC_TD2, dk_ + PA[e] * 32, dvp + PB[e] * PV, I2, e > 0);
                    if (one) tc_commit(b_d2);
                    __syncwarp();
                }
                {                                            // read-outs of this half's tokens
                    float o[8];
#pragma unroll
                    for (int e = 5; e >= 0; --e) {
                        float y[8];
                        tc_ld8(tm + DC_TD1 + 96 * (e & 1) + 32 * (e >> 1) + 8 * half, y);
#pragma unroll
                        for (int t = 0; t < 8; ++t) o[t] = e == 5 ? y[t] : o[t] + y[t];
                    }
#pragma unroll
                    for (int t = 0; t < 8; ++t) o[t] *= sc[8 * half + t].x;
#pragma unroll
                    for (int s0 = 0; s0 < GC_RUN; s0 += 4) {
                        if (s0 > 8 * half + 7) break;
                        const float u4[4] = {written(s0), written(s0 + 1), written(s0 + 2), written(s0 + 3)};
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            const float4 a = *reinterpret_cast<const float4*>(A + (8 * half + t) * 20 + s0);
                            o[t] = fmaf(a.x, u4[0], fmaf(a.y, u4[1], fmaf(a.z, u4[2], fmaf(a.w, u4[3], o[t]))));
                        }
                    }
                    float sum = 0.f;
#pragma unroll
                    for (int t = 0; t < 8; ++t) sum += o[t];
                    if (__any_sync(0xffffffffu, !(fabsf(sum) < CUDART_INF_F))) {      // zero times a later token's write that is no number: those tokens left out one by one
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            o[t] = 0.f;
#pragma unroll
                            for (int e = 5; e >= 0; --e) {
                                float y[8];
                                tc_ld8(tm + DC_TD1 + 96 * (e & 1) + 32 * (e >> 1) + 8 * half, y);
                                o[t] += y[t];
                            }
                            o[t] *= sc[8 * half + t].x;
#pragma unroll
                            for (int s0 = 0; s0 < GC_RUN; ++s0)
                                if (s0 <= 8 * half + t) o[t] = fmaf(A[(8 * half + t) * 20 + s0], written(s0), o[t]);
                        }
                    }
                    float* const out = p.norm.x + (size_t)(t0 + pos) * p.norm.ldx + (size_t)h * dv + i;
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (8 * half + t < n && i < dv) out[(size_t)(8 * half + t) * p.norm.ldx] = o[t];
                }
                const float f = reinterpret_cast<const float*>(sc)[4 * GC_RUN];
                if (DELTA) {
                    mbar_wait(b_d2, c & 1, 74);
                    tc_fence_after();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        float x[16];
                        tc_ld16(tm + DC_TD2 + 64 * half + 16 * g, x);
#pragma unroll
                        for (int j = 0; j < 16; ++j) S[16 * g + j] = fmaf(S[16 * g + j], f, x[j]);
                    }
                } else {                                     // f32 multiply-adds: the tensor core cuts its sums, which the few roundings of this state would show (7.9e-8 from 64 bits, 8.9e-8 with it)
                    const float* const kc = reinterpret_cast<const float*>(sc) + 128 + i;
                    const f32x2 f2 = pack2(f, f);
                    f32x2 s2[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) s2[j] = prod2(pack2(S[2 * j], S[2 * j + 1]), f2);
#pragma unroll 2
                    for (int t = 0; t < GC_RUN; ++t) {
                        const float kt = kc[t * GC_DMAX];
                        const f32x2 k2 = pack2(kt, kt);
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            const float4 x = *reinterpret_cast<const float4*>(writes + t * GC_DMAX + 64 * half + 2 * j);
                            fma2(s2[j], k2, pack2(x.x, x.y));
                            fma2(s2[j + 1], k2, pack2(x.z, x.w));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float2 x = unpack2(s2[j]);
                        S[2 * j] = x.x; S[2 * j + 1] = x.y;
                    }
                }
                named_bar_sync(1, GC_HALF);                  // all have read the run
                if (tid == 0) mbar_arrive(b_free + 8 * b);
            }
#pragma unroll
            for (int j = 0; j < 64; ++j)
                if (i < dk && 64 * half + j < dv) rec[(size_t)(64 * half + j) * ks * 4] = S[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, DC_TMEM_COLS);
}

}  // namespace b200
