// Softmax attention of prompt steps over the paged cache on the tensor cores: the function of sink_attn.cuh (windows, chunks of the sequence, kept first tokens, a bias per
// distance, a sink term, a gate; no block means), for steps whose keys are not split: enough tokens to fill the chip, or contexts of one key tile of 32 (kx_fill_step).
//
// Queries, keys, values and weights are f32 and stay it: each number travels as three bf16 parts (the first two rounded to nearest, the third takes what is left: 24 bits),
// and a product of two numbers is the six products of parts down to 2^-16 of the first; what is left out is 2^-24 of a product.  The small products are summed first, so
// that eight additions of a score and four of a tile's read-out happen at full size; read-outs of a tile are added to the row in f32 registers.
//
// What bounds it: the tensor core, six times the products of a bf16 kernel (f32 multiply-adds, the form before, take 128 a cycle and SM; these 4096 / 6).  A CTA keeps
// 128 rows -- the query heads of ONE key / value head for 128 / rep consecutive tokens of a sequence -- and walks the keys in tiles of 64:
//   * queries  live in tensor memory (three parts of 64 columns), so that a score MMA reads only the key tile from shared memory;
//   * keys and values   are split by four warps each on the way into shared memory, [eight channels][64 keys][16 bytes]: one layout is the K-major operand of the
//              scores and the MN-major operand of the values;
//   * scores   S = Q K^T, 64 columns of tensor memory; eight warps take half a row each a thread, exchange maxima, and write the weights back as three parts;
//   * values   O = P V, a fresh accumulator every tile, added to the rows' registers one tile later;
//   * one lane issues: the scores of tile t + 1 are multiplied while the softmax of tile t runs, the values of tile t while that of t + 1 does; seven warps split the
//              tiles ahead of it (16 of eight keys a tile, dealt out), two buffers each for keys and values.
// Measured (16 sequences of 128 tokens, 16 query heads on 4 key heads of 128 channels, in f32 multiply-adds before and here): 113 -> 34 us at 128 tokens of context, 454 -> 76 at
// 576, 805 -> 122 at 1024 (130 with descriptors worked out by the issuing lane alone); one prompt of 1000 tokens 376 -> 59, of 20 tokens 25 -> 15; 16 prompts of 1024 tokens, four
// layers of width 2048, 22.1 -> 15.7 ms.  Distance from 64 bits (2-norm): 6.2e-7 -> 3.0e-7 at 1024 tokens, 1.42e-6 -> 3.5e-7 at 6000, 1.6e-7 -> 1.4e-7 at 20.
// Where most rows are empty and the context is a tile the multiply-add form is the better one (64 sequences of 32 tokens, one query head a key head, 32 channels: 64 -> 74 us): short_attn.cuh.
#pragma once
#include "bf16_parts.cuh"
#include "linear_umma.cuh"
#include "sink_attn.cuh"

namespace b200 {

constexpr int PT_ROWS = 128, PT_KT = 64, PT_DMAX = 128;
constexpr int PT_SOFT = 256, PT_CONV_WARPS = 7, PT_THREADS = PT_SOFT + 32 * PT_CONV_WARPS + 32;      // sixteen warps: 128 registers a thread
// tensor memory: queries (3 x 64 columns), scores, weights (3 x 32), read-outs of a tile
constexpr uint32_t PT_TQ = 0, PT_TS = 192, PT_TP = 256, PT_TO = 352, PT_TMEM_COLS = 512;

struct PromptAttnParams {
    SinkAttnParams a;
    int qt;                        // tokens of a CTA: PT_ROWS / (query heads of a key head)
};

__host__ __device__ inline int pt_up16(int d) { return (d + 15) & ~15; }
// two key tiles and two value tiles in three parts, later the finished rows
__host__ __device__ inline size_t prompt_attn_smem(int dk, int dv) {
    const size_t tiles = (size_t)2 * 3 * PT_KT * 2 * (pt_up16(dk) + pt_up16(dv)), out = (size_t)PT_ROWS * (pt_up16(dv) + 4) * 4;
    return (tiles > out ? tiles : out) + 128;
}

// One row (token t at position pos, query head h of key head c) worked out again by a warp, key by key.  A key behind a token has weight zero in the tiles below, and zero times a
// value that is not finite is not a number: a later token of the CTA's rows would reach the earlier ones; and parts of a number that is not finite are not numbers.  Only
// rows that came out so get here.
__device__ __noinline__ void prompt_attn_row(const SinkAttnParams& p, const float* q, const int* tbl, int c, int h, int t, int pos) {
    const int lane = threadIdx.x & 31, d = 4 * lane, low = sa_low(p, pos);
    int nkeep, jlo;
    sa_segments(p, pos, pos, nkeep, jlo);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), qv = d < p.dk ? *reinterpret_cast<const float4*>(q + d) : zero;
    float4 acc = zero;
    float m = -CUDART_INF_F, l = 0.f;
    for (int i = 0; i < nkeep + pos - jlo + 1; ++i) {
        const int at = i < nkeep ? i : jlo + i - nkeep;
        if (at > pos || (at < low && at >= p.keep)) continue;
        const float* row = p.cache + sa_token_row(tbl, p.page, at) * (size_t)p.D;
        const float4 k = d < p.dk ? *reinterpret_cast<const float4*>(row + p.koff + (size_t)c * p.dk + d) : zero;
        const float4 v = d < p.dv ? *reinterpret_cast<const float4*>(row + p.voff + (size_t)c * p.dv + d) : zero;
        float dot = fmaf(qv.x, k.x, fmaf(qv.y, k.y, fmaf(qv.z, k.z, qv.w * k.w)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float sc = dot * p.scale + (p.bias ? p.bias[(size_t)h * (p.nb + 1) + min(pos - at, p.nb)] : 0.f);
        const float mn = fmaxf(m, sc), w = sc > -CUDART_INF_F ? expf(sc - mn) : 0.f, scl = m > -CUDART_INF_F ? expf(m - mn) : 0.f;
        l = l * scl + w;
        m = mn;
        acc.x = fmaf(w, v.x, acc.x * scl); acc.y = fmaf(w, v.y, acc.y * scl); acc.z = fmaf(w, v.z, acc.z * scl); acc.w = fmaf(w, v.w, acc.w * scl);
    }
    if (d >= p.dv) return;
    const float sk = p.sink ? p.sink[h] : -CUDART_INF_F, mx = fmaxf(m, sk), f0 = m > -CUDART_INF_F ? expf(m - mx) : 0.f;
    const float f = f0 / (l * f0 + (p.sink ? expf(sk - mx) : 0.f));
    const float o[4] = {acc.x * f, acc.y * f, acc.z * f, acc.w * f};
    for (int e = 0; e < 4; ++e) {
        const float g = p.gate ? lin_sigmoid(p.gate[(size_t)t * p.ldg + (p.gate_heads ? (size_t)h : (size_t)h * p.dv + d + e)]) : 1.f;
        p.out[(size_t)t * p.ldo + (size_t)h * p.dv + d + e] = o[e] * g * p.out_mul;
    }
}

// RUNS: runs of eight channels of keys and values (16), 0: any.  WHOLE: sizes, strides and offsets are multiples of eight floats
template <int RUNS, bool WHOLE>
__global__ void __launch_bounds__(PT_THREADS, 1) prompt_attn_kernel(const __grid_constant__ PromptAttnParams pp) {
    const SinkAttnParams& p = pp.a;
    extern __shared__ __align__(16) uint8_t pt_smem_raw[];
    __shared__ int s_tile[2], s_again[PT_ROWS], s_hi[PT_ROWS], s_lo[PT_ROWS], s_kept[PT_ROWS];
    __shared__ float s_max[2][2][PT_ROWS], s_sum[PT_ROWS], s_gate[PT_ROWS];
    __shared__ int s_off[PT_ROWS];
    __shared__ __align__(8) unsigned long long s_bar[13];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = smem_u32(s_bar);
    // (key and value tiles have two buffers)
    const uint32_t b_q = bar, b_kfull = bar + 8, b_kfree = bar + 24, b_vfull = bar + 40, b_vfree = bar + 56, b_sfull = bar + 72, b_sfree = bar + 80, b_pfull = bar + 88,
                   b_ofull = bar + 96;
    if (tid == 0) {
        mbar_init(b_q, PT_SOFT / 32);
        for (int i = 0; i < 16; i += 8) {
            mbar_init(b_kfull + i, PT_KT / 8); mbar_init(b_kfree + i, 1);
            mbar_init(b_vfull + i, PT_KT / 8); mbar_init(b_vfree + i, 1);
        }
        mbar_init(b_sfull, 1); mbar_init(b_sfree, PT_SOFT / 32);
        mbar_init(b_pfull, PT_SOFT / 32); mbar_init(b_ofull, 1);
        mbar_fence_init();
    }
    if (warp == PT_THREADS / 32 - 1) tc_alloc(smem_u32(&s_tmem), PT_TMEM_COLS);
    if (tid < PT_ROWS) s_again[tid] = 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&s_tmem);
    pdl_launch_dependents();                                // behind the allocation: see linear_umma.cuh
    pdl_wait();
    if (warp == 0) step_token_run_back(p.meta, pp.qt, blockIdx.x, s_tile);
    __syncthreads();
    const int si = s_tile[0];
    if (si >= 0) {
        const int first = s_tile[1] * pp.qt, nq = min(pp.qt, p.meta.slot_count()[si] - first), t0 = p.meta.slot_start()[si] + first;
        const int slot = p.meta.slot_id()[si], pos0 = p.sm.tok_pos()[t0], pos1 = pos0 + nq - 1;
        const int dk = RUNS ? 8 * RUNS : p.dk, dv = RUNS ? 8 * RUNS : p.dv, rep = p.H / p.G, c = blockIdx.y, R = nq * rep, D = p.D;
        const int nck = RUNS ? RUNS : pt_up16(dk) / 8, ncv = RUNS ? RUNS : pt_up16(dv) / 8;      // runs of eight channels
        const uint32_t raw = smem_u32(pt_smem_raw), tiles = (raw + 127u) & ~127u;
        uint8_t* const sK = pt_smem_raw + (tiles - raw);                     // [2 tiles][3 parts][runs][64 keys][16 bytes]
        uint8_t* const sV = sK + (size_t)6 * nck * PT_KT * 16;
        const int* const tbl = p.table + (size_t)slot * p.stride;
        int nkeep, jlo;
        sa_segments(p, pos0, pos1, nkeep, jlo);
        const int nkeys = nkeep + pos1 - jlo + 1, ntiles = (nkeys + PT_KT - 1) / PT_KT;
        auto position = [&](int i) { return i < nkeep ? i : jlo + i - nkeep; };      // kept tokens first, then the window

        if (warp == PT_THREADS / 32 - 1) {
            // ===================== MMA issuer: one elected lane; the whole warp walks, so that descriptors are uniform values =====================
            const bool one = elect_one();
            const uint32_t IDESC_S = umma_idesc_bf16(PT_ROWS, PT_KT), IDESC_O = umma_idesc_bf16(PT_ROWS, 8 * ncv) | (1u << 16);      // values: N contiguous
            constexpr uint32_t RUN = PT_KT * 16;             // bytes between runs of eight channels
            // (the address field counts 16 bytes)
            const uint64_t dk0 = umma_desc(tiles, RUN, 128), dv0 = umma_desc(tiles + 6 * nck * RUN, 128, RUN);
            constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // parts of a product, the smallest first
            const uint32_t kpart = nck * (RUN / 16), vpart = ncv * (RUN / 16);
            auto values = [&](const int t) {
                const int b = t & 1;
                mbar_wait(b_vfull + 8 * b, (t >> 1) & 1, 41);
                mbar_wait(b_pfull, b, 42);
                tc_fence_after();
                const uint64_t d0 = dv0 + 3 * b * vpart;
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int k = 0; k < PT_KT / 16; ++k)
                        if (one) tc_mma_f16_ts(tmem + PT_TO, tmem + PT_TP + PA[i] * 32 + k * 8, d0 + PB[i] * vpart + k * 16, IDESC_O, i + k > 0);
                if (one && t + 2 < ntiles) tc_commit(b_vfree + 8 * b);
                if (one) tc_commit(b_ofull);
            };
            mbar_wait(b_q, 0, 43);
            for (int t = 0; t < ntiles; ++t) {
                const int b = t & 1;
                mbar_wait(b_kfull + 8 * b, (t >> 1) & 1, 44);
                if (t > 0) mbar_wait(b_sfree, (t - 1) & 1, 45);
                tc_fence_after();
                const uint64_t d0 = dk0 + 3 * b * kpart;
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int k = 0; k < PT_DMAX / 16; ++k)
                        if (2 * k < nck && one) tc_mma_f16_ts(tmem + PT_TS, tmem + PT_TQ + PA[i] * 64 + k * 8, d0 + PB[i] * kpart + 2 * k * (RUN / 16), IDESC_S, i + k > 0);
                if (one && t + 2 < ntiles) tc_commit(b_kfree + 8 * b);
                if (one) tc_commit(b_sfull);
                if (t > 0) values(t - 1);
            }
            values(ntiles - 1);
            __syncwarp();
        } else if (warp >= PT_SOFT / 32) {
            // ===================== f32 rows of the cache -> three bf16 parts: eight keys of a key or value tile at a time, dealt out among the warps =====================
            const int k8 = lane & 7, cq = lane >> 3;         // a key of the eight, every fourth run of eight channels
            const float* const base = p.cache + (size_t)c * dk + p.koff;
            const ptrdiff_t vgap = (ptrdiff_t)p.voff + (size_t)c * dv - ((ptrdiff_t)p.koff + (size_t)c * dk);
            // rows behind the last key hold the last one's values (their weights are zero)
            auto locate = [&](const int n) {
                return base + (n & 8 ? vgap : 0) + sa_token_row(tbl, p.page, position(min((n >> 4) * PT_KT + (n & 7) * 8 + k8, nkeys - 1))) * (size_t)D;
            };
            auto fetch = [&](const int n, const float* const src, float (&x)[4][8]) {
                const int d = n & 8 ? dv : dk;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int ch = 8 * (4 * q + cq);
                    pt_load8<WHOLE>(x[q], src + ch, d - ch);
                }
            };
            auto store = [&](const int n, float (&x)[4][8]) {
                const bool isv = n & 8;
                const int t = n >> 4, b = t & 1, nc = isv ? ncv : nck;
                if (t > 1) mbar_wait((isv ? b_vfree : b_kfree) + 8 * b, ((t >> 1) - 1) & 1, 46);
                uint8_t* const to = (isv ? sV : sK) + (size_t)b * 3 * nc * (PT_KT * 16) + ((n & 7) * 8 + k8) * 16;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int run = 4 * q + cq;
                    if (run >= nc) continue;
                    uint4 part[3];
                    pt_split8(x[q], part);
#pragma unroll
                    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(to + (size_t)(i * nc + run) * (PT_KT * 16)) = part[i];
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive((isv ? b_vfull : b_kfull) + 8 * b);
            };
            const int total = 16 * ntiles;
            int n = warp - PT_SOFT / 32;
            float x0[4][8], x1[4][8];
            fetch(n, locate(n), x0);                         // (there are sixteen at least)
            const float* src = locate(n + PT_CONV_WARPS);
            // the next eight keys are on their way while these are split, the page of those behind them is being looked up
            for (; n < total; n += 2 * PT_CONV_WARPS) {
                const int n1 = n + PT_CONV_WARPS, n2 = n + 2 * PT_CONV_WARPS;
                if (n1 < total) fetch(n1, src, x1);
                src = locate(n2);
                store(n, x0);
                if (n2 < total) fetch(n2, src, x0);
                src = locate(n2 + PT_CONV_WARPS);
                if (n1 < total) store(n1, x1);
            }
        } else {
            // ===================== softmax: thread = (row, half of the tile's keys, half of the output's channels) =====================
            const int half = warp >> 2, row = tid & (PT_ROWS - 1);
            const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            {
                const bool in = row < R;
                const int tq = row / rep, h = c * rep + row - tq * rep;
                // Key idx of the walk is visible if idx <= hi and (idx >= lo or idx < kept): the row's own position and window in the walk's count (rows beyond the last see
                // nothing; the kept tokens lie before every row's window).  In shared memory: the loop below has no registers to spare; either half writes the same
                const int pq = in ? pos0 + tq : -1, shift = jlo - nkeep;
                s_hi[row] = pq - shift; s_lo[row] = sa_low(p, pq) - shift; s_kept[row] = max(p.keep - shift, nkeep);
                s_off[row] = in ? (t0 + tq) * p.ldo + h * dv : -1;
                s_gate[row] = in && p.gate && p.gate_heads ? p.gate[(size_t)(t0 + tq) * p.ldg + h] : 0.f;
                const float* const qrow = p.q + (size_t)(t0 + tq) * p.ldq + (size_t)h * dk;
                float v[8][8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int d = 64 * half + 8 * i;
                    pt_load8<WHOLE>(v[i], qrow + d, in ? dk - d : 0);
                }
#pragma unroll
                for (int part = 0; part < 3; ++part)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {            // 32 channels: 16 columns of the part
                        uint32_t r[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) r[i] = pt_take(v[4 * e + i / 4][2 * (i & 3)], v[4 * e + i / 4][2 * (i & 3) + 1]);
                        tc_st16(tm + PT_TQ + part * 64 + half * 32 + e * 16, r);
                    }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_q);
            }
            const int low1 = sa_low(p, pos1);
            float m = -CUDART_INF_F, l = 0.f, scl = 0.f;
            float o[64];
#pragma unroll
            for (int i = 0; i < 64; ++i) o[i] = 0.f;
            auto add_tile = [&]() {                          // read-outs of a finished tile, whose rescaling of the row is `scl`
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (64 * half + 16 * q >= 8 * ncv) break;
                    float v[16];
                    tc_ld16(tm + PT_TO + 64 * half + 16 * q, v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[16 * q + i] = fmaf(o[16 * q + i], scl, v[i]);
                }
            };
            for (int t = 0; t < ntiles; ++t) {
                mbar_wait(b_sfull, t & 1, 48);
                tc_fence_after();
                float s[32];
                tc_ld32(tm + PT_TS + 32 * half, s);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_sfree);
                // does every row see every key of the tile?
                const int i0 = t * PT_KT, a0 = position(i0), a1 = position(i0 + PT_KT - 1);
                float mx = -CUDART_INF_F;
                if (i0 + PT_KT <= nkeys && i0 >= nkeep && a1 <= pos0 && a0 >= low1 && !p.bias) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) { s[j] *= p.scale; mx = fmaxf(mx, s[j]); }
                } else {
                    const int i1 = i0 + 32 * half, hj = s_hi[row] - i1, lj = s_lo[row] - i1, kj = s_kept[row] - i1;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const bool vis = j <= hj && (j >= lj || j < kj);
                        s[j] = vis ? s[j] * p.scale : -CUDART_INF_F;
                    }
                    if (p.bias && row < R) {
                        const float* const bias = p.bias + (size_t)(c * rep + row % rep) * (p.nb + 1);
                        const int pq = pos0 + row / rep;
#pragma unroll
                        for (int j = 0; j < 32; ++j) s[j] += bias[min(max(pq - position(i1 + j), 0), p.nb)];
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) mx = fmaxf(mx, s[j]);
                }
                s_max[t & 1][half][row] = mx;
                named_bar_sync(1, PT_SOFT);
                const float mn = fmaxf(m, fmaxf(mx, s_max[t & 1][half ^ 1][row])), ref = mn > -CUDART_INF_F ? mn : 0.f;
                const float now = m > -CUDART_INF_F ? expf(m - mn) : 0.f;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 32; ++j) { s[j] = expf(s[j] - ref); sum += s[j]; }
                l = l * now + sum;
                m = mn;
                uint32_t r[3][16];
#pragma unroll
                for (int part = 0; part < 3; ++part)
#pragma unroll
                    for (int i = 0; i < 16; ++i) r[part][i] = pt_take(s[2 * i], s[2 * i + 1]);
                if (t > 0) {                                 // the MMAs of tile t - 1 have read its weights
                    mbar_wait(b_ofull, (t - 1) & 1, 47);
                    tc_fence_after();
                }
#pragma unroll
                for (int part = 0; part < 3; ++part) tc_st16(tm + PT_TP + part * 32 + half * 16, r[part]);
                if (t > 0) add_tile();
                scl = now;
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_pfull);
            }
            mbar_wait(b_ofull, (ntiles - 1) & 1, 47);
            tc_fence_after();
            add_tile();
            // both halves' sums; the sink joins the denominator.  Every MMA has completed: the tiles' memory takes the rows
            if (half == 1) s_sum[row] = l;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 64; ++i) sum += o[i];
            const bool in = row < R;
            if (in && !(fabsf(sum) < CUDART_INF_F)) s_again[row] = 1;
            named_bar_sync(1, PT_SOFT);
            if (half == 0) {
                l += s_sum[row];
                const float sk = p.sink && in ? p.sink[c * rep + row % rep] : -CUDART_INF_F, mx = fmaxf(m, sk), f = m > -CUDART_INF_F ? expf(m - mx) : 0.f;
                s_sum[row] = f / (l * f + (p.sink ? expf(sk - mx) : 0.f)) * (p.gate && p.gate_heads ? lin_sigmoid(s_gate[row]) : 1.f);
                if (in && !(l < CUDART_INF_F)) s_again[row] = 1;
            }
            float* const out = reinterpret_cast<float*>(sK);
            const int pitch = 8 * ncv + 4;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (64 * half + 4 * q < 8 * ncv) *reinterpret_cast<float4*>(out + row * pitch + 64 * half + 4 * q) = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            named_bar_sync(1, PT_SOFT);
            const float mul = p.out_mul;
            if (p.gate == nullptr || p.gate_heads) {
#pragma unroll 4
                for (int r = warp; r < PT_ROWS; r += 8) {
                    const int off = s_again[r] ? -1 : s_off[r];
                    const float f = s_sum[r];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int d = 32 * q + lane;
                        if (off >= 0 && d < dv) p.out[off + d] = out[r * pitch + d] * f * mul;
                    }
                }
            } else {
                for (int r = warp; r < R; r += 8) {
                    if (s_again[r]) continue;
                    const float* const g = p.gate + (size_t)(t0 + r / rep) * p.ldg + (size_t)(c * rep + r % rep) * dv;
                    for (int d = lane; d < dv; d += 32) p.out[s_off[r] + d] = out[r * pitch + d] * s_sum[r] * lin_sigmoid(g[d]) * mul;
                }
            }
            for (unsigned left = __ballot_sync(0xffffffffu, lane < PT_ROWS / 8 && s_again[warp + 8 * (lane & 15)]); left; left &= left - 1) {
                const int r = warp + 8 * (__ffs(left) - 1), t = t0 + r / rep, hr = c * rep + r % rep;
                prompt_attn_row(p, p.q + (size_t)t * p.ldq + (size_t)hr * dk, tbl, c, hr, t, pos0 + r / rep);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == PT_THREADS / 32 - 1) tc_dealloc(tmem, PT_TMEM_COLS);
}

}  // namespace b200
