// Latent attention of prompt steps on the tensor cores (serving precision): the function of latent_attn_tc_kernel (latent_attn.cuh), for steps whose keys are not split: many
// tokens, or contexts of fewer than four key tiles of 32 (kx_fill_step).
//
// Queries, latent rows and weights travel as two bf16 parts each (16 bits of a number where the 16-row form rounds to TF32's 11), products as the three of parts that count;
// sums and softmax are f32.  All heads read the same latent row, and its first rk entries are the value too, so one staged tile serves both products.
//
// What bounds it: shared memory and the tensor core's time a launch of few columns takes.  A CTA keeps 64 rows (up to 16 heads x 4 tokens, 8 x 8 and so on), whose queries
// fill 147 KB, and walks the keys 32 at a time:
//   * keys     eight warps (a key a thread) split a tile 128 entries at a time as the MMAs leave them, and ask for the next tile at once:
//              [eight entries][32 high, 32 low][16 bytes], the K-major operand of the scores (high and low parts side by side) and the MN-major operand of the values;
//   * scores   S [64 high, 64 low][32 high, 32 low] = [Q_high; Q_low] [K_high | K_low]^T: all four products of parts in one MMA of full height (products of 64 rows apart took 58 cycles
//              a launch where one of 128 takes 50);
//   * softmax  four warps, a row in two threads (16 keys each) that exchange their halves of the sums.  The weights go to shared memory in parts.  The reference of a row's
//              exponentials follows its maximum only when that has grown by more than e^8 (weights stay below 3000, the division at the end takes the factor out): the
//              accumulator is rescaled in the first tiles and hardly ever later;
//   * values   O^T [channels][64 rows] += V^T P^T, 128 channels a time: full height whatever the rows, channels in lanes, so that the rows go out coalesced.
// Measured (2048 tokens of eight sequences, 16 heads, rows of 576 floats; on mma.sync with TF32 operands and here): 337 -> 148 us from the first token, 685 -> 271 at 256 to 512 tokens
// of context; one prompt of 700 tokens 320 -> 106.  Distance from 64 bits (2-norm): 3.7e-4 -> 5.4e-6.
// Where the line lies: one tile and few heads are level (30 tokens of three sequences, three heads of 32 floats: 14.5 and 14.5 us), 20 tokens of 16 heads 31 -> 24.
#pragma once
#include "bf16_parts.cuh"
#include "latent_attn.cuh"
#include "linear_umma.cuh"

namespace b200 {

constexpr int LP_ROWS = 64, LP_KT = 32, LP_CONV_WARPS = 8, LP_THREADS = 32 * (4 + LP_CONV_WARPS + 1);
constexpr int LP_MAX_D = 576, LP_MAX_RK = 512;               // entries of a latent row; of a value
constexpr uint32_t LP_TS = 256, LP_TMEM_COLS = 512;          // tensor memory: four accumulators of 64 columns, scores
constexpr float LP_SLACK = 8.f;
constexpr int LP_RUN = LP_ROWS * 16, LP_QRUN = 2 * LP_RUN;   // bytes between runs of eight entries of keys, of queries
constexpr int LP_PIECES = (LP_MAX_D + 127) / 128;            // a tile's pieces of 128 entries

struct LatentPromptParams {
    LatentAttnParams a;            // part and nsplit are not read
    float* out;                    // [T, H * rk]
    int hg, qt;                    // heads and tokens of a CTA: hg * qt <= LP_ROWS
};

__host__ __device__ inline int lp_runs(int D) { return 2 * ((D + 15) / 16); }
__host__ __device__ inline int lp_key_runs(int D, int rk) { return lp_runs(D) > 16 * ((rk + 127) / 128) ? lp_runs(D) : 16 * ((rk + 127) / 128); }      // the last 128 channels read past a short row
__host__ __device__ inline size_t latent_prompt_smem(int D, int rk) { return (size_t)(2 * lp_runs(D) + lp_key_runs(D, rk)) * LP_RUN + 2 * LP_ROWS * LP_KT * 2 + 128; }

// a barrier of the four softmax warps that tells whether any thread said so
__device__ __forceinline__ bool lp_any(const bool mine) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((int)mine) : "memory");
    return any != 0;
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

// WHOLE: rows of a multiple of eight floats
template <bool WHOLE>
__global__ void __launch_bounds__(LP_THREADS, 1) latent_prompt_kernel(const __grid_constant__ LatentPromptParams pp) {
    const LatentAttnParams& p = pp.a;
    extern __shared__ __align__(16) uint8_t lp_smem_raw[];
    __shared__ int s_tile[2], s_again[LP_ROWS], s_off[LP_ROWS];      // s_off: a row's place in the output, -1: no row
    __shared__ float s_f[LP_ROWS], s_half[2][LP_ROWS];       // rescaling of a row, later 1 / denominator; what its two threads tell one another
    __shared__ __align__(8) unsigned long long s_bar[4 + 2 * LP_PIECES];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = smem_u32(s_bar), b_q = bar, b_sfull = bar + 8, b_pfull = bar + 16, b_ofull = bar + 24, b_kfull = bar + 32, b_kfree = b_kfull + 8 * LP_PIECES;
    if (tid == 0) {
        mbar_init(b_q, 4 + LP_CONV_WARPS);
        for (int i = 0; i < LP_PIECES; ++i) { mbar_init(b_kfull + 8 * i, LP_CONV_WARPS); mbar_init(b_kfree + 8 * i, 1); }
        mbar_init(b_sfull, 1); mbar_init(b_pfull, 4); mbar_init(b_ofull, 1);
        mbar_fence_init();
    }
    if (warp == LP_THREADS / 32 - 1) tc_alloc(smem_u32(&s_tmem), LP_TMEM_COLS);
    if (tid < LP_ROWS) s_again[tid] = 0;
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
        const int first = s_tile[1] * pp.qt, nt = min(pp.qt, p.meta.slot_count()[si] - first), t0 = p.meta.slot_start()[si] + first;
        const int slot = p.meta.slot_id()[si], pos0 = p.sm.tok_pos()[t0], nkeys = pos0 + nt, ntiles = (nkeys + LP_KT - 1) / LP_KT;
        const int HG = pp.hg, h0 = blockIdx.y * HG, D = p.rk + p.dr, rk = p.rk, nr = lp_runs(D), nch = (rk + 127) / 128;
        const uint32_t raw = smem_u32(lp_smem_raw), sq = (raw + 127u) & ~127u, sk = sq + 2 * nr * LP_RUN, sp = sk + lp_key_runs(D, rk) * LP_RUN;
        uint8_t* const gq = lp_smem_raw + (sq - raw);        // queries [runs][64 high, 64 low][16 bytes]
        uint8_t* const gk = lp_smem_raw + (sk - raw);        // keys [runs][32 high, 32 low][16 bytes]
        uint8_t* const gp = lp_smem_raw + (sp - raw);        // weights [2 parts][4 runs of eight keys][64 rows][16 bytes]; before them sums on their way [2][16 keys][64 rows]
        const int* const tab = p.table + (size_t)slot * p.stride;
        const int r8 = lane & 7, rq = lane >> 3;             // one of eight rows, every fourth run
        if (tid < LP_ROWS) {
            const int qi = tid / HG, h = h0 + tid - qi * HG;
            s_off[tid] = qi < nt && h < p.H ? ((t0 + qi) * p.H + h) * rk : -1;
        }
        if (warp < 4 + LP_CONV_WARPS) {
            // queries: eight rows x four runs a warp and time, four such pieces on their way together
            constexpr int NW = 4 + LP_CONV_WARPS;
            const int pieces = 8 * ((nr + 3) / 4);
            for (int i0 = warp; i0 < pieces; i0 += 4 * NW) {
                float v[4][8];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + u * NW, r = 8 * (i & 7) + r8, run = 4 * (i >> 3) + rq;
                    const int qi = r / HG, h = h0 + r - qi * HG;
                    pt_load8<WHOLE>(v[u], p.q + (size_t)(t0 + qi) * p.H * D + (size_t)h * D + 8 * run, i < pieces && qi < nt && h < p.H ? D - 8 * run : 0);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + u * NW, r = 8 * (i & 7) + r8, run = 4 * (i >> 3) + rq;
                    if (i >= pieces || run >= nr) continue;
                    uint4 part[2];
                    pt_split8(v[u], part);
#pragma unroll
                    for (int e = 0; e < 2; ++e) *reinterpret_cast<uint4*>(gq + (size_t)run * LP_QRUN + e * LP_RUN + r * 16) = part[e];
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(b_q);
        }
        if (warp == LP_THREADS / 32 - 1) {
            // ===================== MMA issuer: one elected lane; the whole warp walks, so that descriptors are uniform values (worked out by one lane, they cost 72 cycles a launch) =====================
            const bool one = elect_one();
            const uint32_t IDS = umma_idesc_bf16(2 * LP_ROWS, 2 * LP_KT), IDO = umma_idesc_bf16(128, LP_ROWS) | (1u << 15);      // values: M contiguous
            // (the address field counts 16 bytes)
            const uint64_t dq = umma_desc(sq, LP_QRUN, 128), dk = umma_desc(sk, LP_RUN, 128), dv = umma_desc(sk, 128, LP_RUN), dp = umma_desc(sp, LP_RUN, 128);
            constexpr uint32_t STEP = 2 * (LP_RUN / 16), PLOW = 4 * (LP_RUN / 16);
            mbar_wait(b_q, 0, 51);
            for (int t = 0; t < ntiles; ++t) {
                for (int c = 0; 16 * c < nr; ++c) {
                    mbar_wait(b_kfull + 8 * c, t & 1, 52);
                    if (c == 0) tc_fence_after();
                    const uint64_t qc = dq + c * (16 * STEP), kc = dk + c * (8 * STEP);
                    if (nr - 16 * c >= 16) {
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (one) tc_mma_f16(tmem + LP_TS, qc + k * (2 * STEP), kc + k * STEP, IDS, c + k > 0);
                    } else {
#pragma unroll 1
                        for (int k = 0; k < (nr - 16 * c) / 2; ++k)
                            if (one) tc_mma_f16(tmem + LP_TS, qc + k * (2 * STEP), kc + k * STEP, IDS, c + k > 0);
                    }
                }
                if (one) tc_commit(b_sfull);
                mbar_wait(b_pfull, t & 1, 53);
                tc_fence_after();
                for (int c = 0; c < nch; ++c) {
                    const uint64_t dc = dv + (uint32_t)(16 * c * (LP_RUN / 16));
#pragma unroll
                    for (int i = 0; i < 3; ++i)              // low V x high P, high x low, high x high
#pragma unroll
                        for (int k = 0; k < LP_KT / 16; ++k)
                            if (one) tc_mma_f16(tmem + c * LP_ROWS, dc + (i == 0 ? 32 : 0) + 16 * k, dp + (i == 1 ? PLOW : 0) + k * STEP, IDO, t > 0 || i + k > 0);
                    if (one && t + 1 < ntiles) tc_commit(b_kfree + 8 * c);
                }
            }
            if (one) tc_commit(b_ofull);
            __syncwarp();
        } else if (warp >= 4) {
            // ===================== latent rows of the cache -> two bf16 parts: a key a thread, eight entries of every eighth run =====================
            const int w = warp - 4, key = 8 * (w & 3) + r8, run0 = 4 * (w >> 2) + rq;
            float x[9][8];
            auto fetch = [&](const int t) {
                const int kj = min(t * LP_KT + key, nkeys - 1);      // rows behind the last key hold the last one's values (their weights are zero)
                const float* const src = p.cache + ((size_t)tab[kj / p.page] * p.page + kj % p.page) * D;
#pragma unroll
                for (int j = 0; j < 9; ++j) pt_load8<WHOLE>(x[j], src + 8 * (run0 + 8 * j), D - 8 * (run0 + 8 * j));
            };
            fetch(0);
            for (int t = 0; t < ntiles; ++t) {
#pragma unroll
                for (int j = 0; j < 9; ++j) {
                    const int run = run0 + 8 * j, c = j >> 1;
                    if (8 * j >= nr) break;
                    // entries that are no values are free when the first values are (their scores came before)
                    if (!(j & 1) && t > 0) mbar_wait(b_kfree + 8 * (c < nch ? c : 0), (t - 1) & 1, 54);
                    if (run < nr) {
                        uint4 part[2];
                        pt_split8(x[j], part);
#pragma unroll
                        for (int e = 0; e < 2; ++e) *reinterpret_cast<uint4*>(gk + (size_t)run * LP_RUN + e * (LP_KT * 16) + key * 16) = part[e];
                    }
                    if ((j & 1) || 8 * (j + 1) >= nr) {      // the piece is whole
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(b_kfull + 8 * c);
                    }
                }
                if (t + 1 < ntiles) fetch(t + 1);            // (during the scores: asked for behind them 294 us where this takes 270, piece by piece as the stores go 293)
            }
        } else {
            // ===================== softmax: row = accumulator row modulo 64, keys 16 half .. of a tile =====================
            const int half = warp >> 1, row = 32 * (warp & 1) + lane, qi = row / HG;
            const uint32_t tm = tmem + ((uint32_t)(32 * warp) << 16);
            const int last = qi < nt && h0 + row - qi * HG < p.H ? pos0 + qi : -1;       // last key the row sees
            float* const gx = reinterpret_cast<float*>(gp);
            float m = -CUDART_INF_F, ref = -CUDART_INF_F, l = 0.f;
            for (int t = 0; t < ntiles; ++t) {
                mbar_wait(b_sfull, t & 1, 55);
                tc_fence_after();
                float s[LP_KT / 2];
                {
                    float a[32], b[32];
                    tc_ld32(tm + LP_TS, a);
                    tc_ld32(tm + LP_TS + LP_KT, b);
                    // the upper warps hold the low queries' sums: each gives the other the half of the keys it works on
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float u = a[j] + b[j], v = a[16 + j] + b[16 + j];
                        s[j] = half ? v : u;
                        gx[(half * 16 + j) * LP_ROWS + row] = half ? u : v;
                    }
                }
                named_bar_sync(1, 128);
                const int left = last - t * LP_KT - 16 * half;
                float mx = -CUDART_INF_F;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    s[j] += gx[((half ^ 1) * 16 + j) * LP_ROWS + row];
                    s[j] = j <= left ? s[j] * p.scale : -CUDART_INF_F;
                    mx = fmaxf(mx, s[j]);
                }
                s_half[half][row] = mx;
                named_bar_sync(1, 128);
                m = fmaxf(m, fmaxf(mx, s_half[half ^ 1][row]));
                const bool grown = m > ref + LP_SLACK;       // (the first score a row sees: from -inf)
                if (lp_any(grown)) {
                    const float f = grown ? (ref > -CUDART_INF_F ? expf(ref - m) : 0.f) : 1.f;
                    if (grown) ref = m;
                    l *= f;
                    if (!half) s_f[row] = f;
                    named_bar_sync(1, 128);
                    if (t > 0)
                        for (int c = 0; c < nch * (LP_ROWS / 16); ++c) {
                            float v[16];
                            uint32_t u[16];
                            tc_ld16(tm + 16 * c, v);
#pragma unroll
                            for (int j = 0; j < 16; ++j) u[j] = __float_as_uint(v[j] * s_f[16 * (c & 3) + j]);
                            tc_st16(tm + 16 * c, u);
                        }
                    tc_wait_st();
                }
                const float base = ref > -CUDART_INF_F ? ref : 0.f;
#pragma unroll
                for (int j = 0; j < 16; ++j) { s[j] = expf(s[j] - base); l += s[j]; }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    float v[8];
                    uint4 part[2];
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = s[8 * q + j];
                    pt_split8(v, part);
#pragma unroll
                    for (int e = 0; e < 2; ++e) *reinterpret_cast<uint4*>(gp + (size_t)(4 * e + 2 * half + q) * LP_RUN + row * 16) = part[e];
                }
                fence_proxy_async_smem();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_pfull);
            }
            s_half[half][row] = l;
            named_bar_sync(1, 128);                          // (nobody reads the rescaling any more)
            if (!half) {
                l += s_half[1][row];
                if (last >= 0 && !(l < CUDART_INF_F)) s_again[row] = 1;
                s_f[row] = 1.f / l;
            }
        }
        __syncthreads();
        mbar_wait(b_ofull, 0, 56);
        tc_fence_after();
        // finished rows: a warp takes 32 channels (its quarter of the lanes) of every third accumulator
        if (warp < 4 + LP_CONV_WARPS) {
            for (int c = warp >> 2; c < nch; c += (4 + LP_CONV_WARPS) / 4) {
                const int ch = 128 * c + 32 * (warp & 3) + lane;
#pragma unroll 1
                for (int g = 0; g < LP_ROWS; g += 16) {
                    float v[16];
                    tc_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c * LP_ROWS + g, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int off = s_off[g + j];
                        if (off < 0 || ch >= rk) continue;
                        if (!(fabsf(v[j]) < CUDART_INF_F)) s_again[g + j] = 1;
                        pp.out[off + ch] = v[j] * s_f[g + j];
                    }
                }
            }
        }
        __syncthreads();
        for (int r = 0; r < LP_ROWS; ++r)
            if (s_again[r] && warp < 8) latent_prompt_row(pp, tab, h0 + r % HG, t0 + r / HG, pos0 + r / HG, 64 * warp, 64);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == LP_THREADS / 32 - 1) tc_dealloc(tmem, LP_TMEM_COLS);
}

}  // namespace b200
