// Projection GEMM of prompt steps (17 .. 128 tokens; from 65 on gemm_pair.cuh where that applies, which leaves launches of a few tiles of a long k and the one-block
// tiles of every length to the forms here):  Y[T, N] = X[T, K] (f16) * W[N, K]^T (f16), f32 accumulate.
//
// Same operands, segments, epilogues and stream-K fix-up as gemm.cuh (its decode kernel reads the same weight blocks); replaces
// the projection dispatches of `Runtime::infer` (reference crates/ai00-core/src/run.rs:1143) in steps that hold a prompt.
//
// What bounds it: the weight stream (a 128 x 64 weight half block is 16 KB and meets 16 KB of tokens).  So a tile takes ALL tokens of
// the step: a weight byte is read once per step.
//   * stages hold 64 k (half a weight block, contiguous in both operands' layouts);
//   * one MMA of N = 16 MT per k16 step; all descriptor fields are compile-time constants.  An MMA of N = 128 takes 64 cycles
//     then (8192 FMA per cycle, the tensor core's rate), N = 256 128;
//   * EIGHT epilogue warps, two per TMEM lane quarter, each draining every second group of 16 tokens straight from TMEM: with
//     four warps holding the whole accumulator in registers the epilogue was longer than the main loop;
//   * partial tiles of a split k range lie in the workspace as [token group][4-token quad][row] float4, so that a warp writes and
//     reads 512 contiguous bytes (one row per lane with the tokens side by side was 32 sectors per request);
//     Measured (100 tokens, 7B widths, ncu): low-rank stages 68 -> 27 and 43 -> 27 us, R/K/V/G 75 -> 42, output 25 -> 18, channel
//     mix 67 -> 45 and 36 -> 32;
//   * launches with at least half as many tiles as SMs give every CTA whole tiles (WIDE_BY_TILE), the others (low-rank stages)
//     cut their block sequence over the SMs and the last arriver of a tile sums the parts in fixed order.
#pragma once
#include "gemm.cuh"

namespace b200 {

constexpr int WIDE_EPI_WARPS = 8, WIDE_EPI_THREADS = WIDE_EPI_WARPS * 32;
constexpr int WIDE_THREADS = WIDE_EPI_THREADS + 64;         // + MMA warp + TMA producer warp
constexpr int WIDE_KS = 64;                                 // k per stage
constexpr int WIDE_STAGE_BUDGET = 204800;

// SHORT: launches whose tiles are one block long (second low-rank stages) are all epilogue: a ring of one block and a single
// accumulator, so that two CTAs share an SM, and up to four CTAs share the token groups of a tile
template <int MT, bool SHORT = false>
struct WideCfg {
    static constexpr int W_BYTES = GEMM_BN * WIDE_KS * 2;   // 16 KB
    static constexpr int A_BYTES = MT * 16 * WIDE_KS * 2;   // 2 KB per 16 tokens
    static constexpr int STAGE_BYTES = W_BYTES + A_BYTES;
    static constexpr int NSTAGE = SHORT ? 2 : WIDE_STAGE_BUDGET / STAGE_BYTES;
    static constexpr int NACC = SHORT ? 1 : 2;              // accumulators
    static constexpr int PAIR = MT >= 4 && !SHORT ? 2 : 1;  // 16-token groups an epilogue warp handles at a time (SHORT: half the registers)
    static constexpr int OUT_HALVES = GEMM_BN * GEMM_STAGE_PITCH;            // transpose buffer of one group (6 KB)
    static constexpr int OUT_BYTES = 2 * PAIR * OUT_HALVES * 2;
    static constexpr int BAR_OFF = NSTAGE * STAGE_BYTES + OUT_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + (2 * NSTAGE + 4) * 8 + 16;
    static constexpr int TMEM_COLS = NACC * 16 * MT < 32 ? 32 : NACC * 16 * MT;     // 32 .. 512 columns
    static_assert(SMEM_BYTES <= 227 * 1024 - 1024, "one CTA per SM, two if SHORT");
};

// block range of a CTA: whole tiles, or an equal share of the block sequence
__device__ __forceinline__ int wide_tile_block(const GemmParams& p, int t) {
    int s = 0;
    while (s + 1 < p.nseg && t >= p.seg[s + 1].tile_begin) ++s;
    return p.seg[s].blk_begin + (t - p.seg[s].tile_begin) * p.seg[s].KB;
}

template <int MT, bool SHORT = false>
__global__ void __launch_bounds__(WIDE_THREADS, SHORT ? 2 : 1) gemm_wide_kernel(const __grid_constant__ GemmParams p, const int by_tile, const int total_tiles) {
    using Cfg = WideCfg<MT, SHORT>;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int s_last;
    __half* const s_out = reinterpret_cast<__half*>(smem + Cfg::NSTAGE * Cfg::STAGE_BYTES);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t full_bar = smem_base + Cfg::BAR_OFF;
    const uint32_t empty_bar = full_bar + Cfg::NSTAGE * 8;
    const uint32_t tfull_bar = empty_bar + Cfg::NSTAGE * 8;
    const uint32_t tempty_bar = tfull_bar + 2 * 8;
    const uint32_t tmem_slot = tempty_bar + 2 * 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long TB = p.total_blocks;
    const int G = gridDim.x, cta = blockIdx.x;
    int b0, b1;
    if (by_tile) {
        const int t0 = (int)((long long)cta * total_tiles / G), t1 = (int)((long long)(cta + 1) * total_tiles / G);
        b0 = wide_tile_block(p, t0);
        b1 = t1 < total_tiles ? wide_tile_block(p, t1) : p.total_blocks;
    } else {
        b0 = (int)((long long)cta * TB / G);
        b1 = (int)((long long)(cta + 1) * TB / G);
    }
    if (tid == 0) {
        trace_stamp(p.trace, 0);
        for (int s = 0; s < Cfg::NSTAGE; ++s) {
            mbar_init(full_bar + s * 8, 1);
            mbar_init(empty_bar + s * 8, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(tfull_bar + s * 8, 1);
            mbar_init(tempty_bar + s * 8, WIDE_EPI_WARPS);
        }
        mbar_fence_init();
    }
    if (warp == WIDE_EPI_WARPS) tc_alloc(tmem_slot, Cfg::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + (tmem_slot - smem_base));
    pdl_launch_dependents();

    if (warp == WIDE_EPI_WARPS + 1) {
        // ===================== producer: one lane streams half blocks =====================
        if (lane == 0) {
            const uint64_t pol_w = l2_policy_evict_first();
            const uint64_t pol_a = l2_policy_evict_last();
            const int nst = 2 * (b1 - b0);
            const uint8_t* W = p.W + (size_t)b0 * GEMM_WBYTES;          // half blocks follow one another
            const int npre = min(nst, Cfg::NSTAGE);
            for (int i = 0; i < npre; ++i) {                            // weights never change: requested before the wait
                mbar_expect_tx(full_bar + i * 8, Cfg::STAGE_BYTES);
                bulk_g2s_hint(smem_base + i * Cfg::STAGE_BYTES, W + (size_t)i * Cfg::W_BYTES, Cfg::W_BYTES, full_bar + i * 8, pol_w);
            }
            pdl_wait();
            if (p.trace && cta == 0 && blockIdx.y == 0) p.trace[2] = globaltimer_ns();      // (trace_stamp is thread 0's)
            int seg = gemm_find_seg(p, b0);
            int kb = (b0 - p.seg[seg].blk_begin) % p.seg[seg].KB, KB = p.seg[seg].KB;
            int left = p.seg[seg].blk_begin + p.seg[seg].tiles * KB - b0;
            // SHORT: blockIdx.z = 128-token tile of a longer step
            auto operand = [&]() {
                const uint8_t* a = reinterpret_cast<const uint8_t*>(p.seg[seg].A);
                return SHORT ? a + ((size_t)(blockIdx.z >> 1) * p.seg[seg].a_tile * A16_KB_HALVES + (size_t)(blockIdx.z & 1) * (A16_KB_HALVES / 2)) * 2 : a;
            };
            const uint8_t* A0 = operand();
            int stage = 0;
            uint32_t ephase = 1;
            for (int i = 0; i < nst; ++i) {
                const uint32_t st = smem_base + stage * Cfg::STAGE_BYTES, fb = full_bar + stage * 8;
                if (i >= Cfg::NSTAGE) {
                    mbar_wait(empty_bar + stage * 8, ephase, 14);
                    mbar_expect_tx(fb, Cfg::STAGE_BYTES);
                    bulk_g2s_hint(st, W + (size_t)i * Cfg::W_BYTES, Cfg::W_BYTES, fb, pol_w);
                }
                // eight k8 chunks of all token rows of the step: contiguous in the A16 layout (common.cuh)
                bulk_g2s_hint(st + Cfg::W_BYTES, A0 + (size_t)kb * (A16_KB_HALVES * 2) + (i & 1) * Cfg::A_BYTES, Cfg::A_BYTES, fb, pol_a);
                if (++stage == Cfg::NSTAGE) { stage = 0; ephase ^= 1; }
                if (i & 1) {
                    if (++kb == KB) kb = 0;
                    if (--left == 0 && i + 1 < nst) {
                        ++seg;
                        kb = 0;
                        KB = p.seg[seg].KB;
                        left = p.seg[seg].tiles * KB;
                        A0 = operand();
                    }
                }
            }
        }
    } else if (warp == WIDE_EPI_WARPS) {
        // ===================== MMA issuer: one lane =====================
        if (lane == 0) {
            constexpr uint32_t IDESC = umma_idesc_f16(GEMM_BN, 16 * MT);
            constexpr uint32_t A_LBO = 16 * MT * 16;        // bytes between the k8 chunks of the token operand
            int stage = 0;
            uint32_t phase = 0;
            unsigned segcount = 0;
            SegWalk w;
            for (w.init(p, b0, b1); !w.done(); w.next(), ++segcount) {
                const int nst = 2 * w.nblk();
                const unsigned acc = segcount % Cfg::NACC, use = segcount / Cfg::NACC;
                if (use > 0) mbar_wait(tempty_bar + acc * 8, (use - 1) & 1u, 11);
                tc_fence_after();
                const uint32_t d0 = tmem_base + acc * (16 * MT);
                uint32_t accumulate = 0;
                for (int i = 0; i < nst; ++i) {
                    mbar_wait(full_bar + stage * 8, phase, 12);
                    tc_fence_after();
                    const uint32_t st = smem_base + stage * Cfg::STAGE_BYTES;
#pragma unroll
                    for (int k16 = 0; k16 < WIDE_KS / 16; ++k16) {
                        tc_mma_f16(d0, umma_desc(st + k16 * 2 * GEMM_W_LBO, GEMM_W_LBO, GEMM_W_SBO),
                                   umma_desc(st + Cfg::W_BYTES + k16 * 2 * A_LBO, A_LBO, GEMM_A_SBO), IDESC, accumulate);
                        accumulate = 1;
                    }
                    tc_commit(empty_bar + stage * 8);
                    if (++stage == Cfg::NSTAGE) { stage = 0; phase ^= 1; }
                }
                tc_commit(tfull_bar + acc * 8);
            }
            if (p.trace) {
                unsigned smid;
                asm volatile("mov.u32 %0, %smid;" : "=r"(smid));
                trace_cta(p.trace, 0, smid);
                trace_cta(p.trace, 1, globaltimer_ns());
            }
        }
    } else {
        // ===================== epilogue: 8 warps; thread = output row, group = every second 16-token group =====================
        pdl_wait();
        if (tid == 0) trace_stamp(p.trace, 5);
        const int nrows = *p.nrows;
        const int grp = warp >> 2, row = tid & (GEMM_BN - 1);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        constexpr int P = Cfg::PAIR;                            // 16-token groups of this warp: mt = grp + 2 i, i in [i0, i1)
        // gridDim.y CTAs share a tile of a SHORT launch: each multiplies all tokens and finishes its share of them
        const int i0 = blockIdx.y * (MT / 2) / gridDim.y, i1 = (blockIdx.y + 1) * (MT / 2) / gridDim.y;
        const int m0 = SHORT ? (int)blockIdx.z * (16 * MT) : 0;     // first token of this CTA's tile
        unsigned segcount = 0;
        SegWalk w;
        for (w.init(p, b0, b1); !w.done(); w.next(), ++segcount) {
            const GemmSeg& sg = p.seg[w.seg];
            const unsigned acc = segcount % Cfg::NACC, use = segcount / Cfg::NACC;
            mbar_wait(tfull_bar + acc * 8, use & 1u, 13);
            tc_fence_after();
            const uint32_t tm = tmem_base + lane_base + acc * (16 * MT);
            int ncontrib = 1, c_first = 0;
            const int gtile = sg.tile_begin + w.tile_local;
            if (!by_tile) {
                const unsigned tb0 = (unsigned)(sg.blk_begin + w.tile_local * sg.KB);
                c_first = (int)(((unsigned long long)(tb0 + 1) * (unsigned)G - 1) / (unsigned)TB);
                const int c_last = (int)(((unsigned long long)(tb0 + sg.KB) * (unsigned)G - 1) / (unsigned)TB);
                ncontrib = c_last - c_first + 1;
            }
            auto drained = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar + acc * 8);
            };
            float* const ws0 = p.ws + (size_t)gtile * p.max_contrib * (GEMM_BN * 16 * MT) + row * 4;
            if (ncontrib > 1) {
                float* const mine = ws0 + (size_t)(cta - c_first) * (GEMM_BN * 16 * MT);
#pragma unroll 1
                for (int i = i0; i < i1; ++i) {
                    const int mt = grp + 2 * i;
                    float v[16];
                    tc_ld16(tm + mt * 16, v);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<float4*>(mine + (size_t)(mt * 4 + j) * (GEMM_BN * 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                drained();
                // publish: the barrier orders every thread's stores before thread 0's gpu-scope release, one counter bump per CTA
                named_bar_sync(1, WIDE_EPI_THREADS);
                if (tid == 0) {
                    const unsigned old = atom_add_acq_rel_gpu(p.counters + gtile, 1u);
                    s_last = (old == (unsigned)(ncontrib - 1));
                    if (s_last) p.counters[gtile] = 0;
                }
                named_bar_sync(1, WIDE_EPI_THREADS);
                if (!*(volatile int*)&s_last) continue;
            }
            const int n = w.tile_local * GEMM_BN + row;
            const int segN = sg.N, out_mode = sg.out_mode, ldo = sg.ldo;
            const bool row_ok = n < segN, lerp = (out_mode == OUT_LERP_A16);
            const float bias = (row_ok && sg.bias) ? sg.bias[n] : 0.f;
            const float mu = (lerp && row_ok) ? sg.aux2[n] : 0.f;
            const int mmax = min(nrows - m0, MT * 16);         // tokens of the tile
            // the 16-token groups i .. i + P - 1: accumulators (TMEM, or the parts in contributor order, all loads of two contributors in flight)
            auto load = [&](const int i, float (&v)[P][16]) {
                if (SHORT || ncontrib == 1) {
#pragma unroll
                    for (int q = 0; q < P; ++q) tc_ld16(tm + (grp + 2 * (i + q)) * 16, v[q]);
                    return;
                }
#pragma unroll
                for (int q = 0; q < P; ++q)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[q][j] = 0.f;
                for (int s0 = 0; s0 < ncontrib; s0 += 2) {
                    float4 x[2][P][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int q = 0; q < P; ++q) {
                            const float* src = ws0 + (size_t)(s0 + u) * (GEMM_BN * 16 * MT) + (size_t)((grp + 2 * (i + q)) * 4) * (GEMM_BN * 4);
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                x[u][q][j] = s0 + u < ncontrib ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)j * (GEMM_BN * 4))) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int q = 0; q < P; ++q)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                v[q][4 * j] += x[u][q][j].x; v[q][4 * j + 1] += x[u][q][j].y; v[q][4 * j + 2] += x[u][q][j].z; v[q][4 * j + 3] += x[u][q][j].w;
                            }
                }
            };
            auto body = [&](auto act_c) {
                constexpr int ACT_C = decltype(act_c)::value;
#pragma unroll 1
                for (int i = i0; i < i1; i += P) {
                    float v[P][16];
                    load(i, v);
                    if (ncontrib == 1 && i + P >= i1) drained();
                    if (out_mode == OUT_F32) {
                        if (row_ok) {
                            float* o = reinterpret_cast<float*>(sg.out) + (size_t)m0 * ldo + n;
#pragma unroll
                            for (int q = 0; q < P; ++q)
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    const int m = (grp + 2 * (i + q)) * 16 + j;
                                    if (m < mmax) o[(size_t)m * ldo] = apply_act(v[q][j] + bias, ACT_C);
                                }
                        }
                        continue;
                    }
                    // A16 outputs: transposed through shared memory into 16-byte chunks of 8 rows (see gemm.cuh)
                    if ((grp + 2 * i) * 16 >= mmax) continue;            // uniform over the 128 threads of the group
                    if (lerp) {
                        float x0[P][16], x1[P][16];                     // operands of the tokens, requested together
#pragma unroll
                        for (int q = 0; q < P; ++q)
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int m = (grp + 2 * (i + q)) * 16 + j;
                                const bool ok = row_ok && m < mmax;
                                const size_t a_ = (size_t)(m0 + m) * sg.ld_aux + n;
                                x0[q][j] = ok ? sg.aux0[a_] : 0.f;
                                x1[q][j] = ok ? sg.aux1[a_] : 0.f;
                            }
#pragma unroll
                        for (int q = 0; q < P; ++q)
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[q][j] = x0[q][j] + x1[q][j] * (mu + apply_act(v[q][j] + bias, ACT_C));
                    } else {
#pragma unroll
                        for (int q = 0; q < P; ++q)
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[q][j] = apply_act(v[q][j] + bias, ACT_C);
                    }
                    __half* const stage = s_out + grp * P * Cfg::OUT_HALVES;
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        uint4 h0, h1;
                        h0.x = pack_h2(v[q][0], v[q][1]); h0.y = pack_h2(v[q][2], v[q][3]); h0.z = pack_h2(v[q][4], v[q][5]); h0.w = pack_h2(v[q][6], v[q][7]);
                        h1.x = pack_h2(v[q][8], v[q][9]); h1.y = pack_h2(v[q][10], v[q][11]); h1.z = pack_h2(v[q][12], v[q][13]); h1.w = pack_h2(v[q][14], v[q][15]);
                        if (!row_ok) h0 = h1 = make_uint4(0, 0, 0, 0);
                        uint4* dst = reinterpret_cast<uint4*>(stage + q * Cfg::OUT_HALVES + row * GEMM_STAGE_PITCH);
                        dst[0] = h0; dst[1] = h1;
                    }
                    named_bar_sync(2 + grp, GEMM_BN);
                    const int row0 = w.tile_local * GEMM_BN;
#pragma unroll
                    for (int q = 0; q < 2 * P; ++q) {
                        const int e = row + GEMM_BN * (q & 1), mt = grp + 2 * (i + (q >> 1));
                        const int c = e >> 4, m = e & 15, nc = row0 + c * 8;
                        if (nc < segN && mt * 16 + m < mmax) {
                            const __half* src = stage + (q >> 1) * Cfg::OUT_HALVES + (c * 8) * GEMM_STAGE_PITCH + m;
                            uint32_t r[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                r[k] = (uint32_t)__half_as_ushort(src[2 * k * GEMM_STAGE_PITCH]) | ((uint32_t)__half_as_ushort(src[(2 * k + 1) * GEMM_STAGE_PITCH]) << 16);
                            __half* base = reinterpret_cast<__half*>(sg.out);
                            int nn = nc;
                            if (sg.grp > 0) {
                                const int gi = nc / sg.grp;
                                base += (size_t)gi * sg.grp_stride;
                                nn = nc - gi * sg.grp;
                            }
                            *reinterpret_cast<uint4*>(base + a16_index(m0 + mt * 16 + m, nn, ldo)) = make_uint4(r[0], r[1], r[2], r[3]);
                        }
                    }
                    named_bar_sync(2 + grp, GEMM_BN);
                }
            };
            switch (sg.act) {
                case ACT_TANH: body(std::integral_constant<int, ACT_TANH>{}); break;
                case ACT_SIGMOID: body(std::integral_constant<int, ACT_SIGMOID>{}); break;
                case ACT_SILU: body(std::integral_constant<int, ACT_SILU>{}); break;
                case ACT_RELU2: body(std::integral_constant<int, ACT_RELU2>{}); break;
                case ACT_EXPNEGEXP: body(std::integral_constant<int, ACT_EXPNEGEXP>{}); break;
                case ACT_V7DECAY: body(std::integral_constant<int, ACT_V7DECAY>{}); break;
                default: body(std::integral_constant<int, ACT_NONE>{}); break;
            }
        }
        if (tid == 0) trace_stamp(p.trace, 6);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        trace_stamp(p.trace, 7);
        if (p.trace) trace_cta(p.trace, 2, globaltimer_ns());
    }
    if (warp == WIDE_EPI_WARPS) tc_dealloc(tmem_base, Cfg::TMEM_COLS);
}

}  // namespace b200
