// Grouped linear layers of linear.cuh on tcgen05, for steps of more than 16 rows in serving precision: same problem (Y = epi(X W^T),
// groups, device-side row counts and row lists, epilogues), same operand rounding (f32 activations rounded to bf16 once), f32 sums.
//
//   lin_pack_kernel   f32 activations of every group -> bf16 rows [row][K] in a workspace (gathered through the row list)
//   lin_umma_kernel   one persistent CTA per SM (PAIR: two, see below) walks the units (group, 128 outputs, TN rows, k range):
//     * the WEIGHT tile is the 128-row operand, TN rows of activations the other: an output row is a TMEM lane, so that a warp stores
//       32 neighbouring outputs of one row, bias and (gate, up) pairs sit in neighbouring lanes, and weights stay as stored
//       (row-major bf16) -- both operands arrive as 64-wide k boxes in the 128-byte swizzle, edges of N, K and the rows zero filled;
//     * warp roles: TMA producer, MMA issuer, eight epilogue warps that drain one accumulator while the next unit's MMAs run;
//     * units of empty groups do not exist: the walk is over the row counts the step (or the router) left on the device;
//     * launches with fewer units than SMs cut k: every part leaves its raw sums in the workspace and the last arriver adds the parts in
//       order and runs the epilogue.
//   PAIR              clusters of two CTAs share a unit of 256 outputs and TN rows (tcgen05 cta_group::2, gemm_pair.cuh): each holds its 128 weight
//                     rows, half of the activation rows and the accumulators of its outputs, and takes in half the bytes for the same work.
//
// What bounds it: 16 KB of weights and TN x 128 B of rows per 64 k against 4 MMAs of 64 cycles (TN = 128), i.e. the bytes an SM
// pulls from L2; lin_tile_kernel (mma.sync on 64 x 64 tiles, f32 activations through shared memory) ran at 5-9 % of the tensor pipe.
// Measured with PAIR (width 2048, ncu): the 17 projections of four steps of 512 tokens 2295 us, of one step of 2048 now about 1000; 16 prompts of 1024 tokens
// 47.8 -> 32.5 ms, eight documents 7.7 -> 5.1 ms.
// Measured before that: the 17 projections of a 512-token step (four layers of width 2048, ncu) 2970 -> 549 us, packing 78 us beside them; 16 prompts of
// 1024 tokens 124 -> 48 ms, eight documents through latent attention and routed experts 15.3 -> 7.7 ms.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "gemm_pair.cuh"
#include "linear.cuh"

namespace b200 {

constexpr int LU_BM = 128, LU_KS = 64;
constexpr int LU_EPI_WARPS = 8, LU_EPI_THREADS = LU_EPI_WARPS * 32, LU_THREADS = LU_EPI_THREADS + 64;
constexpr int LU_MAX_COUNTERS = 4096;

struct alignas(64) LinUmmaParams {
    CUtensorMap tw, tx;        // weights [groups * N][K], activations [rows of all groups][K]; boxes of 64 k
    LinParams l;
    int groups;
    int ksplit;                // parts of the k range (1: off; one group only)
    unsigned* counters;        // [tiles], zero between launches (ksplit > 1)
};

template <int TN, bool PAIR = false>
struct LuCfg {
    static constexpr int W_BYTES = LU_BM * LU_KS * 2, X_BYTES = (PAIR ? TN / 2 : TN) * LU_KS * 2;
    static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
    static constexpr int NSTAGE = 196608 / STAGE_BYTES > 8 ? 8 : 196608 / STAGE_BYTES;
    static constexpr int BAR_OFF = NSTAGE * STAGE_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + (2 * NSTAGE + 4) * 8 + 16 + 1024;       // + alignment of the ring
    static constexpr int TMEM_COLS = 2 * TN;                                            // 64 .. 512: double-buffered accumulator
};

// K-major operand in the 128-byte swizzle: 8-row atoms of 1024 bytes; a k16 step is 32 bytes further
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) { return umma_idesc_f16(M, N) | (1u << 7) | (1u << 10); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

// PAIR: counted on the barrier at a cluster address (the leader's)
__device__ __forceinline__ void tma2_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

__global__ void __launch_bounds__(256) lin_pack_kernel(const LinParams p, __nv_bfloat16* out) {
    pdl_launch_dependents();
    pdl_wait();
    const int g = blockIdx.y;
    const int rows = p.cnt[(size_t)g * p.cnt_gstride], K8 = p.K >> 3;
    const int base = p.off ? p.off[g] : 0;
    const float* X = p.X + g * p.x_gstride;
    __nv_bfloat16* const o = out + (size_t)(p.off ? base : g * p.max_rows) * p.K;
    const bool vec = (p.ldx % 4 == 0) && ((reinterpret_cast<uintptr_t>(X) & 15) == 0);
    for (int i = blockIdx.x * 256 + threadIdx.x; i < rows * K8; i += gridDim.x * 256) {
        const int r = i / K8, k = (i - r * K8) * 8;
        const float* src = X + (size_t)(p.xlist ? p.xlist[base + r] : base + r) * p.ldx + k;
        float v[8];
        lin_ld8(src, vec, 8, v);
        *reinterpret_cast<uint4*>(o + (size_t)r * p.K + k) =
            make_uint4(pack_bf16x2(make_float2(v[0], v[1])), pack_bf16x2(make_float2(v[2], v[3])), pack_bf16x2(make_float2(v[4], v[5])),
                       pack_bf16x2(make_float2(v[6], v[7])));
    }
}

// walks the units of a CTA: unit = ((group's tiles before it) ...) -> (group, output tile, row tile, k part), row tiles fastest so that
// CTAs that run side by side share a weight tile
template <int TN, bool PAIR>
struct LuWalk {
    const LinUmmaParams* p;
    int u, step, g, ubase, rows, ttiles, mtiles, per;
    __device__ __forceinline__ void load_group() {
        rows = p->l.cnt[(size_t)g * p->l.cnt_gstride];
        ttiles = (rows + TN - 1) / TN;
        per = ttiles * mtiles * p->ksplit;
    }
    __device__ __forceinline__ void init(const LinUmmaParams& p_) {
        p = &p_; u = PAIR ? (int)cluster_id_x() : (int)blockIdx.x; step = PAIR ? (int)ncluster_x() : (int)gridDim.x; g = 0; ubase = 0;
        mtiles = (p_.l.N + (PAIR ? 2 : 1) * LU_BM - 1) / ((PAIR ? 2 : 1) * LU_BM);
        load_group();
        settle();
    }
    __device__ __forceinline__ void settle() {
        while (g < p->groups && u - ubase >= per) {
            ubase += per;
            if (++g < p->groups) load_group();
        }
    }
    __device__ __forceinline__ bool done() const { return g >= p->groups; }
    __device__ __forceinline__ void next() { u += step; settle(); }
    __device__ __forceinline__ int tt() const { return (u - ubase) % ttiles; }
    __device__ __forceinline__ int mt() const { return ((u - ubase) / ttiles) % mtiles; }
    __device__ __forceinline__ int part() const { return (u - ubase) / (ttiles * mtiles); }
    // k slabs of this part
    __device__ __forceinline__ void slabs(int& s0, int& n) const {
        const int all = (p->l.K + LU_KS - 1) / LU_KS, q = (all + p->ksplit - 1) / p->ksplit;
        s0 = part() * q;
        n = min(all, s0 + q) - s0;
    }
};

template <int TN, bool PAIR>
__global__ void __launch_bounds__(LU_THREADS, 1) lin_umma_kernel(const __grid_constant__ LinUmmaParams p) {
    using Cfg = LuCfg<TN, PAIR>;
    extern __shared__ uint8_t lu_smem[];
    __shared__ int s_last;
    const uint32_t ring = (smem_u32(lu_smem) + 1023u) & ~1023u;
    const uint32_t full_bar = ring + Cfg::BAR_OFF, empty_bar = full_bar + Cfg::NSTAGE * 8;
    const uint32_t tfull_bar = empty_bar + Cfg::NSTAGE * 8, tempty_bar = tfull_bar + 16, tmem_slot = tempty_bar + 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = PAIR ? (int)cluster_rank() : 0;         // 0: the leader, which issues the MMAs of both
    if (tid == 0) {
        for (int s = 0; s < Cfg::NSTAGE; ++s) { mbar_init(full_bar + s * 8, 1); mbar_init(empty_bar + s * 8, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(tfull_bar + s * 8, 1); mbar_init(tempty_bar + s * 8, (PAIR ? 2 : 1) * LU_EPI_WARPS); }
        mbar_fence_init();
    }
    if (warp == LU_EPI_WARPS) {
        if constexpr (PAIR) tc_alloc2(tmem_slot, Cfg::TMEM_COLS);
        else tc_alloc(tmem_slot, Cfg::TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();                  // the peer's barriers exist before anything arrives there
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
    // only now: a dependent CTA that took its tensor memory first would wait for this grid while this grid waited for columns
    pdl_launch_dependents();
    pdl_wait();
    LuWalk<TN, PAIR> w;
    w.init(p);
    auto out_tile = [&]() { return PAIR ? 2 * w.mt() + rank : w.mt(); };      // 128 outputs of this CTA

    if (warp == LU_EPI_WARPS + 1) {
        if (lane == 0) {
            int stage = 0, done = 0;
            uint32_t ephase = 1;
            const uint32_t lead_full = PAIR ? mapa_u32(full_bar, 0) : 0;
            for (; !w.done(); w.next()) {
                int s0, n;
                w.slabs(s0, n);
                const int wrow = w.g * p.l.N + out_tile() * LU_BM, xrow = (p.l.off ? p.l.off[w.g] : w.g * p.l.max_rows) + w.tt() * TN + rank * (TN / 2);
                for (int i = 0; i < n; ++i, ++done) {
                    mbar_wait(empty_bar + stage * 8, ephase, 21);
                    const uint32_t st = ring + stage * Cfg::STAGE_BYTES, fb = full_bar + stage * 8;
                    if constexpr (PAIR) {
                        if (rank == 0) mbar_expect_tx(fb, 2 * Cfg::STAGE_BYTES);
                        tma2_load_2d(st, &p.tw, (s0 + i) * LU_KS, wrow, lead_full + stage * 8);
                        tma2_load_2d(st + Cfg::W_BYTES, &p.tx, (s0 + i) * LU_KS, xrow, lead_full + stage * 8);
                    } else {
                        mbar_expect_tx(fb, Cfg::STAGE_BYTES);
                        tma_load_2d(st, &p.tw, (s0 + i) * LU_KS, wrow, fb);
                        tma_load_2d(st + Cfg::W_BYTES, &p.tx, (s0 + i) * LU_KS, xrow, fb);
                    }
                    if (++stage == Cfg::NSTAGE) { stage = 0; ephase ^= 1; }
                }
            }
            // PAIR: every stage in use is released before this CTA may end: the leader's last commits arrive here
            for (int i = 0, n = PAIR ? min(done, Cfg::NSTAGE) : 0; i < n; ++i) {
                const int last = done - 1 - i;
                mbar_wait(empty_bar + (last % Cfg::NSTAGE) * 8, (uint32_t)(last / Cfg::NSTAGE) & 1u, 25);
            }
        }
    } else if (warp == LU_EPI_WARPS) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t IDESC = umma_idesc_bf16((PAIR ? 2 : 1) * LU_BM, TN);
            int stage = 0;
            uint32_t phase = 0;
            unsigned cnt = 0;
            for (; !w.done(); w.next(), ++cnt) {
                int s0, n;
                w.slabs(s0, n);
                const unsigned acc = cnt & 1u, use = cnt >> 1;
                if (use > 0) {
                    if constexpr (PAIR) mbar_wait_cluster(tempty_bar + acc * 8, (use - 1) & 1u, 22);
                    else mbar_wait(tempty_bar + acc * 8, (use - 1) & 1u, 22);
                }
                tc_fence_after();
                const uint32_t d = tmem_base + acc * TN;
                uint32_t accumulate = 0;
                for (int i = 0; i < n; ++i) {
                    if constexpr (PAIR) mbar_wait_cluster(full_bar + stage * 8, phase, 23);
                    else mbar_wait(full_bar + stage * 8, phase, 23);
                    tc_fence_after();
                    const uint32_t st = ring + stage * Cfg::STAGE_BYTES;
#pragma unroll
                    for (int k = 0; k < LU_KS / 16; ++k) {
                        if constexpr (PAIR) tc_mma2_f16(d, umma_desc_sw128(st + k * 32), umma_desc_sw128(st + Cfg::W_BYTES + k * 32), IDESC, accumulate);
                        else tc_mma_f16(d, umma_desc_sw128(st + k * 32), umma_desc_sw128(st + Cfg::W_BYTES + k * 32), IDESC, accumulate);
                        accumulate = 1;
                    }
                    if constexpr (PAIR) tc_commit2(empty_bar + stage * 8);
                    else tc_commit(empty_bar + stage * 8);
                    if (++stage == Cfg::NSTAGE) { stage = 0; phase ^= 1; }
                }
                if constexpr (PAIR) tc_commit2(tfull_bar + acc * 8);
                else tc_commit(tfull_bar + acc * 8);
            }
        }
    } else {
        const LinParams& l = p.l;
        const int grp = warp >> 2, row = tid & (LU_BM - 1);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t lead_tempty = PAIR ? mapa_u32(tempty_bar, 0) : 0;
        auto drained = [&](const unsigned acc) {                // this warp has read its part of the accumulator
            tc_fence_before();
            __syncwarp();
            if (lane != 0) return;
            if constexpr (PAIR) mbar_arrive_cluster(lead_tempty + acc * 8);
            else mbar_arrive(tempty_bar + acc * 8);
        };
        unsigned cnt = 0;
        for (; !w.done(); w.next(), ++cnt) {
            const unsigned acc = cnt & 1u, use = cnt >> 1;
            const int g = w.g, n = out_tile() * LU_BM + row, r0 = w.tt() * TN, nr = min(TN, w.rows - r0);
            const int yrow0 = (l.off ? l.off[g] : 0) + r0;
            const bool ok = n < l.N;
            const float bias = ok && l.bias && l.epi != LE_GLU_CLAMP && l.epi != LE_GLU_SILU ? l.bias[(size_t)g * l.N + n] : 0.f;
            if constexpr (PAIR) mbar_wait_cluster(tfull_bar + acc * 8, use & 1u, 24);
            else mbar_wait(tfull_bar + acc * 8, use & 1u, 24);
            tc_fence_after();
            const uint32_t tm = tmem_base + lane_base + acc * TN;
            const int tile = out_tile() * w.ttiles + w.tt();
            float* const ws = l.ws + (size_t)tile * p.ksplit * (LU_BM * TN) + row * 4;
            if (p.ksplit > 1) {
                float* const mine = ws + (size_t)w.part() * (LU_BM * TN);
#pragma unroll 1
                for (int c = grp * 16; c < nr; c += 32) {
                    float v[16];
                    tc_ld16(tm + c, v);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<float4*>(mine + (size_t)(c / 4 + j) * (LU_BM * 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                drained(acc);
                named_bar_sync(1, LU_EPI_THREADS);      // every thread's stores before thread 0's release
                if (tid == 0) {
                    const unsigned old = atom_add_acq_rel_gpu(p.counters + tile, 1u);
                    s_last = (old == (unsigned)(p.ksplit - 1));
                    if (s_last) p.counters[tile] = 0;
                }
                named_bar_sync(1, LU_EPI_THREADS);
                if (!*(volatile int*)&s_last) continue;
            }
            float* const Y = l.Y + g * l.y_gstride;
            const float* const gate = l.gate ? l.gate + (l.epi == LE_MUL_SIGMOID ? g * l.gate_gstride : 0) : nullptr;
            auto body = [&](auto epi_c) {
                constexpr int EPI = decltype(epi_c)::value;
                constexpr bool PAIRS = EPI == LE_GLU_CLAMP || EPI == LE_GLU_SILU || EPI == LE_SPLIT_GLU_RELU;
                constexpr bool GATE = EPI == LE_GATED_ADD || EPI == LE_MUL_SIGMOID, OLD = EPI == LE_GATED_ADD || EPI == LE_ADD;
#pragma unroll 1
                for (int c = grp * 16; c < nr; c += 32) {
                    float v[16], ga[16], old[16];
                    if (GATE || OLD) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const bool in = ok && c + j < nr;
                            if (GATE) ga[j] = in ? gate[(size_t)(yrow0 + c + j) * l.ldg + n] : 0.f;
                            if (OLD) old[j] = in ? Y[(size_t)(yrow0 + c + j) * l.ldy + n] : 0.f;
                        }
                    }
                    if (p.ksplit > 1) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = 0.f;
                        for (int s = 0; s < p.ksplit; ++s)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float4 q = __ldcg(reinterpret_cast<const float4*>(ws + (size_t)s * (LU_BM * TN) + (size_t)(c / 4 + j) * (LU_BM * 4)));
                                v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
                            }
                    } else {
                        tc_ld16(tm + c, v);
                    }
                    if constexpr (PAIRS) {
                        // lanes (2 i, 2 i + 1) = (gate, up); N and split are even.  Of two neighbouring rows the even lane finishes the first, the odd lane
                        // the second: one exchange and one gated unit a lane for two rows (a gated unit of every row in the even lanes alone took
                        // 28 us a unit of 256 outputs x 256 rows where its MMAs take 13)
                        const int odd = lane & 1;
                        const bool glu = EPI != LE_SPLIT_GLU_RELU || n >= l.split;
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const float x = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
                            const float ga_ = odd ? x : v[j], up = odd ? v[j + 1] : x;
                            if (EPI == LE_SPLIT_GLU_RELU && !glu) {
#pragma unroll
                                for (int q = 0; q < 2; ++q)
                                    if (ok && c + j + q < nr) Y[(size_t)(yrow0 + c + j + q) * l.ldy + n] = v[j + q] + bias;
                                continue;
                            }
                            const int r = c + j + odd;
                            if (!ok || r >= nr) continue;
                            if constexpr (EPI == LE_SPLIT_GLU_RELU) {
                                l.Y2[(size_t)(yrow0 + r) * l.ldy2 + ((n - l.split) >> 1)] = fmaxf(ga_, 0.f) * up;
                            } else {
                                const float y = EPI == LE_GLU_CLAMP ? lin_glu(ga_, up, l.limit) : ga_ * lin_sigmoid(ga_) * up;
                                if (l.Y16) l.Y16[(size_t)(yrow0 + r) * l.ldy + (n >> 1)] = __float2bfloat16(y);
                                else Y[(size_t)(yrow0 + r) * l.ldy + (n >> 1)] = y;
                            }
                        }
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const bool in = ok && c + j < nr;
                        float* const yr = Y + (size_t)(yrow0 + c + j) * l.ldy;
                        if (in) {
                            const float a = v[j] + bias;
                            float y = a;
                            if constexpr (EPI == LE_SIGMOID) y = lin_sigmoid(a);
                            else if constexpr (EPI == LE_GELU_ERF) y = 0.5f * a * (1.f + erff(a * 0.70710678118654752f));
                            else if constexpr (EPI == LE_RELU_SQ) { const float r = fmaxf(a, 0.f); y = r * r; }
                            else if constexpr (EPI == LE_GATED_ADD) y = old[j] + ga[j] * a;
                            else if constexpr (EPI == LE_ADD) y = fmaf(l.limit, a, old[j]);
                            else if constexpr (EPI == LE_MUL_SIGMOID) y = a * lin_sigmoid(ga[j]);
                            else if constexpr (EPI == LE_TANH_CAP) y = l.limit * tanhf(a / l.limit);
                            yr[n] = y;
                        }
                    }
                }
            };
            switch (l.epi) {
                case LE_SIGMOID: body(std::integral_constant<int, LE_SIGMOID>{}); break;
                case LE_GATED_ADD: body(std::integral_constant<int, LE_GATED_ADD>{}); break;
                case LE_GLU_CLAMP: body(std::integral_constant<int, LE_GLU_CLAMP>{}); break;
                case LE_GLU_SILU: body(std::integral_constant<int, LE_GLU_SILU>{}); break;
                case LE_GELU_ERF: body(std::integral_constant<int, LE_GELU_ERF>{}); break;
                case LE_RELU_SQ: body(std::integral_constant<int, LE_RELU_SQ>{}); break;
                case LE_ADD: body(std::integral_constant<int, LE_ADD>{}); break;
                case LE_MUL_SIGMOID: body(std::integral_constant<int, LE_MUL_SIGMOID>{}); break;
                case LE_TANH_CAP: body(std::integral_constant<int, LE_TANH_CAP>{}); break;
                case LE_SPLIT_GLU_RELU: body(std::integral_constant<int, LE_SPLIT_GLU_RELU>{}); break;
                default: body(std::integral_constant<int, LE_STORE>{}); break;
            }
            if (p.ksplit == 1) drained(acc);
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) {
        cluster_sync_all();                                  // no CTA leaves while its peer's MMAs read its shared memory or arrive on its barriers
        tc_fence_after();
        if (warp == LU_EPI_WARPS) tc_dealloc2(tmem_base, Cfg::TMEM_COLS);
    } else if (warp == LU_EPI_WARPS) {
        tc_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

}  // namespace b200
