// Projection GEMM of steps of more than 64 tokens (one GPU, f16 weights):  Y[T, N] = X[T, K] (f16) * W[N, K]^T (f16), f32 accumulate, on pairs of SMs.
//
// Same weight blocks, segments and epilogues as gemm.cuh / gemm_wide.cuh; replaces the projection dispatches of `Runtime::infer` (reference
// crates/ai00-core/src/run.rs:1143) in steps that hold long prompts.
//
// What bounds it: the bytes an SM takes in.  One SM that multiplies 128 weight rows by 256 tokens reads 48 KB per 64 k (and its tensor core reads
// them again from shared memory); two SMs that share one 256 x 256 tile (tcgen05 cta_group::2) read 32 KB each for the same work.
//   * a cluster of two CTAs owns a unit = 256 weight rows x NTOK tokens: each CTA keeps its 128 rows of weights, half of the tokens and the
//     accumulators of its 128 rows; one thread of the leader issues every MMA of both;
//   * both operands lie in memory in the order the tensor core reads them, so a stage of 64 k is one box of plain 1 KB rows per operand: tiled TMA
//     (not the untiled copy) because its arrival may be counted on the leader's barrier;
//   * steps hold up to 2048 tokens, the units of a launch (token tiles fastest, so that neighbours share weights) are dealt to persistent clusters;
//   * NTOK = 256, or 128 where the launch would leave more of its last wave empty with 256 than the narrower tile costs (pair_plan in engine.cu);
//   * eight epilogue warps drain one accumulator while the next unit's MMAs run; f16 operands are transposed warp by warp.
// Measured (3B widths, 1792 tokens a launch against seven launches of 256 tokens on single SMs, ncu): R/K/V/G 253 -> 83 us (1.13 PFLOP/s), output 132 -> 27,
// channel mix 307 -> 96 and 171 -> 61, first low-rank stage 225 -> 23; 32 prompts of 512 tokens 53.5 -> 21.5 ms.
// 100 tokens of 7B widths (weights from HBM): 42 -> 34, 18 -> 18, 45 -> 37 and 32 -> 29 us.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "gemm.cuh"

namespace b200 {

constexpr int PAIR_EPI_WARPS = 8, PAIR_EPI_THREADS = PAIR_EPI_WARPS * 32;
constexpr int PAIR_THREADS = PAIR_EPI_THREADS + 64;         // + MMA warp + TMA producer warp
constexpr int PAIR_PITCH = 40;                              // halves per row of a warp's transpose buffer (32 tokens + padding)

struct alignas(64) PairParams {
    CUtensorMap tw, ta;         // weight blocks as rows of 1 KB; the token operands as [2 KB rows][2 halves of 1 KB]
    GemmParams g;
    int a_row[GEMM_MAX_SEG];    // first 2 KB row of a segment's token operand
    int a_tile[GEMM_MAX_SEG];   // k blocks between its 256-token tiles
    // segments that continue one another's k range form one chain: units are (chain, pair of 128-row tiles, token tile)
    int nchain;
    int first[GEMM_MAX_SEG + 1];        // first segment of a chain
    int pair_begin[GEMM_MAX_SEG + 1];   // pairs of tiles before it
    int ttiles;                 // token tiles of the step
};

template <int NTOK>
struct PairCfg {
    static constexpr int W_BYTES = GEMM_BN * 64 * 2;        // 16 KB: this CTA's 128 weight rows x 64 k
    static constexpr int A_BYTES = NTOK / 2 * 64 * 2;       // its half of the tokens
    static constexpr int STAGE_BYTES = W_BYTES + A_BYTES;
    static constexpr int NSTAGE = NTOK == 256 ? 6 : 8;
    static constexpr int OUT_OFF = NSTAGE * STAGE_BYTES;
    static constexpr int OUT_BYTES = PAIR_EPI_WARPS * 32 * PAIR_PITCH * 2;
    static constexpr int BAR_OFF = OUT_OFF + OUT_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + (2 * NSTAGE + 4) * 8 + 16 + 128;    // + alignment of the ring
    static constexpr int TMEM_COLS = 2 * NTOK;              // two accumulators
    static_assert(SMEM_BYTES <= 227 * 1024 - 1024, "one CTA per SM");
};

// ---- two-CTA forms of the helpers in common.cuh ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t ncluster_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_wait_cluster(uint32_t bar, uint32_t parity, unsigned tag) {
    if (mbar_try_cluster(bar, parity)) return;
    SpinGuard g;
    while (!mbar_try_cluster(bar, parity)) g.poll(WD_MBAR, bar, parity, tag);
}
__device__ __forceinline__ void tc_alloc2(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_mma2_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void tc_commit2(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}
// tiled loads into this CTA's shared memory, counted on the (leader's) barrier
__device__ __forceinline__ void tma2_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar), "l"(pol)
        : "memory");
}
__device__ __forceinline__ void tma2_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(pol)
        : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// the units of a cluster, token tiles fastest
struct PairWalk {
    const PairParams* p;
    int u, step, total, chain, wp, tt;
    __device__ __forceinline__ void init(const PairParams& p_) {
        p = &p_;
        u = (int)cluster_id_x();
        step = (int)ncluster_x();
        total = p_.pair_begin[p_.nchain] * p_.ttiles;
        chain = 0;
        settle();
    }
    __device__ __forceinline__ bool done() const { return u >= total; }
    __device__ __forceinline__ void settle() {
        if (done()) return;
        const int w = u / p->ttiles;
        tt = u - w * p->ttiles;
        while (w >= p->pair_begin[chain + 1]) ++chain;
        wp = w - p->pair_begin[chain];
    }
    __device__ __forceinline__ void next() { u += step; settle(); }
    __device__ __forceinline__ int stages() const {
        int n = 0;
        for (int s = p->first[chain]; s < p->first[chain + 1]; ++s) n += 2 * p->g.seg[s].KB;
        return n;
    }
};

template <int NTOK>
__global__ void __launch_bounds__(PAIR_THREADS, 1) gemm_pair_kernel(const __grid_constant__ PairParams p) {
    using Cfg = PairCfg<NTOK>;
    extern __shared__ uint8_t pair_smem[];
    const uint32_t ring = (smem_u32(pair_smem) + 127u) & ~127u;
    uint8_t* const ring_p = pair_smem + (ring - smem_u32(pair_smem));
    const uint32_t full_bar = ring + Cfg::BAR_OFF, empty_bar = full_bar + Cfg::NSTAGE * 8;
    const uint32_t tfull_bar = empty_bar + Cfg::NSTAGE * 8, tempty_bar = tfull_bar + 16, tmem_slot = tempty_bar + 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    if (tid == 0) {
        trace_stamp(p.g.trace, 0);
        for (int s = 0; s < Cfg::NSTAGE; ++s) { mbar_init(full_bar + s * 8, 1); mbar_init(empty_bar + s * 8, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(tfull_bar + s * 8, 1); mbar_init(tempty_bar + s * 8, 2 * PAIR_EPI_WARPS); }
        mbar_fence_init();
    }
    if (warp == PAIR_EPI_WARPS) tc_alloc2(tmem_slot, Cfg::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                     // the peer's barriers exist before anything arrives there
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(ring_p + (tmem_slot - ring));
    pdl_launch_dependents();                                // behind the allocation: see linear_umma.cuh
    PairWalk w;
    w.init(p);

    if (warp == PAIR_EPI_WARPS + 1) {
        // ===================== producer: one lane of each CTA =====================
        if (lane == 0) {
            const uint64_t pol_w = l2_policy_evict_first(), pol_a = l2_policy_evict_last();
            const uint32_t lead_full = mapa_u32(full_bar, 0);
            auto load_w = [&](const int stage, const int row) { tma2_load_2d(ring + stage * Cfg::STAGE_BYTES, &p.tw, 0, row, lead_full + stage * 8, pol_w); };
            auto load_a = [&](const int stage, const int tt, const int row) {
                const uint32_t dst = ring + stage * Cfg::STAGE_BYTES + Cfg::W_BYTES;
                if (NTOK == 256) tma2_load_3d(dst, &p.ta, 0, 0, row + (int)rank * 16, lead_full + stage * 8, pol_a);
                else tma2_load_3d(dst, &p.ta, 0, (int)rank, row + (tt & 1) * 16, lead_full + stage * 8, pol_a);
            };
            // weights of the first stages never change: requested before the wait
            int npre = 0;
            if (!w.done()) {
                const GemmSeg& sg = p.g.seg[p.first[w.chain]];
                npre = min(2 * sg.KB, Cfg::NSTAGE);
                const int row = (sg.blk_begin + min(2 * w.wp + (int)rank, sg.tiles - 1) * sg.KB) * 32;
                for (int i = 0; i < npre; ++i) {
                    if (rank == 0) mbar_expect_tx(full_bar + i * 8, 2 * Cfg::STAGE_BYTES);
                    load_w(i, row + i * 16);
                }
            }
            pdl_wait();
            if (p.g.trace && blockIdx.x == 0) p.g.trace[2] = globaltimer_ns();
            int stage = 0, done = 0;
            uint32_t ephase = 1;
            for (; !w.done(); w.next()) {
                for (int s = p.first[w.chain]; s < p.first[w.chain + 1]; ++s) {
                    const GemmSeg& sg = p.g.seg[s];
                    const int wrow = (sg.blk_begin + min(2 * w.wp + (int)rank, sg.tiles - 1) * sg.KB) * 32;
                    const int arow = p.a_row[s] + (NTOK == 256 ? w.tt : w.tt >> 1) * p.a_tile[s] * 32;
                    for (int i = 0; i < 2 * sg.KB; ++i, ++done) {
                        if (done >= npre) {
                            mbar_wait(empty_bar + stage * 8, ephase, 31);
                            if (rank == 0) mbar_expect_tx(full_bar + stage * 8, 2 * Cfg::STAGE_BYTES);
                            load_w(stage, wrow + i * 16);
                        }
                        load_a(stage, w.tt, arow + (i >> 1) * 32 + (i & 1) * 8);
                        if (++stage == Cfg::NSTAGE) { stage = 0; ephase ^= 1; }
                    }
                }
            }
            // every stage in use is released before this CTA may end: the leader's last commits arrive here
            for (int i = 0, n = min(done, Cfg::NSTAGE); i < n; ++i) {
                const int last = done - 1 - i;
                mbar_wait(empty_bar + (last % Cfg::NSTAGE) * 8, (uint32_t)(last / Cfg::NSTAGE) & 1u, 32);
            }
        }
    } else if (warp == PAIR_EPI_WARPS) {
        // ===================== MMA issuer: one lane of the leader =====================
        if (lane == 0 && rank == 0) {
            constexpr uint32_t IDESC = umma_idesc_f16(2 * GEMM_BN, NTOK);
            constexpr uint32_t A_LBO = NTOK / 2 * 16;       // bytes between the k8 chunks of this CTA's tokens
            int stage = 0;
            uint32_t phase = 0;
            unsigned cnt = 0;
            for (; !w.done(); w.next(), ++cnt) {
                const int n = w.stages();
                const unsigned acc = cnt & 1u, use = cnt >> 1;
                if (use > 0) mbar_wait_cluster(tempty_bar + acc * 8, (use - 1) & 1u, 33);
                tc_fence_after();
                const uint32_t d = tmem_base + acc * NTOK;
                uint32_t accumulate = 0;
                for (int i = 0; i < n; ++i) {
                    mbar_wait_cluster(full_bar + stage * 8, phase, 34);
                    tc_fence_after();
                    const uint32_t st = ring + stage * Cfg::STAGE_BYTES;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        tc_mma2_f16(d, umma_desc(st + k * 2 * GEMM_W_LBO, GEMM_W_LBO, GEMM_W_SBO), umma_desc(st + Cfg::W_BYTES + k * 2 * A_LBO, A_LBO, GEMM_A_SBO), IDESC,
                                    accumulate);
                        accumulate = 1;
                    }
                    tc_commit2(empty_bar + stage * 8);
                    if (++stage == Cfg::NSTAGE) { stage = 0; phase ^= 1; }
                }
                tc_commit2(tfull_bar + acc * 8);
            }
            if (p.g.trace) {
                unsigned smid;
                asm volatile("mov.u32 %0, %smid;" : "=r"(smid));
                trace_cta(p.g.trace, 0, smid);
                trace_cta(p.g.trace, 1, globaltimer_ns());
            }
        }
    } else {
        // ===================== epilogue: lane = weight row, warps 0-3 the first half of the tokens, 4-7 the second =====================
        pdl_wait();
        if (tid == 0) trace_stamp(p.g.trace, 5);
        const int nrows = *p.g.nrows;
        const int half = warp >> 2, row = tid & (GEMM_BN - 1);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16, lead_tempty = mapa_u32(tempty_bar, 0);
        __half* const buf = reinterpret_cast<__half*>(ring_p + Cfg::OUT_OFF) + warp * 32 * PAIR_PITCH;
        unsigned cnt = 0;
        for (; !w.done(); w.next(), ++cnt) {
            const GemmSeg& sg = p.g.seg[p.first[w.chain]];
            const unsigned acc = cnt & 1u, use = cnt >> 1;
            const int tile = 2 * w.wp + (int)rank, n = tile * GEMM_BN + row, m0 = w.tt * NTOK + half * (NTOK / 2);
            const int live = tile < sg.tiles ? min(NTOK / 2, nrows - m0) : 0;        // tokens of this warp (an odd last tile has no partner)
            const bool row_ok = n < sg.N;
            const int out_mode = sg.out_mode, ldo = sg.ldo;
            const float bias = (row_ok && live > 0 && sg.bias) ? sg.bias[n] : 0.f;
            const bool lerp = out_mode == OUT_LERP_A16;
            const float mu = (lerp && row_ok && live > 0) ? sg.aux2[n] : 0.f;
            mbar_wait_cluster(tfull_bar + acc * 8, use & 1u, 35);
            tc_fence_after();
            const uint32_t tm = tmem_base + lane_base + acc * NTOK + half * (NTOK / 2);
            auto body = [&](auto act_c) {
                constexpr int ACT_C = decltype(act_c)::value;
#pragma unroll 1
                for (int c = 0; c < live; c += 32) {
                    float v[32];
                    tc_ld32(tm + c, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j] + bias, ACT_C);
                    if (out_mode == OUT_F32) {
                        if (row_ok) {
                            float* const o = reinterpret_cast<float*>(sg.out) + (size_t)(m0 + c) * ldo + n;
                            if (c + 32 <= live) {
#pragma unroll
                                for (int j = 0; j < 32; ++j) o[(size_t)j * ldo] = v[j];
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; ++j)
                                    if (c + j < live) o[(size_t)j * ldo] = v[j];
                            }
                        }
                        continue;
                    }
                    if (ACT_C == ACT_NONE && lerp) {        // low ranks beyond one k block (one-block ones: lora2.cuh, gemm_wide.cuh)
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const bool ok = row_ok && c + j < live;
                            const size_t a_ = (size_t)(m0 + c + j) * sg.ld_aux + n;
                            const float xx = ok ? sg.aux0[a_] : 0.f, sx = ok ? sg.aux1[a_] : 0.f;
                            v[j] = xx + sx * (mu + v[j]);
                        }
                    }
                    // 16-byte chunks of eight rows: the rows of a chunk are lanes of this warp
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint4 h = make_uint4(pack_h2(v[8 * q], v[8 * q + 1]), pack_h2(v[8 * q + 2], v[8 * q + 3]), pack_h2(v[8 * q + 4], v[8 * q + 5]), pack_h2(v[8 * q + 6], v[8 * q + 7]));
                        if (!row_ok) h = make_uint4(0, 0, 0, 0);
                        *reinterpret_cast<uint4*>(buf + lane * PAIR_PITCH + 8 * q) = h;
                    }
                    __syncwarp();
                    const int row0 = tile * GEMM_BN + (warp & 3) * 32;
                    if (c + lane < live) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int nc = row0 + q * 8;
                            if (nc >= sg.N) break;
                            const __half* src = buf + q * 8 * PAIR_PITCH + lane;
                            uint32_t r[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                r[k] = (uint32_t)__half_as_ushort(src[2 * k * PAIR_PITCH]) | ((uint32_t)__half_as_ushort(src[(2 * k + 1) * PAIR_PITCH]) << 16);
                            __half* base = reinterpret_cast<__half*>(sg.out);
                            int nn = nc;
                            if (sg.grp > 0) {
                                const int gi = nc / sg.grp;
                                base += (size_t)gi * sg.grp_stride;
                                nn = nc - gi * sg.grp;
                            }
                            *reinterpret_cast<uint4*>(base + a16_index(m0 + c + lane, nn, ldo)) = make_uint4(r[0], r[1], r[2], r[3]);
                        }
                    }
                    __syncwarp();
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
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead_tempty + acc * 8);
        }
        if (tid == 0) trace_stamp(p.g.trace, 6);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        trace_stamp(p.g.trace, 7);
        if (p.g.trace) trace_cta(p.g.trace, 2, globaltimer_ns());
    }
    cluster_sync_all();                                     // no CTA leaves while its peer's MMAs read its shared memory or arrive on its barriers
    tc_fence_after();
    if (warp == PAIR_EPI_WARPS) tc_dealloc2(tmem_base, Cfg::TMEM_COLS);
}

}  // namespace b200
