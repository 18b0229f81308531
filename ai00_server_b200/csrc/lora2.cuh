// Second stages of RWKV-6's low-rank pairs in prompt steps (more than 16 tokens): the five token-shift lerps
//     mixed_j[t, c] = xx[t, c] + sx[t, c] * (mu_j[c] + sum_k W2_j[c, k] tanh(W1 xxx)_j[t, k])     -> f16 operands of R / K / V / G and the decay
// and the decays  w[t, c] = exp(-exp(bias[c] + sum_k Wd2[c, k] tanh(Wd1 xw)[t, k]))               -> f32
// (reference crates/ai00-core/src/run.rs:1143, web-rwkv's time_mix_w2 / time_decay_w2 products.)
//
// What bounds it: bytes -- two f32 rows in, five f16 rows out for 10 Dm multiply-adds an element.  As projection launches (one-block tiles) every one
// of the five groups read the two rows again and multiplied 128-wide k blocks of which Dm are not padding.  Here a CTA of eight warps takes 128 tokens
// and 64 columns (16 where a step has one tile of tokens and most SMs would idle), keeps its slice of the five matrices in shared memory and the low-rank
// operands of a warp's 16 tokens in registers, and reads xx and sx once; the products are 16 x 8 x 16 mma.sync steps, whose accumulator fragments are
// 16-byte rows of the A16 layout (8 tokens = 128 contiguous bytes).
// Measured (ncu): 1792 tokens of 3B widths 76 -> 41 us (lerps), 18 -> 11 (decays); 100 tokens of 7B widths 15 -> 10 and 14 -> 6.
#pragma once
#include "gemm.cuh"

namespace b200 {

constexpr int LORA2_THREADS = 256, LORA2_TOK = 128, LORA2_COLS = 64;       // columns a CTA takes in steps of several tiles; C is a multiple
constexpr int LORA2_FEW_COLS = 16;                                          // in steps of one tile

struct Lora2Params {
    const __half* w;              // [groups][C][K] row-major
    const __half* low;            // A16, `groups` matrices
    int low_stride;               // halves between them
    int low_th;                   // token rows and tile distance of the operand (common.cuh)
    int C;
    const float* xx;              // ddlerp: [T, C]
    const float* sx;
    const float* mu[5];
    __half* out[5];               // A16
    int out_th;
    const float* bias;            // decay
    float* decay;                 // [T, C]
    MetaView meta;
};

template <int K16, int GROUPS, int COLS>
constexpr size_t lora2_smem() { return (size_t)GROUPS * COLS * (K16 * 16 + 8) * 2; }

// GROUPS = 5: the lerps; 1: the decay
template <int K16, int GROUPS, int COLS>
__global__ void __launch_bounds__(LORA2_THREADS) lora2_kernel(const __grid_constant__ Lora2Params p) {
    constexpr int K = K16 * 16, PITCH = K + 8;              // halves per row of the slice: eight rows of a fragment in different banks
    extern __shared__ __align__(16) __half lora2_w[];       // [GROUPS][COLS][PITCH]
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, tig = lane & 3;
    const int n0 = blockIdx.x * COLS, m0 = blockIdx.y * LORA2_TOK + warp * 16;
    for (int i = tid; i < GROUPS * COLS * (K / 8); i += LORA2_THREADS) {      // weights never change: before the wait
        const int j = i / (COLS * (K / 8)), rem = i - j * (COLS * (K / 8)), r = rem / (K / 8), q = rem - r * (K / 8);
        *reinterpret_cast<uint4*>(lora2_w + ((size_t)j * COLS + r) * PITCH + q * 8) = *reinterpret_cast<const uint4*>(p.w + ((size_t)j * p.C + n0 + r) * K + q * 8);
    }
    pdl_wait();
    __syncthreads();
    const int T = p.meta.T();
    if (m0 >= T) return;
    // low-rank operands of this warp's 16 tokens (rows beyond the step hold whatever an earlier one left and are not stored)
    uint32_t a[GROUPS][K16][4];
#pragma unroll
    for (int j = 0; j < GROUPS; ++j)
#pragma unroll
        for (int k = 0; k < K16; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                a[j][k][q] = *reinterpret_cast<const uint32_t*>(p.low + (size_t)j * p.low_stride + a16_index(m0 + grp + (q & 1) * 8, k * 16 + tig * 2 + (q >> 1) * 8, p.low_th));
    float2 xn[2], sn[2];                                    // the next eight columns' rows, requested while this one's products run
    auto request = [&](const int nt) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + grp + 8 * h, n = n0 + nt * 8 + tig * 2;
            const bool ok = GROUPS == 5 && m < T && nt < COLS / 8;
            xn[h] = ok ? *reinterpret_cast<const float2*>(p.xx + (size_t)m * p.C + n) : make_float2(0.f, 0.f);
            sn[h] = ok ? *reinterpret_cast<const float2*>(p.sx + (size_t)m * p.C + n) : make_float2(0.f, 0.f);
        }
    };
    request(0);
#pragma unroll 2
    for (int nt = 0; nt < COLS / 8; ++nt) {
        const int n = n0 + nt * 8 + tig * 2;
        const float2 x[2] = {xn[0], xn[1]}, s[2] = {sn[0], sn[1]};
        request(nt + 1);
#pragma unroll
        for (int j = 0; j < GROUPS; ++j) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            const __half* wr = lora2_w + ((size_t)j * COLS + nt * 8 + grp) * PITCH + tig * 2;
#pragma unroll
            for (int k = 0; k < K16; ++k)
                mma_16816(c, a[j][k][0], a[j][k][1], a[j][k][2], a[j][k][3], *reinterpret_cast<const uint32_t*>(wr + k * 16),
                          *reinterpret_cast<const uint32_t*>(wr + k * 16 + 8));
            const float2 b = *reinterpret_cast<const float2*>((GROUPS == 5 ? p.mu[j] : p.bias) + n);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m0 + grp + 8 * h;
                if (m >= T) continue;
                if constexpr (GROUPS == 5)
                    *reinterpret_cast<uint32_t*>(p.out[j] + a16_index(m, n, p.out_th)) = pack_h2(x[h].x + s[h].x * (b.x + c[2 * h]), x[h].y + s[h].y * (b.y + c[2 * h + 1]));
                else
                    *reinterpret_cast<float2*>(p.decay + (size_t)m * p.C + n) =
                        make_float2(apply_act(c[2 * h] + b.x, ACT_EXPNEGEXP), apply_act(c[2 * h + 1] + b.y, ACT_EXPNEGEXP));
            }
        }
    }
}

}  // namespace b200
