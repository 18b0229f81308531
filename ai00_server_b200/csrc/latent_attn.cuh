// Latent ("compressed key/value") attention over a paged cache, in the absorbed form.
//
// A layer caches, per token, one latent row c [rk] (RMS-normed down-projection) and one rotated key part kr [dr] shared by
// all heads: D = rk + dr floats per token and layer.  Per head the key is [W_uk c ; kr] and the value W_uv c, so with
//     qa[h] = W_uk[h]^T q_plain[h]   (rk numbers)           -- a grouped linear over heads, W_uk stored transposed at load
// the score is (qa[h] . c_j + q_rot[h] . kr_j) * scale and the head's output is W_uv[h] (sum_j p_j c_j): the attention itself
// runs over the shared rows [c_j ; kr_j] for all heads (no per-head keys or values are ever materialised), and the two
// up-projections are grouped linears before and after it.  Scores, softmax and the weighted sums are f32.
//
// Paging: the cache of every layer is a pool of pages of `page` tokens; page_table[slot][i] names the page that holds the
// sequence's positions [i * page, (i + 1) * page).  Pages are handed out and taken back by the host (engine state manager);
// a step uploads the table entries it added (page_update_kernel).  A layer that borrows another layer's cache reads that
// layer's pool with the same table.
//
//   rope_rows_kernel     rotate-half rotary embedding on `dims` leading entries of a per-head chunk (positions and angles f32;
//                        frequency table with the long-context rescaling folded in at load, magnitude factor on cos and sin)
//   kv_write_kernel      c = rms(kv[:rk]) * w, kr = rope(kv[rk:]) -> cache row of (slot, position)
//   latent_attn_kernel   QB consecutive tokens of one sequence x HG heads per CTA share every key tile; online softmax; the
//                        context may be split over blockIdx.z (long contexts at small batch), partial (o, m, l) per split
//   latent_merge_kernel  combines the splits in fixed order and normalises
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include "common.cuh"

namespace b200 {

// per-step sequence metadata that follows the MetaView block in the same upload
struct SeqMeta {
    const int* base;
    int maxT;
    __host__ __device__ int n_upd() const { return base[0]; }
    __host__ __device__ int n_chunks() const { return base[1]; }
    __host__ __device__ const int* tok_pos() const { return base + 8; }                     // [maxT] position of the token in its sequence
    __host__ __device__ const int* chunk_start() const { return base + 8 + maxT; }          // [maxT] first token of an attention chunk
    __host__ __device__ const int* chunk_count() const { return base + 8 + 2 * maxT; }      // [maxT] tokens of the chunk (one sequence)
    __host__ __device__ const int* upd() const { return base + 8 + 3 * maxT; }              // [maxT][3] (slot, index, page)
    __host__ __device__ static size_t ints(int maxT) { return 8 + 6 * (size_t)maxT; }
};

// The run-th run of at most qt tokens of one sequence, counted through the step's sequences, found by one warp: out = (sequence of the step or -1, run within it)
__device__ __forceinline__ void step_token_run(const MetaView& meta, const int qt, const int run, int* out) {
    const int lane = threadIdx.x & 31, nslots = meta.nslots();
    int left = run, found = -1;
    for (int s0 = 0; s0 < nslots && found < 0; s0 += 32) {
        const int s = s0 + lane, n = s < nslots ? (meta.slot_count()[s] + qt - 1) / qt : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, left < upto);
        if (hit) {
            const int l = __ffs(hit) - 1;
            left -= __shfl_sync(0xffffffffu, upto - n, l);
            found = s0 + l;
        } else {
            left -= __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (lane == 0) { out[0] = found; out[1] = left; }
}

// the same counted from the last run (later tokens have more keys: they start first); launches have CTAs for more runs than there are, and those come last
__device__ __forceinline__ void step_token_run_back(const MetaView& meta, const int qt, const int back, int* out) {
    const int lane = threadIdx.x & 31, nslots = meta.nslots();
    int total = 0;
    for (int s = lane; s < nslots; s += 32) total += (meta.slot_count()[s] + qt - 1) / qt;
    const int run = __reduce_add_sync(0xffffffffu, total) - 1 - back;
    if (run >= 0) step_token_run(meta, qt, run, out);
    else if (lane == 0) out[0] = -1;
}

struct PageUpdateParams { SeqMeta sm; int* table; int stride; };

__global__ void page_update_kernel(const PageUpdateParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int n = p.sm.n_upd();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int* u = p.sm.upd() + 3 * i;
        p.table[(size_t)u[0] * p.stride + u[1]] = u[2];
    }
}

struct RopeParams {
    const float* src; int lds, s_head, s_off;      // element (t, h, i) at src[t * lds + h * s_head + s_off + i]
    float* dst; int ldd, d_head, d_off;
    int heads, dims, width;                        // rotate the first `dims` of `width` entries; the rest are copied
    const float* freq;                             // [dims / 2]
    float mag;
    MetaView meta; SeqMeta sm;
    const double* pair_freq = nullptr;             // set: neighbouring entries (2i, 2i + 1) turn together (angle reduced in double)
};

// the pair (2i, 2i + 1) of `s` turned by position * freq[i]; returns entry i of the result
__device__ __forceinline__ float rot_pair_entry(const float* s, int i, int pos, const double* freq) {
    float cs, sn;
    rot_cos_sin(pos, freq[i >> 1], cs, sn);
    const float u = s[i & ~1], v = s[i | 1];
    return (i & 1) ? v * cs + u * sn : u * cs - v * sn;
}

__global__ void __launch_bounds__(128) rope_rows_kernel(const RopeParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    const float pos = (float)p.sm.tok_pos()[t];
    const int half = p.dims >> 1;
    for (int e = threadIdx.x; e < p.heads * p.width; e += blockDim.x) {
        const int h = e / p.width, i = e % p.width;
        const float* s = p.src + (size_t)t * p.lds + (size_t)h * p.s_head + p.s_off;
        float* d = p.dst + (size_t)t * p.ldd + (size_t)h * p.d_head + p.d_off;
        if (i >= p.dims) { d[i] = s[i]; continue; }
        if (p.pair_freq) { d[i] = rot_pair_entry(s, i, p.sm.tok_pos()[t], p.pair_freq); continue; }
        const int j = i < half ? i : i - half;
        const float a = pos * p.freq[j];
        const float cs = cosf(a) * p.mag, sn = sinf(a) * p.mag;
        const float u = s[j], v = s[j + half];
        d[i] = i < half ? u * cs - v * sn : v * cs + u * sn;
    }
}

struct KvWriteParams {
    const float* kv; int ld;                       // [T, rk + dr] down-projection rows
    float* cache;                                  // pool of this layer: [pages][page][D]
    const int* table; int stride; int page;
    const float* weight;                           // [rk]
    int rk, dr, dims;
    const float* freq; float mag, eps;
    MetaView meta; SeqMeta sm;
    const double* pair_freq = nullptr;             // as in RopeParams
};

__global__ void __launch_bounds__(128) kv_write_kernel(const KvWriteParams p) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[32];
    const int t = blockIdx.x;
    if (t >= p.meta.T()) return;
    const int slot = p.meta.tok_slot()[t], ipos = p.sm.tok_pos()[t];
    const float* src = p.kv + (size_t)t * p.ld;
    const int D = p.rk + p.dr;
    float* dst = p.cache + ((size_t)p.table[(size_t)slot * p.stride + ipos / p.page] * p.page + ipos % p.page) * D;
    float ss = 0.f;
    for (int i = threadIdx.x; i < p.rk; i += blockDim.x) ss = fmaf(src[i], src[i], ss);
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        ss = 0.f;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) ss += red[i];
    }
    const float r = 1.f / sqrtf(ss / (float)p.rk + p.eps);
    for (int i = threadIdx.x; i < p.rk; i += blockDim.x) dst[i] = src[i] * r * p.weight[i];
    const float pos = (float)ipos;
    const int half = p.dims >> 1;
    for (int i = threadIdx.x; i < p.dr; i += blockDim.x) {
        const float* s = src + p.rk;
        if (i >= p.dims) { dst[p.rk + i] = s[i]; continue; }
        if (p.pair_freq) { dst[p.rk + i] = rot_pair_entry(s, i, ipos, p.pair_freq); continue; }
        const int j = i < half ? i : i - half;
        const float a = pos * p.freq[j];
        const float cs = cosf(a) * p.mag, sn = sinf(a) * p.mag;
        const float u = s[j], v = s[j + half];
        dst[p.rk + i] = i < half ? u * cs - v * sn : v * cs + u * sn;
    }
}

struct LatentAttnParams {
    const float* q;                                // [T, H * D]: per head [qa (rk) ; q_rot (dr)]
    const float* cache;
    const int* table; int stride; int page;
    float* part;                                   // [T][H][nsplit][rk + 2]: unnormalised o, running max, running sum
    int H, rk, dr, nsplit;
    float scale;
    MetaView meta; SeqMeta sm;
};

constexpr int LA_KT = 32;                          // keys per tile (one per lane in the score phase)
constexpr int LA_THREADS = 128;
constexpr int LA_MAX_RK_CHUNKS = 16;               // rk <= 512

template <int QB, int HG>
__host__ __device__ constexpr size_t latent_attn_smem(int D) {
    return ((size_t)QB * HG * D + (size_t)LA_KT * (D + 1) + (size_t)QB * HG * LA_KT) * sizeof(float);
}

template <int QB, int HG>
__global__ void __launch_bounds__(LA_THREADS) latent_attn_kernel(const LatentAttnParams p) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int R = QB * HG;                     // (token, head) rows of this CTA
    constexpr int RPW = R / 4;                     // rows per warp
    static_assert(R % 4 == 0, "rows must split over four warps");
    const int ci = blockIdx.x;
    if (ci >= p.sm.n_chunks()) return;
    const int t0 = p.sm.chunk_start()[ci], nt = p.sm.chunk_count()[ci];
    const int h0 = blockIdx.y * HG;
    const int D = p.rk + p.dr, rk = p.rk;
    const int slot = p.meta.tok_slot()[t0];
    const int pos0 = p.sm.tok_pos()[t0];           // chunk tokens sit at consecutive positions pos0, pos0 + 1, ...
    const int nkeys = pos0 + nt;                   // keys 0 .. pos0 + nt - 1 are visible to the last token
    const int tiles = (nkeys + LA_KT - 1) / LA_KT;
    const int per = (tiles + p.nsplit - 1) / p.nsplit;
    const int tile_lo = blockIdx.z * per, tile_hi = min(tiles, tile_lo + per);

    extern __shared__ float la_smem[];
    float* sq = la_smem;                             // [R][D]
    float* sk = sq + (size_t)R * D;                // [LA_KT][D + 1]
    float* sp = sk + (size_t)LA_KT * (D + 1);      // [R][LA_KT]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    for (int e = threadIdx.x; e < R * D; e += LA_THREADS) {
        const int r = e / D, d = e % D;
        const int qi = r / HG, h = h0 + r % HG;
        sq[e] = (qi < nt && h < p.H) ? p.q[(size_t)(t0 + qi) * p.H * D + (size_t)h * D + d] : 0.f;
    }
    float m[RPW], l[RPW], o[RPW][LA_MAX_RK_CHUNKS];
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
        m[i] = -CUDART_INF_F; l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < LA_MAX_RK_CHUNKS; ++c) o[i][c] = 0.f;
    }
    const int* tab = p.table + (size_t)slot * p.stride;
    for (int tile = tile_lo; tile < tile_hi; ++tile) {
        const int kb = tile * LA_KT;
        __syncthreads();                           // previous tile fully consumed (and sq written, first time)
        for (int e = threadIdx.x; e < LA_KT * D; e += LA_THREADS) {
            const int j = e / D, d = e % D;
            const int kj = kb + j;
            float v = 0.f;
            if (kj < nkeys) v = p.cache[((size_t)tab[kj / p.page] * p.page + kj % p.page) * D + d];
            sk[(size_t)j * (D + 1) + d] = v;
        }
        __syncthreads();
        // scores: lane = key
        float s[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) s[i] = 0.f;
        const float* kr = sk + (size_t)lane * (D + 1);
        for (int d = 0; d < D; ++d) {
            const float kv = kr[d];
#pragma unroll
            for (int i = 0; i < RPW; ++i) s[i] = fmaf(sq[(size_t)(warp * RPW + i) * D + d], kv, s[i]);
        }
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
            const int r = warp * RPW + i;
            const int qi = r / HG;
            const bool live = qi < nt && (kb + lane) <= pos0 + qi;          // causal: key position <= query position
            const float sc = live ? s[i] * p.scale : -CUDART_INF_F;
            float mx = sc;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
            const float mn = fmaxf(m[i], mx);
            float pj = 0.f, corr = 1.f;
            if (mn > -CUDART_INF_F) {
                pj = live ? expf(sc - mn) : 0.f;
                corr = expf(m[i] - mn);            // m = -inf -> 0
            }
            float ps = pj;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, of);
            l[i] = l[i] * corr + ps;
            m[i] = mn;
#pragma unroll
            for (int c = 0; c < LA_MAX_RK_CHUNKS; ++c) o[i][c] *= corr;
            sp[(size_t)r * LA_KT + lane] = pj;
        }
        __syncwarp();
        // weighted sum of the latent rows: lane = latent channel (mod 32)
#pragma unroll
        for (int c = 0; c < LA_MAX_RK_CHUNKS; ++c) {
            const int d = c * 32 + lane;
            if (c * 32 >= rk) break;
            if (d < rk) {
                for (int j = 0; j < LA_KT; ++j) {
                    const float kv = sk[(size_t)j * (D + 1) + d];
#pragma unroll
                    for (int i = 0; i < RPW; ++i) o[i][c] = fmaf(sp[(size_t)(warp * RPW + i) * LA_KT + j], kv, o[i][c]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
        const int r = warp * RPW + i;
        const int qi = r / HG, h = h0 + r % HG;
        if (qi >= nt || h >= p.H) continue;
        float* dst = p.part + (((size_t)(t0 + qi) * p.H + h) * p.nsplit + blockIdx.z) * (rk + 2);
#pragma unroll
        for (int c = 0; c < LA_MAX_RK_CHUNKS; ++c) {
            const int d = c * 32 + lane;
            if (d < rk) dst[d] = o[i][c];
        }
        if (lane == 0) { dst[rk] = m[i]; dst[rk + 1] = l[i]; }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Tensor-core variant for the serving precision: the same CTA shape (16 (token, head) rows, 32-key tiles, online softmax in
// f32) with both products on mma.sync m16n8k8 TF32 (operands rounded to TF32, f32 accumulation):
//   scores  S[16 x 32]  = Q[16 x D] . K^T      warp w owns keys 8 (w % 4) .. + 7 and half of the channels, in two chains of sums
//   output  O[16 x rk] += P[16 x 32] . C       warp w owns an eighth of the latent channels, 4 k-steps per 8 channels
// Scores go through shared memory between the two so that the softmax keeps the row-per-warp form of the f32 kernel.
// Row strides are = 4 (mod 32) floats: fragment loads are bank-conflict free in the score phase, and in the output phase with keys 2 t and 2 t + 1 of eight in the places t and t + 4.
// What bounds it: the chain of a CTA that holds two or three tiles (fetch, scores, softmax, output), not bytes.  A row is fetched by a warp (one division by the page size a row; one
// for every sixteen bytes, and the queries word by word with two more, before).
// Measured (a decode step of sixteen sequences of 780 keys, 16 heads, rank 512 and 64 rotated, in place): 63 us of the step -> 29.
// ------------------------------------------------------------------------------------------------------------------
// nearest TF32 value, ties away from zero (what cvt.rna does), in integer operations: every operand of every product is rounded, and the
// conversion's issue rate was what the two products waited for.  A NaN stays one (the addition would carry it into another value).
__device__ __forceinline__ uint32_t to_tf32(float v) { return v != v ? 0x7FFFE000u : (__float_as_uint(v) + 0x1000u) & 0xFFFFE000u; }
__device__ __forceinline__ void mma_tf32_1688(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__host__ __device__ inline int la_pad8(int n) { return (n + 7) & ~7; }
__host__ __device__ inline int la_stride(int D) { const int dp = la_pad8(D); return dp + ((4 - dp % 32) + 32) % 32; }
__host__ __device__ inline size_t latent_attn_tc_smem(int D) {
    return ((size_t)16 * la_stride(D) + (size_t)LA_KT * la_stride(D) + 2 * 16 * 32 + 64) * sizeof(float);      // two CTAs of an SM at 576 channels
}
constexpr int LT_THREADS = 256, LT_MAX_NT = 8;     // 8-channel tiles per warp: rk <= 512

template <int QB, int HG>
__global__ void __launch_bounds__(LT_THREADS) latent_attn_tc_kernel(const LatentAttnParams p) {
    pdl_launch_dependents();
    pdl_wait();
    static_assert(QB * HG == 16, "one m16 tile of (token, head) rows");
    const int ci = blockIdx.x;
    if (ci >= p.sm.n_chunks()) return;
    const int t0 = p.sm.chunk_start()[ci], nt = p.sm.chunk_count()[ci];
    const int h0 = blockIdx.y * HG;
    const int D = p.rk + p.dr, rk = p.rk, Dp = la_pad8(D), DS = la_stride(D);
    const int slot = p.meta.tok_slot()[t0];
    const int pos0 = p.sm.tok_pos()[t0];
    const int nkeys = pos0 + nt;
    const int tiles = (nkeys + LA_KT - 1) / LA_KT;
    const int per = (tiles + p.nsplit - 1) / p.nsplit;
    const int tile_lo = blockIdx.z * per, tile_hi = min(tiles, tile_lo + per);

    extern __shared__ __align__(16) float la_tc_smem[];
    float* sq = la_tc_smem;                        // [16][DS]
    float* sk = sq + (size_t)16 * DS;              // [LA_KT][DS]
    float* ss = sk + (size_t)LA_KT * DS;           // [2][16][32] scores of the two halves of the channels (columns turned: at()); probabilities in the first
    float* scorr = ss + 2 * 16 * 32;               // [16] rescale of the running output
    float* sml = scorr + 16;                       // [16][2] final (m, l)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const int* tab = p.table + (size_t)slot * p.stride;
    const bool vec = (D % 4 == 0);
    auto at = [](const int r, const int c) { return r * 32 + (c ^ ((r & 7) << 2)); };
    auto fetch = [&](const int kb) {               // a row of the cache per warp and turn
        for (int j = warp; j < LA_KT; j += LT_THREADS / 32) {
            const int kj = kb + j;
            float* const dst = sk + (size_t)j * DS;
            if (kj < nkeys) {
                const float* const src = p.cache + ((size_t)tab[kj / p.page] * p.page + kj % p.page) * D;
                if (vec) {
                    const uint32_t da = (uint32_t)__cvta_generic_to_shared(dst);
                    for (int c = lane; c < D / 4; c += 32) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(da + 16 * c), "l"(src + 4 * c) : "memory");
                } else {
                    for (int d = lane; d < D; d += 32) dst[d] = src[d];
                }
            } else {
                for (int d = lane; d < D; d += 32) dst[d] = 0.f;
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (tile_lo < tile_hi) fetch(tile_lo * LA_KT);
#pragma unroll
    for (int r = warp; r < 16; r += LT_THREADS / 32) {
        const int qi = r / HG, h = h0 + r % HG;
        const bool live = qi < nt && h < p.H;
        const float* const src = p.q + (live ? (size_t)(t0 + qi) * p.H * D + (size_t)h * D : 0);
        float* const dst = sq + (size_t)r * DS;
        if (vec) {
            for (int c = lane; c < D / 4; c += 32) {
                const float4 x = live ? *reinterpret_cast<const float4*>(src + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<uint4*>(dst + 4 * c) = make_uint4(to_tf32(x.x), to_tf32(x.y), to_tf32(x.z), to_tf32(x.w));
            }
        } else {
            for (int d = lane; d < D; d += 32) dst[d] = live ? __uint_as_float(to_tf32(src[d])) : 0.f;
        }
        for (int d = D + lane; d < DS; d += 32) dst[d] = 0.f;
    }
    for (int j = warp; j < LA_KT; j += LT_THREADS / 32)       // pad columns of the key tile stay zero
        for (int d = D + lane; d < DS; d += 32) sk[(size_t)j * DS + d] = 0.f;
    constexpr int RPW = 16 / (LT_THREADS / 32);
    float m[RPW], l[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) { m[i] = -CUDART_INF_F; l[i] = 0.f; }
    const int cw = la_pad8((rk + 7) / 8);          // latent channels per warp, a multiple of 8
    const int steps = Dp / 8, s_lo = (warp >> 2) ? (steps + 1) / 2 : 0, s_hi = (warp >> 2) ? steps : (steps + 1) / 2;      // this warp's channels of the scores
    float o[LT_MAX_NT][4];
#pragma unroll
    for (int n = 0; n < LT_MAX_NT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    for (int tile = tile_lo; tile < tile_hi; ++tile) {
        const int kb = tile * LA_KT;
        if (tile > tile_lo) {
            __syncthreads();                       // the previous tile is consumed
            fetch(kb);
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        {   // scores of keys 8 * (warp % 4) .. + 7
            float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            const float* qa0 = sq + (size_t)gq * DS + tq;
            const float* qa1 = sq + (size_t)(gq + 8) * DS + tq;
            const float* kb0 = sk + (size_t)((warp & 3) * 8 + gq) * DS + tq;
            auto step = [&](const int ks, float (&c)[4]) {
                uint32_t a[4], b[2];
                a[0] = __float_as_uint(qa0[ks]); a[1] = __float_as_uint(qa1[ks]); a[2] = __float_as_uint(qa0[ks + 4]); a[3] = __float_as_uint(qa1[ks + 4]);
                b[0] = to_tf32(kb0[ks]); b[1] = to_tf32(kb0[ks + 4]);
                mma_tf32_1688(c, a, b);
            };
            int s = s_lo;
#pragma unroll 4
            for (; s + 1 < s_hi; s += 2) { step(8 * s, acc[0]); step(8 * s + 8, acc[1]); }
            if (s < s_hi) step(8 * s, acc[0]);
            float* const d = ss + (warp >> 2) * 16 * 32;
            const int c = (warp & 3) * 8 + tq * 2;
            *reinterpret_cast<float2*>(d + at(gq, c)) = make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
            *reinterpret_cast<float2*>(d + at(gq + 8, c)) = make_float2(acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < RPW; ++i) {            // softmax rows 2 * warp, + 1, lane = key
            const int r = warp * RPW + i;
            const int qi = r / HG;
            const bool live = qi < nt && (kb + lane) <= pos0 + qi;
            const float sc = live ? (ss[at(r, lane)] + ss[16 * 32 + at(r, lane)]) * p.scale : -CUDART_INF_F;
            float mx = sc;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
            const float mn = fmaxf(m[i], mx);
            float pj = 0.f, corr = 1.f;
            if (mn > -CUDART_INF_F) {
                pj = live ? expf(sc - mn) : 0.f;
                corr = expf(m[i] - mn);
            }
            float ps = pj;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, of);
            l[i] = l[i] * corr + ps;
            m[i] = mn;
            ss[at(r, lane)] = __uint_as_float(to_tf32(pj));
            if (lane == 0) scorr[r] = corr;
        }
        __syncthreads();
        {   // output: this warp's latent channels
            uint32_t a[4][4];
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const float2 u = *reinterpret_cast<const float2*>(ss + at(gq, ks * 8 + 2 * tq)), v = *reinterpret_cast<const float2*>(ss + at(gq + 8, ks * 8 + 2 * tq));
                a[ks][0] = __float_as_uint(u.x); a[ks][1] = __float_as_uint(v.x);
                a[ks][2] = __float_as_uint(u.y); a[ks][3] = __float_as_uint(v.y);
            }
            const float c0 = scorr[gq], c1 = scorr[gq + 8];
#pragma unroll
            for (int n = 0; n < LT_MAX_NT; ++n) {
                const int cb = warp * cw + n * 8;
                if (n * 8 >= cw || cb >= rk) break;
                o[n][0] *= c0; o[n][1] *= c0; o[n][2] *= c1; o[n][3] *= c1;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    uint32_t b[2];
                    b[0] = to_tf32(sk[(size_t)(ks * 8 + 2 * tq) * DS + cb + gq]);
                    b[1] = to_tf32(sk[(size_t)(ks * 8 + 2 * tq + 1) * DS + cb + gq]);
                    mma_tf32_1688(o[n], a[ks], b);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RPW; ++i)
        if (lane == 0) { sml[(warp * RPW + i) * 2] = m[i]; sml[(warp * RPW + i) * 2 + 1] = l[i]; }
    __syncthreads();
#pragma unroll
    for (int hrow = 0; hrow < 2; ++hrow) {
        const int r = gq + hrow * 8;
        const int qi = r / HG, h = h0 + r % HG;
        if (qi >= nt || h >= p.H) continue;
        float* dst = p.part + (((size_t)(t0 + qi) * p.H + h) * p.nsplit + blockIdx.z) * (rk + 2);
#pragma unroll
        for (int n = 0; n < LT_MAX_NT; ++n) {
            const int cb = warp * cw + n * 8;
            if (n * 8 >= cw || cb >= rk) break;
            const int d = cb + tq * 2;
            if (d < rk) dst[d] = o[n][hrow * 2];
            if (d + 1 < rk) dst[d + 1] = o[n][hrow * 2 + 1];
        }
        if (warp == 0 && tq == 0) { dst[rk] = sml[r * 2]; dst[rk + 1] = sml[r * 2 + 1]; }
    }
}

struct LatentMergeParams {
    const float* part;
    float* out;                                    // [T, H * rk]
    int H, rk, nsplit;
    MetaView meta;
};

constexpr int LM_MAX_SPLIT = 16;                   // parts of a step's keys at most: what SeqModel::max_split begins with

// parts of a token's head -> its output.  The parts' factors are worked out once, and a thread requests its channel of eight parts at a time (part after part, with the factor of each
// behind two dependent reads, before: 9.6 us of the step above, 6.5 now)
__global__ void __launch_bounds__(128) latent_merge_kernel(const LatentMergeParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, h = blockIdx.y;
    if (t >= p.meta.T()) return;
    __shared__ float s_f[LM_MAX_SPLIT];
    const float* src = p.part + ((size_t)t * p.H + h) * p.nsplit * (p.rk + 2);
    const size_t pitch = p.rk + 2;
    float M = -CUDART_INF_F;
#pragma unroll 8
    for (int z = 0; z < p.nsplit; ++z) M = fmaxf(M, src[z * pitch + p.rk]);
    float Lsum = 0.f;
#pragma unroll 8
    for (int z = 0; z < p.nsplit; ++z) {
        const float mz = src[z * pitch + p.rk], lz = src[z * pitch + p.rk + 1];
        if (mz > -CUDART_INF_F) Lsum += lz * expf(mz - M);
    }
    for (int z = threadIdx.x; z < p.nsplit; z += blockDim.x) {
        const float mz = src[z * pitch + p.rk];
        s_f[z] = mz > -CUDART_INF_F ? expf(mz - M) : -1.f;
    }
    __syncthreads();
    const float inv = 1.f / Lsum;
    for (int d = threadIdx.x; d < p.rk; d += blockDim.x) {
        float acc = 0.f;
#pragma unroll 8
        for (int z = 0; z < p.nsplit; ++z) {
            const float f = s_f[z], x = src[z * pitch + d];
            if (f >= 0.f) acc += x * f;
        }
        p.out[(size_t)t * p.H * p.rk + (size_t)h * p.rk + d] = acc * inv;
    }
}

}  // namespace b200
