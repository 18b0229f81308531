// GPU front half of token sampling: penalties + allowed-token mask + bias + softmax + top-k, per slot, on the logits the
// head projection left in HBM.  Only <= 128 (token id, probability) pairs per slot cross PCIe.
//
// Replaces, for samplers that need only the head of the sorted distribution (Nucleus with top_k <= 128, greedy), what the
// reference does per generated token per slot:
//   crates/ai00-core/src/run.rs:664-697   output.to_vec() (num_vocab f32 = 256 KiB D2H), Sampler::transform (penalties,
//                                         sampler/nucleus.rs:61-67), Formatter::transform (BNF mask, sampler/bnf.rs:37-40),
//                                         bias add (run.rs:679-681), softmax round trip (2 x 256 KiB, run.rs:1164-1190)
//   crates/ai00-core/src/sampler/nucleus.rs:69-80   full-vocabulary radix sort, `.rev().take(top_k)`
// The random draw, top_p cut, temperature and the penalty update (nucleus.rs:81-123) stay on the host: they need the
// sampler's state and RNG and touch <= top_k numbers.
//
// Order of the candidates: adjusted logit descending, token id ascending on ties -- a strict total order, so results are
// reproducible.  (The reference sorts probabilities with an unstable radix sort: any order of equal probabilities is a
// valid outcome there; this is one of them, because the probability is a non-decreasing function of the logit.)
//
// Shape: one launch, a cluster of eight CTAs per row, an eighth of the row each, in registers (32 elements a thread).  Nothing here is
// bandwidth (16 rows x 256 KB from L2): instructions and trips through the cluster are the cost.
//   * the best element of every thread gives two lower bounds of the row's top_k-th: the smallest over the CTAs of the (top_k / 8)-th best
//     thread, and the largest over the CTAs of the top_k-th best thread.  Elements at or above the larger bound are candidates: about
//     1.7 top_k of them for a smooth row.  All of this compares ordered logits alone, 32 bits an element;
//   * candidates carry their place in the total order, one 64-bit key (ordered logit, inverted id).  A CTA with more than it may share (many
//     equal logits, or the row's best in few threads) keeps its own best top_k, found with whole keys;
//   * what a CTA has to say goes into the others' shared memory before a cluster barrier, so that no remote read is waited for: bounds and softmax
//     statistics at the first, candidates at the second.  Every CTA ranks its own candidates against all: a rank below top_k IS the output position.
//     Softmax statistics are combined in CTA order.
// Results go straight to pinned host memory.  Measured at rows of 65536: see the figures at topk_kernel.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace b200 {

constexpr int TOPK_MAX = 128;
constexpr int TOPK_CTAS = 8, TOPK_THREADS = 256;                // CTAs of a row (one cluster), threads of a CTA
constexpr int TOPK_PER_THREAD = 32;                             // elements
constexpr int TOPK_SLICE = TOPK_THREADS * TOPK_PER_THREAD;      // elements of a CTA: 8192
constexpr int TOPK_MAX_V = TOPK_CTAS * TOPK_SLICE;              // 65536
constexpr int TOPK_LIST = 4096;                                 // list of a CTA: what is left after a cut (32 elements of top_k threads at most); a first pass may count more and collects again
static_assert(TOPK_LIST >= TOPK_PER_THREAD * TOPK_MAX, "a CTA's own best top_k come from top_k threads");
constexpr int TOPK_SHARE = 512;                                 // candidates a CTA may share
constexpr int TOPK_PITCH_PAD = 4;                               // eight CTAs' lists, read side by side, start in different banks
constexpr int TOPK_INLINE = 64;                                 // rows whose slots travel as kernel parameters
__host__ __device__ constexpr int topk_slice(int V) { return ((V + TOPK_CTAS - 1) / TOPK_CTAS + 3) & ~3; }      // elements of a CTA
// entries of its list, and bytes of shared memory (a small vocabulary cannot fill either: more CTAs to an SM)
__host__ __device__ constexpr int topk_list(int V) { return topk_slice(V) < TOPK_LIST ? topk_slice(V) : TOPK_LIST; }
__host__ __device__ constexpr int topk_pitch(int V) { return (topk_slice(V) < TOPK_SHARE ? topk_slice(V) : TOPK_SHARE) + TOPK_PITCH_PAD; }
__host__ __device__ constexpr size_t topk_smem(int V) { return ((size_t)topk_list(V) + (size_t)TOPK_CTAS * topk_pitch(V)) * 8; }

struct TopkParams {
    const float* keep;          // [S][V] last logits row of every slot
    int V;
    const int* slot;            // [nrows] (null: slot_inline)
    int slot_inline[TOPK_INLINE];
    // adjustments (all null: none)
    const int* pen_off;         // [nrows + 1]
    const unsigned* pen_tok;    // logits[tok] -= val   (entries of one row have distinct tokens)
    const float* pen_val;
    const int* bias_off;        // [nrows + 1]
    const unsigned* bias_tok;   // logits[tok] += val   (distinct tokens within a row)
    const float* bias_val;
    const unsigned* allow;      // optional [nrows][ceil(V / 32)]: bit = 1 -> token allowed; disallowed -> -inf
    int top_k;
    unsigned* out_id;           // [nrows][top_k], pinned host memory
    float* out_p;               // [nrows][top_k]
};

// larger logit, larger number (-0 and +0 are one value); 0 is below every logit
__device__ __forceinline__ unsigned topk_order(float x) {
    const unsigned b = __float_as_uint(x == 0.f ? 0.f : x);
    return b ^ (0x80000000u | (unsigned)((int)b >> 31));
}
// strict total order as one number: larger logit first, then smaller id; 0 is below every element
__device__ __forceinline__ unsigned long long topk_key(unsigned order, unsigned id) { return ((unsigned long long)order << 32) | (unsigned)~id; }
__device__ __forceinline__ float topk_logit(unsigned long long key) {
    const unsigned o = (unsigned)(key >> 32);
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// top_k = 128 of rows of 65536, launches back to back: 20.5 us of one row and 24.7 of sixteen with whole keys throughout and remote reads (of 28.7 thousand cycles of a CTA
// 8.5 went into ranking the threads' best, 5.0 into picking candidates, 3.0 into each thread's best, 3.5 into remote reads); here 14.0 and 18.5 (15.1 thousand cycles: 2.7 for the
// ranking, 2.7 for the candidates).  A decode step with its sampling, 3B widths and one sequence: 414 -> 406 us; 7B widths, sixteen: 561 -> 552.
__global__ void __cluster_dims__(TOPK_CTAS, 1, 1) __launch_bounds__(TOPK_THREADS) topk_kernel(const __grid_constant__ TopkParams p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char topk_smem[];
    unsigned long long* const list = reinterpret_cast<unsigned long long*>(topk_smem);      // [topk_list(V)]
    unsigned long long* const all = list + topk_list(p.V);                                  // [TOPK_CTAS][topk_pitch(V)], written by the CTAs of the cluster
    float* const sx = reinterpret_cast<float*>(topk_smem);                                  // [cnt] while lists are applied
    __shared__ __align__(16) unsigned s_best[TOPK_THREADS];
    __shared__ __align__(16) unsigned long long s_key[TOPK_THREADS];
    __shared__ unsigned s_few, s_full;                      // the (top_k / 8)-th and the top_k-th best thread
    __shared__ unsigned long long s_cut;
    __shared__ __align__(16) uint4 s_stat[TOPK_CTAS];       // every CTA's two bounds, max and sum exp(x - max)
    __shared__ int s_cnt[TOPK_CTAS];                        // and how many candidates it shares
    __shared__ float red[32];
    __shared__ int s_n;
    static_assert(TOPK_THREADS / 32 == TOPK_CTAS, "a warp for every CTA of the cluster");
    cluster.barrier_arrive();                               // (waited for before the first write to another CTA: all have begun)
    const int cta = blockIdx.x, row = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int slice = topk_slice(p.V);
    const int lo = min(cta * slice, p.V), cnt = min(lo + slice, p.V) - lo;
    const float* const src = p.keep + (size_t)(p.slot ? p.slot[row] : p.slot_inline[row]) * p.V + lo;
    // slices below four elements a thread are dealt out one by one: with whole float4 too few threads would hold any for the bounds below
    const bool quads = slice >= 4 * TOPK_THREADS, vec = quads && (p.V & 3) == 0;        // (rows and slices start on 16-byte boundaries)
    auto index = [&](int j) { return quads ? ((j >> 2) * TOPK_THREADS + tid) * 4 + (j & 3) : j * TOPK_THREADS + tid; };     // place of x[j] in the slice
    float x[TOPK_PER_THREAD];
#pragma unroll
    for (int q = 0; q < TOPK_PER_THREAD / 4; ++q) {
        const int i = index(4 * q);
        if (vec && i + 3 < cnt) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(src + i));
            x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) x[4 * q + e] = index(4 * q + e) < cnt ? __ldcg(src + index(4 * q + e)) : -INFINITY;
        }
    }
    if (p.pen_off || p.bias_off || p.allow) {
#pragma unroll
        for (int j = 0; j < TOPK_PER_THREAD; ++j)
            if (index(j) < cnt) sx[index(j)] = x[j];
        __syncthreads();
        auto apply = [&](const int* off, const unsigned* tok, const float* val, const float sign) {
            for (int e = off[row] + tid; e < off[row + 1]; e += TOPK_THREADS) {
                const int i = (int)tok[e] - lo;
                if (tok[e] < (unsigned)p.V && i >= 0 && i < cnt) sx[i] = fmaf(sign, val[e], sx[i]);
            }
        };
        // Sampler::transform (penalties), Formatter::transform (tokens the grammar does not allow), bias: in this order
        if (p.pen_off) apply(p.pen_off, p.pen_tok, p.pen_val, -1.f);
        __syncthreads();
        if (p.allow) {
            const unsigned* allow = p.allow + (size_t)row * ((p.V + 31) / 32);
            for (int i = tid; i < cnt; i += TOPK_THREADS)
                if (!((allow[(lo + i) >> 5] >> ((lo + i) & 31)) & 1u)) sx[i] = -INFINITY;
        }
        __syncthreads();
        if (p.bias_off) apply(p.bias_off, p.bias_tok, p.bias_val, 1.f);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < TOPK_PER_THREAD; ++j)
            if (index(j) < cnt) x[j] = sx[index(j)];
    }
    // softmax statistics of the slice (places behind the slice hold -inf), best element of the thread
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < TOPK_PER_THREAD; ++j) mx = fmaxf(mx, x[j]);
    unsigned o[TOPK_PER_THREAD], best = 0;                  // 0: not an element
#pragma unroll
    for (int j = 0; j < TOPK_PER_THREAD; ++j) {
        o[j] = cnt == TOPK_SLICE || index(j) < cnt ? max(topk_order(x[j]), 1u) : 0u;
        best = max(best, o[j]);
    }
    s_best[tid] = best;
    if (tid == 0) { s_few = s_full = ~0u; s_cut = 0; s_n = 0; }
    mx = block_max_any(mx, red);
    float sum = 0.f;
    if (mx > -INFINITY) {
#pragma unroll
        for (int j = 0; j < TOPK_PER_THREAD; ++j) sum += expf(x[j] - mx);
    }
    sum = block_sum_any(sum, red);                          // (its barriers also publish s_best)
    int above = 0;
#pragma unroll 16
    for (int i = 0; i < TOPK_THREADS; i += 4) {
        const uint4 b = *reinterpret_cast<const uint4*>(s_best + i);
        above += (b.x > best) + (b.y > best) + (b.z > best) + (b.w > best);
    }
    // the k-th best is the least of those with fewer than k above them (0 where fewer than k threads hold elements)
    const unsigned least_few = __reduce_min_sync(0xffffffffu, above < (p.top_k + TOPK_CTAS - 1) / TOPK_CTAS ? best : ~0u);
    const unsigned least_full = __reduce_min_sync(0xffffffffu, above < p.top_k ? best : ~0u);
    if (lane == 0) {
        atomicMin(&s_few, least_few);
        atomicMin(&s_full, least_full);
    }
    __syncthreads();
    cluster.barrier_wait();
    if (tid < TOPK_CTAS) *cluster.map_shared_rank(&s_stat[cta], tid) = make_uint4(s_few, s_full, __float_as_uint(mx), __float_as_uint(sum));
    cluster.sync();
    unsigned few = ~0u, full = 0;
    float M = -INFINITY;
#pragma unroll
    for (int c = 0; c < TOPK_CTAS; ++c) { few = min(few, s_stat[c].x); full = max(full, s_stat[c].y); M = fmaxf(M, __uint_as_float(s_stat[c].z)); }
    const unsigned bound = max(max(few, full), 1u);
    // elements from `least` on -> list, in any order; how many there are
    auto collect = [&](const unsigned long long least) {
        unsigned mask = 0;
#pragma unroll
        for (int j = 0; j < TOPK_PER_THREAD; ++j) mask |= (unsigned)(topk_key(o[j], (unsigned)(lo + index(j))) >= least) << j;
        const int mine = __popc(mask);
        int at = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, at, d);
            if (lane >= d) at += v;
        }
        int wbase = 0;
        if (lane == 31 && at) wbase = atomicAdd(&s_n, at);
        at += __shfl_sync(0xffffffffu, wbase, 31) - mine;
        if (mask) {
#pragma unroll
            for (int j = 0; j < TOPK_PER_THREAD; ++j)
                if (mask >> j & 1u) {
                    if (at < topk_list(p.V)) list[at] = topk_key(o[j], (unsigned)(lo + index(j)));
                    ++at;
                }
        }
        __syncthreads();
        return s_n;
    };
    int n = collect(topk_key(bound, ~0u));
    if (n > TOPK_SHARE) {                                   // the CTA's own best top_k: elements from its top_k-th best thread on (at most 32 top_k), ranked
        unsigned long long bkey = 0;
#pragma unroll
        for (int j = 0; j < TOPK_PER_THREAD; ++j)
            if (o[j] >= bound) bkey = max(bkey, topk_key(o[j], (unsigned)(lo + index(j))));
        s_key[tid] = bkey;
        __syncthreads();
        int over = 0;
#pragma unroll 16
        for (int i = 0; i < TOPK_THREADS; i += 2) {
            const ulonglong2 b2 = *reinterpret_cast<const ulonglong2*>(s_key + i);
            over += (b2.x > bkey) + (b2.y > bkey);
        }
        if (bkey && over == p.top_k - 1) s_cut = bkey;
        if (tid == 0) s_n = 0;
        __syncthreads();
        n = collect(max(s_cut, topk_key(bound, ~0u)));
        unsigned long long key[TOPK_LIST / TOPK_THREADS];
        int rank[TOPK_LIST / TOPK_THREADS];
        for (int u = 0; u < TOPK_LIST / TOPK_THREADS; ++u) {
            const int i = tid + u * TOPK_THREADS;
            key[u] = i < n ? list[i] : 0;
            rank[u] = 0;
            for (int k = 0; k < n && i < n; ++k) rank[u] += list[k] > key[u];
        }
        __syncthreads();
        for (int u = 0; u < TOPK_LIST / TOPK_THREADS; ++u)
            if (tid + u * TOPK_THREADS < n && rank[u] < p.top_k) list[rank[u]] = key[u];
        n = min(n, p.top_k);
        __syncthreads();
    }
    const int pitch = topk_pitch(p.V);
    {                                                       // warp w: to CTA w
        unsigned long long* const to = cluster.map_shared_rank(all, warp) + cta * pitch;
        for (int i = lane; i < n; i += 32) to[i] = list[i];
        if (lane == 0) *cluster.map_shared_rank(&s_cnt[cta], warp) = n;
    }
    cluster.sync();                                         // nothing remote is touched from here on: a CTA may leave when it is done
    float denom = 0.f;
#pragma unroll
    for (int c = 0; c < TOPK_CTAS; ++c) {
        const float m = __uint_as_float(s_stat[c].z);
        if (m > -INFINITY) denom += __uint_as_float(s_stat[c].w) * expf(m - M);
    }
    const float inv = 1.0f / denom;
    const int seg = lane >> 2, nseg = s_cnt[seg];           // four lanes to a CTA's list
    for (int i = warp; i < n; i += TOPK_THREADS / 32) {
        const unsigned long long key = list[i];
        int rank = 0;
        for (int k = lane & 3; k < nseg; k += 4) rank += all[seg * pitch + k] > key;
        rank = __reduce_add_sync(0xffffffffu, rank);
        if (lane == 0 && rank < p.top_k) {
            // same expression as softmax_kernel (misc.cuh): exp(x - max) * (1 / sum)
            const float v = topk_logit(key);
            p.out_id[(size_t)row * p.top_k + rank] = ~(unsigned)key;
            p.out_p[(size_t)row * p.top_k + rank] = v > -INFINITY ? expf(v - M) * inv : 0.f;
        }
    }
    if (cta == 0)
        for (int i = p.V + tid; i < p.top_k; i += TOPK_THREADS) {       // a vocabulary smaller than top_k
            p.out_id[(size_t)row * p.top_k + i] = 0xFFFFFFFFu;
            p.out_p[(size_t)row * p.top_k + i] = 0.f;
        }
}

// ---------------------------------------------------------------------------------------
// Last logits row of every slot that produced one in this step -> keep[slot][V].  The rows of a step are overwritten by
// the next step, which may belong to other slots (the reference samples every slot in its own task while the infer loop
// goes on, run.rs:1230-1240), so the front half above reads from this per-slot copy.  Tensor parallel: rank 0 gathers the
// vocabulary shards of all ranks (rows complete after the step's last rendezvous).
// ---------------------------------------------------------------------------------------
struct KeepParams {
    const float* shard[8];      // [R][Vl] logits shard of every rank (peer mapped)
    int world, Vl, V;
    MetaView meta;
    float* keep;                // [S][V]
};
constexpr int KEEP_THREADS = 256;
constexpr int KEEP_CHUNKS = 8;

__global__ void __launch_bounds__(KEEP_THREADS) keep_rows_kernel(const __grid_constant__ KeepParams p) {
    pdl_launch_dependents();
    const int r = blockIdx.x;
    const int R = p.meta.R();
    const int t = (r < R) ? p.meta.out_tok()[r] : 0;
    const bool live = r < R && p.meta.tok_last()[t] != 0;
    const int slot = live ? p.meta.tok_slot()[t] : 0;
    pdl_wait();
    if (!live) return;
    float* dst = p.keep + (size_t)slot * p.V;
    auto copy = [&](auto vec_t) {                           // whole float4 where every row begins on a 16-byte boundary
        using T = decltype(vec_t);
        const int n = p.Vl / (int)(sizeof(T) / 4);
        for (int q = 0; q < p.world; ++q) {
            const T* src = reinterpret_cast<const T*>(p.shard[q] + (size_t)r * p.Vl);
            T* d = reinterpret_cast<T*>(dst + (size_t)q * p.Vl);
            for (int i = blockIdx.y * KEEP_THREADS + threadIdx.x; i < n; i += KEEP_CHUNKS * KEEP_THREADS) d[i] = __ldcg(src + i);
        }
    };
    if ((p.Vl & 3) == 0) copy(float4{});
    else copy(0.f);
}

}  // namespace b200
