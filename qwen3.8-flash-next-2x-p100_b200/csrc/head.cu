// Head-side kernels: per-row argmax, the sampler's 64 candidates, embedding rows, RMS norm rows.
//
// fnx_argmax replaces argmax / k_argmax (engine/src/kernels.hpp:433, engine/src/kernels.cu:1056-1083): the same
// total order, value first and the lower index on ties.  fnx_top_tokens replaces top_tokens / k_topk_rows
// (engine/src/kernels.hpp:445, engine/src/topk.cuh:17-155) without penalties or logit bias: the 64 largest by the
// 64-bit key (ordered logit bits, ~index), which has no ties.
#include <cooperative_groups.h>

#include "fnx_common.cuh"

namespace cg = cooperative_groups;

namespace fnxb {

// float -> uint32 with the same order
__device__ __forceinline__ uint32_t fkey(float v) {
    const uint32_t b = __float_as_uint(v);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float fkey_inv(uint32_t k) { return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k); }
__device__ __forceinline__ unsigned long long key64(float v, int i) { return ((unsigned long long) fkey(v) << 32) | (uint32_t) ~i; }

// the largest key of a warp's 32 (every lane gets it)
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
    const unsigned hi = (unsigned) (k >> 32), top = __reduce_max_sync(0xffffffffu, hi);
    return ((unsigned long long) top << 32) | __reduce_max_sync(0xffffffffu, hi == top ? (unsigned) k : 0u);
}

// Both kernels below take a row by a cluster of NB blocks, a slice each.  Few rows want many blocks; but clusters are placed whole, on SMs of one group, and the
// chip holds 15 of eight blocks, 33 of four and 74 of two at the pace of a lone one: every further round of them costs what a block for a whole row
// would have taken.  Argmax over rows of 40,528, us a launch with 8, 4, 2 and 1 blocks: 5 rows 2.6, 2.9, 4.1, 5.3; 16 rows 3.6, 2.9, 4.1, 5.4; 33 rows 3.8,
// 3.6, 4.1, 5.4; 74 rows 9.3, 6.2, 4.3, 5.5; 75 rows 9.4, 6.2, 6.2, 5.5; 4,000 rows 431, 227, 161, 112.
static int blocks_by_rows(int T) { return T <= 15 ? 8 : T <= 33 ? 4 : T <= 74 ? 2 : 1; }
// A short row gains nothing by more blocks (1 row of 4,096: 2.0 us with eight and with one; of 8,192 2.1 and 2.3).  Where a slice takes long, a second round of
// fours costs more than eight blocks two to an SM (28 rows of 100,000: 5.7 and 4.7, of 40,528 3.6 and 3.8; 40 rows of 262,144, two blocks 13.2, eight 12.3).
static int argmax_blocks(int T, int V) { return V < 8192 ? 1 : V >= 100000 && T > 24 && T <= 40 ? 8 : blocks_by_rows(T); }
// the candidates' second look and their counting cost less in one block up to here (5 rows of 8,192: 5.8 us, with eight 6.8; of 40,528 10.5 and 8.3)
static int top_blocks(int T, int V) { return V < 16384 ? 1 : blocks_by_rows(T); }

// The slices' largest keys meet in the first block's shared memory.  Bound by latency: the launch, the slice's way, one barrier of the cluster.  (Sixteen blocks
// that met in device memory, an atomic maximum and an arrival counter: 4.5 us a launch for five rows of 151,936, 7.6 for twenty; 4.0 and 5.7 now.)
template <int NB>
__global__ void __cluster_dims__(1, NB, 1) __launch_bounds__(1024, 2) k_argmax(const float* __restrict__ logits, int V, const int* __restrict__ map, int* __restrict__ best_i,
                                                                            float* __restrict__ best_v, unsigned* __restrict__ err) {
    __shared__ unsigned long long red[32], every[NB];
    cg::cluster_group cluster = cg::this_cluster();
    if (NB > 1) cluster.sync();   // (the first block's shared memory is there)
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x, nb = NB;
    const float* l = logits + (size_t) t * V;
    unsigned long long best = 0;
    bool bad = false;
    // this block's slice, in float4 units where the row allows; four float4 per thread in flight
    const int V4 = (((uintptr_t) l & 15) == 0) ? V / 4 : 0;
    const int a4 = (int) ((long long) V4 * blockIdx.y / nb), b4 = (int) ((long long) V4 * (blockIdx.y + 1) / nb);
    for (int i0 = a4 + tid; i0 < b4; i0 += 4096) {
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = i0 + 1024 * j < b4 ? reinterpret_cast<const float4*>(l)[i0 + 1024 * j] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + 1024 * j;
            if (i >= b4) continue;
            const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                bad |= !isfinite(e[c]);
                const unsigned long long k = key64(e[c], 4 * i + c);
                best = k > best ? k : best;
            }
        }
    }
    for (int i = 4 * V4 + (int) blockIdx.y * 1024 + tid; i < V; i += nb * 1024) {   // what float4 units do not cover
        const float v = l[i];
        bad |= !isfinite(v);
        const unsigned long long k = key64(v, i);
        best = k > best ? k : best;
    }
    best = warp_max_key(best);
    if ((tid & 31) == 0) red[tid >> 5] = best;
    if (bad) atomicOr(err, (unsigned) FNX_ERR_LOGITS);
    __syncthreads();
    if (tid < 32) {
        best = warp_max_key(red[tid]);
        if (NB > 1 && tid == 0) *cluster.map_shared_rank(every + blockIdx.y, 0) = best;
    }
    if (NB > 1) cluster.sync();
    if (blockIdx.y == 0 && tid < 32) {
        if (NB > 1) best = warp_max_key(tid < nb ? every[tid] : 0ull);
        if (tid == 0) {
            const int row = (int) ~(uint32_t) best;
            best_i[t] = map ? map[row] : row;
            if (best_v) best_v[t] = fkey_inv((uint32_t) (best >> 32));
        }
    }
}

// The 64 candidates of a row.  In a slice a warp's second largest lane maximum bounds the 64th largest value of the block from below as soon as it is the
// smallest of the 32 warps' (64 values are at or above it), so a second look at the slice leaves a few values more than needed (170 of 19,000 where they
// are random), which find their places by counting; the first block then merges the slices' sorted 64 by searching the others for each.  A slice with more
// than TOP_CAP values that high (many equal logits) is selected digit by digit.
// Bound by two looks at the row and a dozen block barriers: with a block a row and nine looks 20 rows of 151,936 logits took 162 us, 4,000 of 40,528 1,115; 14 and
// 237 now, equal logits 178 and 40 (20 rows).
constexpr int TOP_CAP = 1024, TOP_THREADS = 1024;
constexpr int TOP_LD = 8;   // loads in flight a thread

// keys of the slice [lo, hi) at or above `thr` into sel, at most cap of them; returns how many there are (every thread; ends with a barrier)
__device__ __forceinline__ unsigned top_collect(const float* __restrict__ l, int lo, int hi, unsigned long long thr, unsigned long long* sel, unsigned cap, unsigned* count, int tid) {
    if (tid == 0) *count = 0;
    __syncthreads();
    for (int i0 = lo + tid; i0 < hi; i0 += TOP_THREADS * TOP_LD) {
        float v[TOP_LD];
#pragma unroll
        for (int j = 0; j < TOP_LD; ++j) v[j] = i0 + j * TOP_THREADS < hi ? l[i0 + j * TOP_THREADS] : 0.f;
#pragma unroll
        for (int j = 0; j < TOP_LD; ++j) {
            const int i = i0 + j * TOP_THREADS;
            const unsigned long long k = key64(v[j], i);
            if (i < hi && k >= thr) {
                const unsigned at = atomicAdd(count, 1u);
                if (at < cap) sel[at] = k;
            }
        }
    }
    __syncthreads();
    return *count;
}

template <int NB>
__global__ void __cluster_dims__(1, NB, 1) __launch_bounds__(TOP_THREADS) k_top_tokens(const float* __restrict__ logits, int V, float* __restrict__ out_v, int* __restrict__ out_i) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ __align__(16) unsigned long long sel[TOP_CAP + 4];
    __shared__ unsigned long long top[FNX_TOPK_N], every[NB][FNX_TOPK_N];
    __shared__ unsigned low[TOP_THREADS / 32], high[TOP_THREADS / 32], hist[256], count, need_s;
    __shared__ unsigned long long prefix_s;
    cg::cluster_group cluster = cg::this_cluster();
    const int t = blockIdx.x, part = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float* l = logits + (size_t) t * V;
    const int lo = (int) ((long long) V * part / NB), hi = (int) ((long long) V * (part + 1) / NB);
    unsigned mx = 0;
    int from = lo + tid;
    if (hi - lo < TOP_THREADS) {   // a short slice: alike for every warp, up to a value a lane
        const int a = (hi - lo) * warp / 32, b = (hi - lo) * (warp + 1) / 32;
        from = lane < b - a ? lo + a + lane : hi;
    }
    for (int i0 = from; i0 < hi; i0 += TOP_THREADS * TOP_LD) {
        float v[TOP_LD];
#pragma unroll
        for (int j = 0; j < TOP_LD; ++j) v[j] = i0 + j * TOP_THREADS < hi ? l[i0 + j * TOP_THREADS] : l[i0];
#pragma unroll
        for (int j = 0; j < TOP_LD; ++j) mx = max(mx, fkey(v[j]));
    }
    const unsigned first = __reduce_max_sync(0xffffffffu, mx);
    const int who = __ffs(__ballot_sync(0xffffffffu, mx == first)) - 1;
    const unsigned second = __reduce_max_sync(0xffffffffu, lane == who ? 0u : mx);
    if (lane == 0) {
        low[warp] = second;
        high[warp] = first;
    }
    __syncthreads();
    const unsigned bound = __reduce_min_sync(0xffffffffu, low[lane]);
    unsigned n = top_collect(l, lo, hi, (unsigned long long) bound << 32, sel, TOP_CAP, &count, tid);
    if (n > TOP_CAP) {
        // passes of 8 bits from the top: after pass p the first 8 (p + 1) bits of the slice's 64th largest key are known.  It lies between the bound and the
        // largest value: what these two have in common at the top is known before (equal logits: the value, four passes of eight)
        const int known = __clz(bound ^ __reduce_max_sync(0xffffffffu, high[lane])) / 8;
        if (tid == 0) {
            prefix_s = known ? ((unsigned long long) bound << 32) & ~0ull << (64 - 8 * known) : 0ull;
            need_s = FNX_TOPK_N;
        }
        for (int pass = known; pass < 8; ++pass) {
            const int shift = 56 - 8 * pass;
            if (tid < 256) hist[tid] = 0;
            __syncthreads();
            const unsigned long long prefix = prefix_s, mask = pass == 0 ? 0ull : ~0ull << (shift + 8);
            for (int i = lo + tid; i < hi; i += TOP_THREADS) {
                const unsigned long long k = key64(l[i], i);
                if ((k & mask) == prefix) atomicAdd(&hist[(unsigned) (k >> shift) & 255u], 1u);
            }
            __syncthreads();
            if (tid == 0) {
                unsigned need = need_s, b = 255;
                for (;; --b) {
                    if (hist[b] >= need) break;
                    need -= hist[b];
                    if (b == 0) break;
                }
                need_s = need;
                prefix_s = prefix | ((unsigned long long) b << shift);
            }
            __syncthreads();
        }
        n = top_collect(l, lo, hi, prefix_s, sel, TOP_CAP, &count, tid);   // (keys are distinct: 64)
        if (n > TOP_CAP) n = TOP_CAP;
    }
    // the slice's 64 largest in order; fewer where the slice holds fewer (0: no key)
    if (tid < FNX_TOPK_N) top[tid] = 0;
    if (tid < 4) sel[n + tid] = 0;
    __syncthreads();
    if (tid < (int) n) {
        const unsigned long long k = sel[tid];
        unsigned rank = 0;
        for (unsigned j = 0; j < n; j += 4) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(sel + j), b = *reinterpret_cast<const ulonglong2*>(sel + j + 2);
            rank += (a.x > k) + (a.y > k) + (b.x > k) + (b.y > k);
        }
        if (rank < FNX_TOPK_N) top[rank] = k;
    }
    if (NB == 1) {
        __syncthreads();
        if (tid < FNX_TOPK_N) {
            out_v[(size_t) t * FNX_TOPK_N + tid] = fkey_inv((uint32_t) (top[tid] >> 32));
            out_i[(size_t) t * FNX_TOPK_N + tid] = (int) ~(uint32_t) top[tid];
        }
        return;
    }
    cluster.sync();
    if (part == 0 && tid < NB * FNX_TOPK_N) every[tid / FNX_TOPK_N][tid % FNX_TOPK_N] = cluster.map_shared_rank(top, tid / FNX_TOPK_N)[tid % FNX_TOPK_N];
    cluster.sync();   // (no block leaves while its keys are read)
    if (part == 0 && tid < NB * FNX_TOPK_N) {
        const int own = tid / FNX_TOPK_N;
        const unsigned long long k = every[own][tid % FNX_TOPK_N];
        unsigned rank = tid % FNX_TOPK_N, at[NB];   // the larger ones: before it in its own list, and in the others
#pragma unroll
        for (int p = 0; p < NB; ++p) at[p] = 0;
#pragma unroll
        for (int step = FNX_TOPK_N / 2; step; step >>= 1)
#pragma unroll
            for (int p = 0; p < NB; ++p)
                if (every[p][at[p] + step - 1] > k) at[p] += step;
#pragma unroll
        for (int p = 0; p < NB; ++p)
            if (p != own) rank += at[p] + (every[p][at[p]] > k ? 1u : 0u);
        if (k && rank < FNX_TOPK_N) {
            out_v[(size_t) t * FNX_TOPK_N + rank] = fkey_inv((uint32_t) (k >> 32));
            out_i[(size_t) t * FNX_TOPK_N + rank] = (int) ~(uint32_t) k;
        }
    }
}

__global__ void k_embed_rows(const __half* __restrict__ table, const int* __restrict__ tok, int H, float* __restrict__ R) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < H) R[(size_t) t * H + i] = __half2float(table[(size_t) tok[t] * H + i]);
}

__global__ void __launch_bounds__(256) k_rmsnorm(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int n, float eps) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float red[8];
    const int r = blockIdx.x, tid = threadIdx.x;
    const float* xr = x + (size_t) r * n;
    float ss = 0.f;
    for (int i = tid; i < n; i += 256) ss += xr[i] * xr[i];
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    ss = 0.f;
    for (int j = 0; j < 8; ++j) ss += red[j];
    const float sc = rsqrtf(ss / (float) n + eps);
    for (int i = tid; i < n; i += 256) y[(size_t) r * n + i] = xr[i] * sc * w[i];
}

}  // namespace fnxb

using namespace fnxb;

extern "C" int fnx_argmax_mapped(const float* logits, int T, int V, const int* map, int* best_i, float* best_v, unsigned* err, fnx_stream st) {
    FNX_REQUIRE(logits && best_i && err && T >= 1 && V >= 1, "fnx_argmax: bad arguments");
    {
        const int nb = argmax_blocks(T, V);
        auto kernel = nb == 8 ? k_argmax<8> : nb == 4 ? k_argmax<4> : nb == 2 ? k_argmax<2> : k_argmax<1>;
        const cudaError_t le_ = launch_dep(true, kernel, dim3(T, nb), dim3(1024), 0, as_stream(st), logits, V, map, best_i, best_v, err);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_argmax: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_argmax");
    return FNX_OK;
}

extern "C" int fnx_argmax(const float* logits, int T, int V, int* best_i, float* best_v, unsigned* err, fnx_stream st) {
    return fnx_argmax_mapped(logits, T, V, nullptr, best_i, best_v, err, st);
}

extern "C" int fnx_top_tokens(const float* logits, int T, int V, float* out_v, int* out_i, fnx_stream st) {
    FNX_REQUIRE(logits && out_v && out_i && T >= 1 && V >= FNX_TOPK_N, "fnx_top_tokens: bad arguments (vocabulary of at least %d)", FNX_TOPK_N);
    {
        const int nb = top_blocks(T, V);
        auto kernel = nb == 8 ? k_top_tokens<8> : nb == 4 ? k_top_tokens<4> : nb == 2 ? k_top_tokens<2> : k_top_tokens<1>;
        const cudaError_t le_ = launch_dep(true, kernel, dim3(T, nb), dim3(TOP_THREADS), 0, as_stream(st), logits, V, out_v, out_i);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_top_tokens: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_top_tokens");
    return FNX_OK;
}

// ---- the sampler's logit changes (the first half of k_topk_rows, engine/src/topk.cuh:30-45): per window row, the request's
// logit_bias added, then llama.cpp's penalties stage over the row's penalty window: each token of the window once, `repeat`
// multiplying a non-positive logit and dividing a positive one, then frequency x count and presence taken off.
// Row j's window is the last `last_n` tokens of (the sequence's kept tokens, then window rows 0..j): the tokens before the
// one row j's logits choose.  One block per row; the window is staged in shared memory and each thread settles the tokens
// whose first place in the window is its own.
constexpr int ADJ_THREADS = 256;

__global__ void __launch_bounds__(ADJ_THREADS) k_logit_adjust(float* __restrict__ logits, int V, const int* __restrict__ ctx, const int* __restrict__ ctx_n,
                                                             const int* __restrict__ tok, int last_n, float repeat, float freq, float present,
                                                             const int* __restrict__ bias_tok, const float* __restrict__ bias_val, int bias_n) {
    extern __shared__ int win[];
    pdl_wait();
    const int row = blockIdx.x, tid = threadIdx.x;
    float* L = logits + (size_t) row * V;
    for (int i = tid; i < bias_n; i += ADJ_THREADS) {   // each token once in the list
        const int t = bias_tok[i];
        if (t >= 0 && t < V) L[t] += bias_val[i];
    }
    if (last_n <= 0) return;
    const int n = *ctx_n, len = n + row + 1, start = len > last_n ? len - last_n : 0, w = len - start;
    for (int i = tid; i < w; i += ADJ_THREADS) {
        const int at = start + i;
        win[i] = at < n ? ctx[at] : tok[at - n];
    }
    __syncthreads();   // the window staged, and a token in both lists has its bias in before its penalty
    for (int i = tid; i < w; i += ADJ_THREADS) {
        const int t = win[i];
        if (t < 0 || t >= V) continue;
        bool first = true;
        for (int j = 0; j < i && first; ++j) first = win[j] != t;
        if (!first) continue;
        int cnt = 1;
        for (int j = i + 1; j < w; ++j) cnt += win[j] == t;
        float l = L[t];
        l = l <= 0.f ? l * repeat : l / repeat;
        L[t] = __fsub_rn(__fsub_rn(l, __fmul_rn((float) cnt, freq)), present);   // each step rounded, as written (no fused multiply-add)
    }
}

extern "C" int fnx_logit_adjust(float* logits, int T, int V, const int* ctx, const int* ctx_n, const int* tok, int last_n, float repeat, float freq,
                                float present, const int* bias_tok, const float* bias_val, int bias_n, fnx_stream st) {
    FNX_REQUIRE(logits && T >= 1 && T <= FNX_MAX_ROWS && V >= 1, "fnx_logit_adjust: bad arguments");
    FNX_REQUIRE(last_n >= 0 && last_n <= FNX_PENALTY_CAP, "fnx_logit_adjust: a penalty window of %d tokens (0..%d)", last_n, FNX_PENALTY_CAP);
    FNX_REQUIRE(last_n == 0 || (ctx && ctx_n && tok), "fnx_logit_adjust: penalties need the context and the window's tokens");
    FNX_REQUIRE(last_n == 0 || repeat > 0.f, "fnx_logit_adjust: repeat penalty %g (> 0)", (double) repeat);
    FNX_REQUIRE(bias_n >= 0 && (bias_n == 0 || (bias_tok && bias_val)), "fnx_logit_adjust: a bias list of %d entries without its arrays", bias_n);
    {
        const cudaError_t le_ = launch_dep(true, k_logit_adjust, dim3(T), dim3(ADJ_THREADS), sizeof(int) * (size_t) (last_n > 0 ? last_n : 1), as_stream(st), logits, V, ctx,
                                         ctx_n, tok, last_n, repeat, freq, present, bias_tok, bias_val, bias_n);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_logit_adjust: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_logit_adjust");
    return FNX_OK;
}

extern "C" int fnx_embed_rows(const void* table_f16, const int* tok, int T, int H, float* R, fnx_stream st) {
    FNX_REQUIRE(table_f16 && tok && R && T >= 1, "fnx_embed_rows: bad arguments");
    {
        const cudaError_t le_ = launch_dep(true, k_embed_rows, dim3(dim3((H + 255) / 256, T)), dim3(256), 0, as_stream(st), (const __half*) table_f16, tok, H, R);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_embed_rows: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_embed_rows");
    return FNX_OK;
}

// The draft layer's input rows (the step of mtp_enqueue that no other layer has, engine/src/engine.cu:2103-2113):
// R[t] = fc_hid . rmsnorm(h[t]) * hnorm  +  fc_emb . rmsnorm(table[tok[t]]) * enorm.  The embedding rows pass through emb.
extern "C" int fnx_mtp_input(const void* fc_hid, const void* fc_emb, const void* table_f16, const float* hnorm, const float* enorm, float eps,
                             const float* h, int ldh, const int* tok, int T, int H, float* emb, float* R, unsigned* err, fnx_stream st) {
    FNX_REQUIRE(fc_hid && fc_emb && table_f16 && hnorm && enorm && h && tok && emb && R, "fnx_mtp_input: null pointer");
    FNX_REQUIRE(T >= 1 && ldh >= H, "fnx_mtp_input: %d rows, row stride %d for %d columns", T, ldh, H);
    FNX_TRY(fnx_embed_rows(table_f16, tok, T, H, emb, st));
    const int per = fnx_dense_rows(H);
    for (int t0 = 0; t0 < T; t0 += per) {
        const int nt = T - t0 < per ? T - t0 : per;
        FNX_TRY(fnx_dense(fc_hid, H, H, h + (size_t) t0 * ldh, ldh, nt, hnorm, eps, R + (size_t) t0 * H, H, 0, err, st));
    }
    for (int t0 = 0; t0 < T; t0 += per) {
        const int nt = T - t0 < per ? T - t0 : per;
        FNX_TRY(fnx_dense(fc_emb, H, H, emb + (size_t) t0 * H, H, nt, enorm, eps, R + (size_t) t0 * H, H, 1, err, st));
    }
    return FNX_OK;
}

extern "C" int fnx_rmsnorm(const float* x, const float* w, float* y, int rows, int n, float eps, fnx_stream st) {
    FNX_REQUIRE(x && w && y && rows >= 1 && n >= 1, "fnx_rmsnorm: bad arguments");
    {
        const cudaError_t le_ = launch_dep(true, k_rmsnorm, dim3(rows), dim3(256), 0, as_stream(st), x, w, y, n, eps);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_rmsnorm: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_rmsnorm");
    return FNX_OK;
}
