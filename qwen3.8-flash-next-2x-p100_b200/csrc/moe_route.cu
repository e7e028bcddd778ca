// MoE routing and combine.
//
// fnx_router_route replaces router_route / k_router_route (engine/src/kernels.hpp:294-296, engine/src/moe.cuh:258-515)
// and its simple form route / k_topk + k_jobs (engine/src/kernels.cu:338-398): router logits (f32 weights, fixed summation order), the
// top K per row with their renormalised softmax, the job list.  fnx_moe_combine replaces k_combine (engine/src/kernels.cu:412-419).
#include <algorithm>

#include <cooperative_groups.h>

#include "fnx_common.cuh"
#include <cstdlib>

#include "moe_route.cuh"
#include "nat_image.cuh"

namespace cg = cooperative_groups;

namespace fnxb {

// ---- the window form, in two launches: the logits over the whole chip, then one block that picks and lists the jobs (with programmatic
// launch the second costs about 1.3 us; an arrival counter and fences inside the first cost more).
//
// Block = ROWS expert rows, warp = one 256-column slice of all of them, lane = 8 consecutive columns (so that a warp holds a block
// of the rows' image in the quantiser's order): a row's slice feeds ROWS x 8 products per lane straight from registers.  TOK rows
// at a time make TOK x ROWS = 32 sums per lane, which cross the warp by halving (31 shuffles: lane i ends with sum i); the slices
// are then added in double.  A row's logits do not depend on the rows it comes with, nor on ROWS.  Everything that depends on no
// other kernel (the weights, the norm weights) is loaded before the rows are waited for.  f32 products and sums.
// Windows: 4 expert rows a block (129 blocks), block y = 0 of block column t also leaves row t's image (nat_image.cuh) for the experts'
// products; bound by the rows' way to every block (T x 8 KB each) and latency: 5 rows 14 -> 4.5 us, 20 rows 34 -> 10 us (with the pick
// 10 and 20), when one launch did both, eight rows at a time through shared memory.  Prompts: k_router_tiles below.
constexpr int RT_ROWS = 4;

template <int ROWS, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_router_logits(const float* __restrict__ Wr, const float* __restrict__ x, const float* __restrict__ norm_w, float eps, int T,
                                                          int E, int H, float* __restrict__ logits, unsigned* __restrict__ err, uint8_t* __restrict__ img) {
    constexpr int TOK = 32 / ROWS;
    extern __shared__ float sm[];                 // two buffers of psum [warps][32], ss [warps][TOK]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, NW = H / 256;
    const int row0 = blockIdx.x * ROWS, c = warp * 256 + lane * 8;
    float w[ROWS][8], nw[8];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (row0 + r <= E) {
            const float4* p = reinterpret_cast<const float4*>(Wr + (size_t) (row0 + r) * H + c);
            a = __ldg(p);
            b = __ldg(p + 1);
        }
        w[r][0] = a.x; w[r][1] = a.y; w[r][2] = a.z; w[r][3] = a.w;
        w[r][4] = b.x; w[r][5] = b.y; w[r][6] = b.z; w[r][7] = b.w;
    }
    if (norm_w) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(norm_w + c)), b = __ldg(reinterpret_cast<const float4*>(norm_w + c) + 1);
        nw[0] = a.x; nw[1] = a.y; nw[2] = a.z; nw[3] = a.w;
        nw[4] = b.x; nw[5] = b.y; nw[6] = b.z; nw[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) nw[i] = 1.0f;
    }
    pdl_wait();
    pdl_launch_dependents();
    constexpr int LD = THREADS <= 256 ? TOK : 4;   // rows whose loads are in flight together
    float4 xa[LD], xb[LD];
    auto fetch = [&](int t) {
#pragma unroll
        for (int i = 0; i < LD; ++i) {
            xa[i] = xb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t + i < T) {
                const float4* p = reinterpret_cast<const float4*>(x + (size_t) (t + i) * H + c);
                xa[i] = p[0];
                xb[i] = p[1];
            }
        }
    };
    constexpr bool AHEAD = THREADS <= 256;   // the next rows' loads run under the products (where the registers allow)
    if (AHEAD) fetch(0);
    int buf = 0;
    for (int t0 = 0; t0 < T; t0 += TOK, buf ^= 1) {
        float v[32];   // sum t ROWS + r
        float sq[TOK];
#pragma unroll
        for (int h = 0; h < TOK; h += LD) {
            if (!AHEAD) fetch(t0 + h);
            float e[LD][8];
#pragma unroll
            for (int t = 0; t < LD; ++t) {
                e[t][0] = xa[t].x; e[t][1] = xa[t].y; e[t][2] = xa[t].z; e[t][3] = xa[t].w;
                e[t][4] = xb[t].x; e[t][5] = xb[t].y; e[t][6] = xb[t].z; e[t][7] = xb[t].w;
            }
            if (AHEAD) fetch(t0 + h + LD);
#pragma unroll
            for (int t = 0; t < LD; ++t) {
                float ss = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    ss = fmaf(e[t][i], e[t][i], ss);
                    e[t][i] *= nw[i];
                }
                sq[h + t] = ss;
                if (img && t0 + h + t == (int) blockIdx.x && t0 + h + t < T) ni_quant(img, NW, e[t], norm_w ? ss : 0.f, t0 + h + t, warp, lane);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    float s = 0.f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) s = fmaf(w[r][i], e[t][i], s);
                    v[(h + t) * ROWS + r] = s;
                }
            }
        }
        // 32 sums over 32 lanes: at step o a lane keeps the half of its values whose index has the bit its lane number has
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
#pragma unroll
        for (int o = TOK / 2; o >= 1; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float keep = up ? sq[i + o] : sq[i], give = up ? sq[i] : sq[i + o];
                sq[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        float ss = sq[0];
#pragma unroll
        for (int o = TOK; o < 32; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        float* psum = sm + buf * NW * (32 + TOK);
        float* sqs = psum + NW * 32;
        psum[warp * 32 + lane] = v[0];
        if (lane < TOK) sqs[warp * TOK + lane] = ss;
        __syncthreads();   // (the buffers alternate: the last readers of this one passed the barrier of the step between)
        if (tid < 32) {
            const int t = tid / ROWS, r = tid % ROWS;
            double sd = 0.0, q = 0.0;   // (a handful of additions: the slices' own rounding is what the logits keep)
            for (int j = 0; j < NW; ++j) {
                sd += (double) psum[j * 32 + tid];
                q += (double) sqs[j * TOK + t];
            }
            float s = (float) sd;
            if (norm_w) s *= rsqrtf((float) q / (float) H + eps);
            if (t0 + t < T && row0 + r <= E) {
                logits[(size_t) (t0 + t) * (E + 1) + row0 + r] = s;
                if (!isfinite(s)) atomicOr(err, (unsigned) FNX_ERR_NONFINITE);
            }
        }
    }
}

// ---- the prompt form: blocks of 16 expert rows whose weights stay in registers, 16 rows of the prompt at a time, on mma.sync.m16n8k8 in
// tf32.  Both operands are split into a high part (the nearest 11 bits) and the 11 bits below it; high x high, high x low and low x
// high keep the products good to 2^-22, as f32 does; sums of 16 columns go on in f32 (the tensor core's own sums are cut off, not rounded:
// over 64 columns the logits came out up to 1.2e-6 small), those of the 128-column slices in double.  Warp = one slice; lane q of a quad holds columns 4 q .. 4 q + 3 of every 16 (the order of columns within a product is
// free), so rows and weights are loaded 16 bytes at a time; two pieces of the rows are in flight, across row tiles.
// Bound by the rows' way to the blocks (33 blocks read each: 128 KB a tile, two thirds of what an SM gets from L2), close behind by the splits
// (integer-logic pipe) and the products.  333 rows x 513 x 2,048: 29 us (11 TFLOP/s of f32 products; 13 us at L2's 6.5 TB/s); f32 products with
// their 31 shuffles per two rows took 53.
// CL = 2: rows of more than 2,048 columns, each half of them in one block of a pair; each block completes half of the sums, reading
// the other's slices through distributed shared memory.  (900 rows x 513 x 4,096: 181 us; k_router_logits over blocks of 32 rows 292, a walk of every
// expert row by blocks of eight rows 225.)
constexpr int RP_ROWS = 16, RP_TOK = 16, RP_SLICE = 128, RP_IT = RP_SLICE / 16, RP_AHEAD = 2, RP_LD = 20, RP_WARPS = 2048 / RP_SLICE;

__device__ __forceinline__ void rp_split(float v, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(v) + 0x1000u) & 0xFFFFE000u;
    lo = __float_as_uint(v - __uint_as_float(hi)) & 0xFFFFE000u;
}
__device__ __forceinline__ void rp_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(RP_WARPS * 32, 1) k_router_tiles(const float* __restrict__ Wr, const float* __restrict__ x, const float* __restrict__ norm_w, float eps, int T, int E,
                                                         int H, float* __restrict__ logits, unsigned* __restrict__ err) {
    __shared__ __align__(16) float psum_[2][RP_WARPS][RP_TOK][RP_LD];
    __shared__ float sqs_[2][RP_WARPS][RP_TOK];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, NW = H / RP_SLICE / CL;
    const int half = CL > 1 ? (int) blockIdx.x % CL : 0, row0 = (int) blockIdx.x / CL * RP_ROWS, c = (half * NW + warp) * RP_SLICE + q * 4, tiles = (T + RP_TOK - 1) / RP_TOK;
    float4 w[2][RP_IT];   // times the norm weights
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const bool live = row0 + 8 * j + g <= E;
        const float* p = Wr + (size_t) (live ? row0 + 8 * j + g : 0) * H + c;
#pragma unroll
        for (int i = 0; i < RP_IT; ++i) w[j][i] = live ? __ldg(reinterpret_cast<const float4*>(p + 16 * i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (norm_w) {
#pragma unroll
        for (int i = 0; i < RP_IT; ++i) {
            const float4 n = __ldg(reinterpret_cast<const float4*>(norm_w + c + 16 * i));
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                w[j][i].x *= n.x; w[j][i].y *= n.y; w[j][i].z *= n.z; w[j][i].w *= n.w;
            }
        }
    }
    pdl_wait();
    pdl_launch_dependents();
    // (rows past the last one repeat it: their sums are not written)
    auto row_of = [&](int tile, int h) { return x + (size_t) min(tile * RP_TOK + g + 8 * h, T - 1) * H + c; };
    int tile = blockIdx.y;
    const float *p0 = row_of(tile, 0), *p1 = row_of(tile, 1);
    float4 xa[RP_AHEAD], xb[RP_AHEAD];
#pragma unroll
    for (int i = 0; i < RP_AHEAD; ++i) {
        xa[i] = *reinterpret_cast<const float4*>(p0 + 16 * i);
        xb[i] = *reinterpret_cast<const float4*>(p1 + 16 * i);
    }
    for (int buf = 0; tile < tiles; tile += gridDim.y, buf ^= 1) {
        const int next = min(tile + (int) gridDim.y, tiles - 1);
        const float *n0 = row_of(next, 0), *n1 = row_of(next, 1);
        float sum[2][4] = {}, hl[2][4] = {}, ss0 = 0.f, ss1 = 0.f;
#pragma unroll
        for (int i0 = 0; i0 < RP_IT; i0 += RP_AHEAD) {
#pragma unroll
            for (int k = 0; k < RP_AHEAD; ++k) {
                float hh[2][4] = {};
                const int i = i0 + k;
                const float a[4] = {xa[k].x, xa[k].y, xa[k].z, xa[k].w}, b[4] = {xb[k].x, xb[k].y, xb[k].z, xb[k].w};
                const int ni = i + RP_AHEAD;
                xa[k] = *reinterpret_cast<const float4*>((ni < RP_IT ? p0 : n0) + 16 * (ni % RP_IT));
                xb[k] = *reinterpret_cast<const float4*>((ni < RP_IT ? p1 : n1) + 16 * (ni % RP_IT));
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    ss0 = fmaf(a[e], a[e], ss0);
                    ss1 = fmaf(b[e], b[e], ss1);
                }
#pragma unroll
                for (int st = 0; st < 2; ++st) {
                    uint32_t ah[4], al[4];
                    rp_split(a[2 * st], ah[0], al[0]);
                    rp_split(b[2 * st], ah[1], al[1]);
                    rp_split(a[2 * st + 1], ah[2], al[2]);
                    rp_split(b[2 * st + 1], ah[3], al[3]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        uint32_t bh0, bl0, bh1, bl1;
                        float w0 = st ? w[j][i].z : w[j][i].x, w1 = st ? w[j][i].w : w[j][i].y;
                        asm volatile("" : "+f"(w0), "+f"(w1));   // (split here: split before the loop they would live in local memory)
                        rp_split(w0, bh0, bl0);
                        rp_split(w1, bh1, bl1);
                        rp_mma(hh[j], ah, bh0, bh1);
                        rp_mma(hl[j], ah, bl0, bl1);
                        rp_mma(hl[j], al, bh0, bh1);
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[j][e] += hh[j][e];
            }
        }
        ss0 += __shfl_xor_sync(0xffffffffu, ss0, 1);
        ss1 += __shfl_xor_sync(0xffffffffu, ss1, 1);
        ss0 += __shfl_xor_sync(0xffffffffu, ss0, 2);
        ss1 += __shfl_xor_sync(0xffffffffu, ss1, 2);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            *reinterpret_cast<float2*>(&psum_[buf][warp][g][8 * j + 2 * q]) = make_float2(sum[j][0] + hl[j][0], sum[j][1] + hl[j][1]);
            *reinterpret_cast<float2*>(&psum_[buf][warp][g + 8][8 * j + 2 * q]) = make_float2(sum[j][2] + hl[j][2], sum[j][3] + hl[j][3]);
        }
        if (q == 0) {
            sqs_[buf][warp][g] = ss0;
            sqs_[buf][warp][g + 8] = ss1;
        }
        // (the buffers alternate: the last readers of this one passed the barrier of the tile between)
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
        for (int o = half * (RP_TOK * RP_ROWS / CL) + tid; o < (half + 1) * (RP_TOK * RP_ROWS / CL); o += NW * 32) {
            const int t = o / RP_ROWS, r = o % RP_ROWS;
            double sd = 0.0, sq = 0.0;
#pragma unroll
            for (int k = 0; k < CL; ++k) {
                const float* ps = &psum_[buf][0][t][r];
                const float* qs = &sqs_[buf][0][t];
                if constexpr (CL > 1) {
                    ps = cg::this_cluster().map_shared_rank(ps, k);
                    qs = cg::this_cluster().map_shared_rank(qs, k);
                }
                for (int j = 0; j < NW; ++j) {
                    sd += (double) ps[j * RP_TOK * RP_LD];
                    sq += (double) qs[j * RP_TOK];
                }
            }
            float s = (float) sd;
            if (norm_w) s *= rsqrtf((float) sq / (float) H + eps);
            if (tile * RP_TOK + t < T && row0 + r <= E) {
                logits[(size_t) (tile * RP_TOK + t) * (E + 1) + row0 + r] = s;
                if (!isfinite(s)) atomicOr(err, (unsigned) FNX_ERR_NONFINITE);
            }
        }
        p0 = n0;
        p1 = n1;
    }
    if constexpr (CL > 1) cg::this_cluster().sync();   // no block may leave while the other still reads its sums
}

// the logits of T rows; windows (img may be given) or prompts
static int router_logits(const float* Wr, const float* x, const float* norm_w, float eps, int T, int E, int H, float* logits, unsigned* err, uint8_t* img, bool early,
                         cudaStream_t st) {
    const int NW = H / 256;
    cudaError_t le;
    if (T <= FNX_MAX_ROWS) {
        const int blocks = (E + RT_ROWS) / RT_ROWS;
        le = launch_dep(early, H <= 2048 ? k_router_logits<RT_ROWS, 256> : k_router_logits<RT_ROWS, 512>,
                        dim3(img && blocks < T ? T : blocks), dim3(NW * 32), (size_t) 2 * NW * (32 + 32 / RT_ROWS) * sizeof(float), st, Wr,
                        x, norm_w, eps, T, E, H, logits, err, img);
    } else {
        const int cl = H > RP_WARPS * RP_SLICE ? 2 : 1, blocks = (E + RP_ROWS) / RP_ROWS * cl, tiles = (T + RP_TOK - 1) / RP_TOK, fit = std::max(1, sm_count() / blocks);
        le = launch_dep(early, cl > 1 ? k_router_tiles<2> : k_router_tiles<1>, dim3(blocks, std::min(tiles, fit)), dim3(H / RP_SLICE / cl * 32), 0, st, Wr, x, norm_w, eps, T, E, H, logits,
                        err);
    }
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_router_logits: launch failed: %s", cudaGetErrorString(le));
}

// One block: the top K of every row (a warp per row), their weights, and the job list, built in shared memory and copied out.  Bound by latency (the
// launch, the logits' way, the ranks, four barriers): eight warps where they are enough, whose barriers cost less, what does not depend on the logits
// before they are waited for (one row and five: 5.5 us a launch with 32 warps that cleared the list behind the picks, 4.3 now.  A list without scans
// over the block, each entry placed by the bits of a map below its expert's: 3.9 and 4.3, 0.4% of a pass of one row).
template <int NTH>
__global__ void __launch_bounds__(NTH) k_router_pick(const float* __restrict__ logits, int T, int E, int K, int e_lo, int e_hi, int add_shared, int* __restrict__ topi,
                                                     float* __restrict__ topw, fnx_job* __restrict__ jobs, int* __restrict__ njobs,
                                                     unsigned long long* __restrict__ stats) {
    extern __shared__ __align__(16) uint8_t pick_smem[];   // the job list
    __shared__ int s_topi[FNX_MAX_ROWS * 32];
    __shared__ unsigned s_rows[RT_MAXE];
    __shared__ int s_base[RT_MAXE], wsum_[32], total_[2];
    __shared__ __align__(16) unsigned scr_[NTH / 32][64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    RtJobSmem js;
    js.s_topi = s_topi; js.s_rows = s_rows; js.s_base = s_base; js.wsum = wsum_; js.total = total_;
    js.js = reinterpret_cast<fnx_job*>(pick_smem);
    rt_clear_jobs<NTH>(js, tid, T, K);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    for (int t = warp; t < T; t += NTH / 32) {
        const float* l = logits + (size_t) t * (E + 1);
        int* ti = topi + t * K;
        float* tw = topw + t * K;
        if (E <= 512) rt_topk_row<16>(l, E, K, lane, scr_[warp], ti, s_topi + t * K, tw, nullptr);
        else rt_topk_row<RT_MAXE / 32>(l, E, K, lane, scr_[warp], ti, s_topi + t * K, tw, nullptr);
        rt_note_picks(js, t, K, e_lo, e_hi, lane);
    }
    rt_build_jobs<NTH>(js, tid, T, E, K, e_lo, e_hi, add_shared);
    const int total = total_[0];
    if (tid == 0) {
        njobs[0] = total;
        if (stats) {
            atomicAdd(&stats[0], (unsigned long long) total_[1]);
            atomicAdd(&stats[1], 1ull);
        }
    }
    constexpr int JW = sizeof(fnx_job) / 4;
    for (int w = tid; w < total * JW; w += NTH) reinterpret_cast<int*>(jobs)[w] = reinterpret_cast<const int*>(js.js)[w];
}

int router_window(const float* Wr, const float* x, const float* norm_w, float eps, int T, int E, int H, int K, int e_lo, int e_hi, int add_shared, float* logits, int* topi,
                  float* topw, fnx_job* jobs, int* njobs, unsigned long long* stats, unsigned* err, uint8_t* img, bool early, cudaStream_t st) {
    FNX_TRY(router_logits(Wr, x, norm_w, eps, T, E, H, logits, err, img, early, st));
    const size_t smem = ((size_t) T * K + (T + FNX_JOB_TOK - 1) / FNX_JOB_TOK) * sizeof(fnx_job);
    const int threads = T <= 8 ? 256 : 1024;   // a warp per row
    auto kernel = T <= 8 ? k_router_pick<256> : k_router_pick<1024>;
    if (int rc = set_smem_limit((const void*) kernel, 64 * 1024)) return rc;
    const cudaError_t le = launch_dep(true, kernel, dim3(1), dim3(threads), smem, st, (const float*) logits, T, E, K, e_lo, e_hi, add_shared, topi, topw, jobs, njobs, stats);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_router_pick: launch failed: %s", cudaGetErrorString(le));
}

// one warp per row: the top K of its E logits and their renormalised softmax weights
__global__ void __launch_bounds__(256) k_topk_rows(const float* __restrict__ logits, int T, int E, int K, int* __restrict__ topi, float* __restrict__ topw) {
    pdl_begin();
    __shared__ __align__(16) unsigned scr_[8][64];
    const int warp = threadIdx.x >> 5, t = blockIdx.x * 8 + warp, lane = threadIdx.x & 31;
    if (t >= T) return;
    const float* l = logits + (size_t) t * (E + 1);
    if (E <= 512) rt_topk_row<16>(l, E, K, lane, scr_[warp], topi + (size_t) t * K, nullptr, topw + (size_t) t * K, nullptr);
    else rt_topk_row<RT_MAXE / 32>(l, E, K, lane, scr_[warp], topi + (size_t) t * K, nullptr, topw + (size_t) t * K, nullptr);
}

// Every load leaves at once: the picks' ids and weights, and every addend whether its pick counts or not (where it does not, nobody wrote the addend: nothing of
// it enters the sum).  Bound by latency: five rows of ten picks 2.6 us a launch, 3.8 where the addends wait for the weights; 32 rows 3.7 and 4.7; the block of
// four launches and this one, five rows, 48.5 us (without a look at the ids 48.1).  With the weights by a warp's lanes a launch among its like takes 2.4, but
// behind a product the block takes 50.5.
__global__ void k_combine(const float* __restrict__ part, const int* __restrict__ topi, const float* __restrict__ topw,
                          const float* __restrict__ logits, int T, int E, int H, int K, int e_lo, int e_hi, int add_shared,
                          float* __restrict__ out, int accumulate) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= H) return;
    float w[32], v[32];
    int id[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        w[k] = v[k] = 0.f;
        id[k] = -1;
        if (k < K) {
            w[k] = topw[t * K + k];
            id[k] = topi[t * K + k];
            v[k] = part[((size_t) t * K + k) * H + i];
        }
    }
    const float shv = add_shared ? part[((size_t) T * K + t) * H + i] : 0.f;
    const float shl = add_shared ? logits[(size_t) t * (E + 1) + E] : 0.f;
    float* o = out + (size_t) t * H + i;
    const float prev = accumulate ? *o : 0.f;
    asm volatile("" ::: "memory");   // (no load behind this)
    // the addends are summed as 2^-32 fixed-point integers: the sum does not depend on their order, so a row's result does not
    // depend on how its picks are split over kernels or expert-parallel ranks
    const unsigned span = (unsigned) max(e_hi - e_lo, 0);
    unsigned long long s = 0ull;
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (k < K && (unsigned) id[k] - (unsigned) e_lo < span && w[k] != 0.f) s += fix_from_float(w[k] * v[k]);
    if (add_shared) s += fix_from_float(sigmoidf_(shl) * shv);
    *o = prev + fix_to_float(s);
}

// k_combine that also leaves the new rows' image for the next dense product (fnx_dense_image): one warp per (256-column block,
// row), the lane's 8 columns of every addend in flight at once; the sums and the residual update are k_combine's, the image
// cells are those the dense kernel's own quantisation (quant_finish) makes of the same values, so the product's bits do not
// change.  The blocks of an image's last live row also clear the rows of its last group that hold nothing.
__global__ void __launch_bounds__(32) k_combine_image(const float* __restrict__ part, const int* __restrict__ topi, const float* __restrict__ topw,
                                                      const float* __restrict__ logits, int T, int E, int H, int K, float* __restrict__ out,
                                                      uint8_t* __restrict__ img_out, const float* __restrict__ img_norm_w, size_t img_stride) {
    pdl_wait();
    pdl_launch_dependents();
    const int blk = blockIdx.x, t = blockIdx.y, lane = threadIdx.x, KB = H / 256;
    const size_t col = (size_t) blk * 256 + lane * 8;
    const float mw = Pick(topi + t * K, topw + t * K, K, lane).weight(0, E);
    float w[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) w[k] = __shfl_sync(0xffffffffu, mw, k);
    const float shl = logits[(size_t) t * (E + 1) + E];
    QuantTask q[1];
    float v[1][8], nw[1][8];
    q[0].src = out + (size_t) t * H + (size_t) blk * 256;
    q[0].t = t % FNX_DENSE_ROWS;
    q[0].blk = blk;
    quant_fetch(q[0], img_norm_w, lane, v[0], nw[0]);   // the old values and the norm weights
    unsigned long long s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0ull;
    // the addends in two halves of up to 16 picks, all of a half's loads in flight at once
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 16) {
        if (k0 >= K) break;
        float4 a[16][2];
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (k0 + k < K) {
                const float4* src = reinterpret_cast<const float4*>(part + ((size_t) t * K + k0 + k) * H + col);
                a[k][0] = src[0];
                a[k][1] = src[1];
            }
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (k0 + k < K && w[k0 + k] != 0.f) {
                const float wk = w[k0 + k];
                const float e8[8] = {a[k][0].x, a[k][0].y, a[k][0].z, a[k][0].w, a[k][1].x, a[k][1].y, a[k][1].z, a[k][1].w};
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] += fix_from_float(wk * e8[i]);
            }
    }
    {
        const float4* src = reinterpret_cast<const float4*>(part + ((size_t) T * K + t) * H + col);
        const float4 a0 = src[0], a1 = src[1];
        const float g = sigmoidf_(shl);
        const float e8[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += fix_from_float(g * e8[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[0][i] += fix_to_float(s[i]);
    float* dst = out + (size_t) t * H + col;
    *reinterpret_cast<float4*>(dst) = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(v[0][4], v[0][5], v[0][6], v[0][7]);
    // the image of the row's group of FNX_DENSE_ROWS
    const int t0 = t - t % FNX_DENSE_ROWS, nt = min((int) FNX_DENSE_ROWS, T - t0), NG = (nt + 3) / 4;
    uint2* cells = reinterpret_cast<uint2*>(img_out + (size_t) (t0 / FNX_DENSE_ROWS) * img_stride);
    float* scales = reinterpret_cast<float*>(cells + (size_t) NG * (H / 32) * 32);
    float* rs = scales + (size_t) NG * KB * 8;
    quant_finish(q, v, nw, H, img_norm_w, cells, scales, rs, lane);
    if (t == t0 + nt - 1)
        for (int td = nt; td < 4 * NG; ++td) {
            const int ng = td >> 2, n = td & 3;
            for (int i = lane; i < 64; i += 32) {   // (sub-block of the column block, level, q)
                const int sbG = blk * 8 + (i >> 3), lvl = (i >> 2) & 1, qq = i & 3;
                cells[((size_t) (ng * (H / 32) + sbG) * 8 + n + 4 * lvl) * 4 + qq] = make_uint2(0u, 0u);
            }
            if (lane < 2) scales[(size_t) (ng * KB + blk) * 8 + n + 4 * lane] = 0.f;
            if (lane == 2) rs[td * 16 + blk] = 0.f;
        }
}

// k_combine for an engine's window: the new rows' image (nat_image.cuh) for the next projection rides along.  One block per (256-column
// block, row): four warps share out the addends (integers: their order does not show), eight columns a lane, and the first one finishes.  Bound by latency: the
// launch, one way to memory, 24 conversions to 64-bit integers a lane (a warp alone had 88 of them, and the norm weights' way on top: 4.4 us a launch for one row and for five, 2.8 and 2.4 now).
constexpr int CN_WARPS = 4, CN_LD = 3;   // addends in flight a warp
__global__ void __launch_bounds__(CN_WARPS * 32) k_combine_nat(const float* __restrict__ part, const float* __restrict__ topw, const float* __restrict__ logits, int T, int E, int H,
                                                               int K, float* __restrict__ out, uint8_t* __restrict__ img, const float* __restrict__ img_norm_w) {
    __shared__ unsigned long long sums[CN_WARPS - 1][8][32];
    const int blk = blockIdx.x, t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, KB = H / 256;
    const size_t col = (size_t) blk * 256 + lane * 8;
    // ahead of the wait: the rows (last written by the output projection), the router's results (by the kernels before the two expert products), weights
    float* dst = out + (size_t) t * H + col;
    float v[8], nw[8];
    if (warp == 0) {
        const float4 o0 = *reinterpret_cast<const float4*>(dst), o1 = *reinterpret_cast<const float4*>(dst + 4);
        const float4 w0 = *reinterpret_cast<const float4*>(img_norm_w + col), w1 = *reinterpret_cast<const float4*>(img_norm_w + col + 4);
        v[0] = o0.x; v[1] = o0.y; v[2] = o0.z; v[3] = o0.w; v[4] = o1.x; v[5] = o1.y; v[6] = o1.z; v[7] = o1.w;
        nw[0] = w0.x; nw[1] = w0.y; nw[2] = w0.z; nw[3] = w0.w; nw[4] = w1.x; nw[5] = w1.y; nw[6] = w1.z; nw[7] = w1.w;
    }
    const float mw = lane < K ? topw[t * K + lane] : 0.f, g = sigmoidf_(logits[(size_t) t * (E + 1) + E]);
    pdl_wait();
    pdl_launch_dependents();
    unsigned long long s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0ull;
    for (int k0 = warp; k0 <= K; k0 += CN_LD * CN_WARPS) {   // (addend K: the shared expert's)
        float4 a[CN_LD][2];
#pragma unroll
        for (int j = 0; j < CN_LD; ++j) {
            const int k = k0 + j * CN_WARPS;
            if (k <= K) {
                const float4* src = reinterpret_cast<const float4*>(part + (k < K ? (size_t) t * K + k : (size_t) T * K + t) * H + col);
                a[j][0] = src[0];
                a[j][1] = src[1];
            }
        }
#pragma unroll
        for (int j = 0; j < CN_LD; ++j) {
            const int k = k0 + j * CN_WARPS;
            if (k <= K) {
                const float pick = __shfl_sync(0xffffffffu, mw, k & 31), wk = k < K ? pick : g;
                const float e8[8] = {a[j][0].x, a[j][0].y, a[j][0].z, a[j][0].w, a[j][1].x, a[j][1].y, a[j][1].z, a[j][1].w};
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] += fix_from_float(wk * e8[i]);
            }
        }
    }
    if (warp) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sums[warp - 1][i][lane] = s[i];
    }
    __syncthreads();
    if (warp) return;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int w = 0; w < CN_WARPS - 1; ++w) s[i] += sums[w][i][lane];
        v[i] += fix_to_float(s[i]);
    }
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        ss = fmaf(v[i], v[i], ss);
        v[i] *= nw[i];
    }
    ni_quant(img, KB, v, ss, t, blk, lane);
}

int moe_combine_nat(const float* part, const float* topw, const float* logits, int T, int E, int H, int K, float* R, uint8_t* img, const float* img_norm_w,
                    cudaStream_t st) {
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS && K >= 1 && K <= 32 && H % 256 == 0, "moe_combine_nat: %d rows of %d, top %d", T, H, K);
    const cudaError_t le = launch_dep(true, k_combine_nat, dim3(H / 256, T), dim3(CN_WARPS * 32), 0, st, part, topw, logits, T, E, H, K, R, img, img_norm_w);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_combine_nat: launch failed: %s", cudaGetErrorString(le));
}

}  // namespace fnxb

using namespace fnxb;

extern "C" int fnx_router_route(const float* Wr, const float* x, const float* norm_w, float eps, int T, int E, int H, int K, int e_lo,
                                int e_hi, int add_shared, float* logits, int* topi, float* topw, fnx_job* jobs, int* njobs,
                                unsigned long long* stats, unsigned* err, fnx_stream st) {
    FNX_REQUIRE(Wr && x && logits && topi && topw && jobs && njobs && err, "fnx_router_route: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS, "fnx_router_route: %d rows (1..%d)", T, FNX_MAX_ROWS);
    FNX_REQUIRE(E >= K && E <= RT_MAXE && K >= 1 && K <= 32, "fnx_router_route: %d experts, top %d not supported", E, K);
    FNX_REQUIRE(H % 256 == 0 && H <= 4096, "fnx_router_route: hidden %d not supported", H);
    FNX_REQUIRE(0 <= e_lo && e_lo <= e_hi && e_hi <= E, "fnx_router_route: expert range [%d, %d) outside [0, %d)", e_lo, e_hi, E);
    FNX_REQUIRE(((uintptr_t) x & 15) == 0 && ((uintptr_t) Wr & 15) == 0 && ((uintptr_t) norm_w & 15) == 0, "fnx_router_route: 16-byte alignment");
    return router_window(Wr, x, norm_w, eps, T, E, H, K, e_lo, e_hi, add_shared, logits, topi, topw, jobs, njobs, stats, err, nullptr, false, as_stream(st));
}

extern "C" int fnx_moe_combine(const float* part, const int* topi, const float* topw, const float* logits, int T, int E, int H, int K,
                               int e_lo, int e_hi, int add_shared, float* out, int accumulate, fnx_stream st) {
    FNX_REQUIRE(part && topi && topw && logits && out, "fnx_moe_combine: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS, "fnx_moe_combine: %d rows", T);
    {
        const cudaError_t le_ = launch_dep(true, k_combine, dim3((H + 255) / 256, T), dim3(256), 0, as_stream(st), part, topi, topw, logits, T, E, H, K, e_lo, e_hi, add_shared, out, accumulate);
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_combine: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_moe_combine");
    return FNX_OK;
}

extern "C" int fnx_moe_experts(const void* Wgu, size_t gu_stride, const void* Wdn, size_t dn_stride, int e_base, const void* Wsh_gu, const void* Wsh_dn,
                               const fnx_job* jobs, const int* njobs, int njobs_max, const int* topi, const float* topw, const float* logits, const float* x,
                               const float* norm_w, float eps, int T, int E, int H, int F, int K, int e_lo, int e_hi, int add_shared, float* h, float* part, float* out,
                               unsigned* err, fnx_stream st) {
    FNX_TRY(fnx_moe_gate_up(Wgu, gu_stride, e_base, Wsh_gu, E, jobs, njobs, njobs_max, x, norm_w, eps, H, F, h, err, st));
    FNX_TRY(fnx_moe_down(Wdn, dn_stride, e_base, Wsh_dn, E, jobs, njobs, njobs_max, h, H, F, part, err, st));
    return fnx_moe_combine(part, topi, topw, logits, T, E, H, K, e_lo, e_hi, add_shared, out, 0, st);
}

extern "C" int fnx_moe_combine_image(const float* part, const int* topi, const float* topw, const float* logits, int T, int E, int H, int K, float* R,
                                     void* img_out, const float* img_norm_w, fnx_stream st) {
    FNX_REQUIRE(part && topi && topw && logits && R && img_out && img_norm_w, "fnx_moe_combine_image: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS && K >= 1 && K <= 32, "fnx_moe_combine_image: %d rows, top %d", T, K);
    FNX_REQUIRE(H == 256 || H == 512 || H == 1024 || H == 2048 || H == 4096, "fnx_moe_combine_image: hidden %d", H);
    FNX_REQUIRE(((uintptr_t) img_out & 15) == 0 && ((uintptr_t) R & 15) == 0 && ((uintptr_t) part & 15) == 0, "fnx_moe_combine_image: 16-byte alignment");
    {
        const cudaError_t le_ = launch_dep(true, k_combine_image, dim3(H / 256, T), dim3(32), 0, as_stream(st), part, topi, topw, logits, T, E, H, K, R, (uint8_t*) img_out,
                                         img_norm_w, fnx_dense_image_bytes(H));
        if (le_ != cudaSuccess) return fail(FNX_E_CUDA, "k_combine_image: launch failed: %s", cudaGetErrorString(le_));
    }
    FNX_LAUNCH_OK("fnx_moe_combine_image");
    return FNX_OK;
}

// ---- the router over a prompt's rows as a tensor-core product (gemm_tma.cu): the normed rows and the f32 weights are split
// into f16 high and low parts (weights times 256 first, so that their low parts stay clear of f16's subnormals); three
// products (high x high, high x low, low x high) restore the f32 operands (the tensor core's truncating f32 accumulation leaves
// the logits good to a few 1e-5).  The shared expert's gate row is a plain dot.
__global__ void __launch_bounds__(256) k_router_split_x(const float* __restrict__ x, const float* __restrict__ norm_w, const float* __restrict__ w_gate, int H,
                                                        float eps, __half* __restrict__ xh, __half* __restrict__ xl, float* __restrict__ logits, int ldl, int E) {
    pdl_begin();
    const int t = blockIdx.x, tid = threadIdx.x;
    const float* xr = x + (size_t) t * H;
    __shared__ float ws[8], s_r;
    float ss = 0.f;
    for (int i = tid * 4; i < H; i += 1024) {
        const float4 v = *reinterpret_cast<const float4*>(xr + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) ws[tid >> 5] = ss;
    __syncthreads();
    if (tid == 0) {
        float a = 0.f;
        for (int w = 0; w < 8; ++w) a += ws[w];
        s_r = norm_w ? rsqrtf(a / (float) H + eps) : 1.0f;
    }
    __syncthreads();
    const float r = s_r;
    float dot = 0.f;
    for (int i = tid * 4; i < H; i += 1024) {
        float4 v = *reinterpret_cast<const float4*>(xr + i);
        if (norm_w) {
            const float4 w = *reinterpret_cast<const float4*>(norm_w + i);
            v.x *= w.x * r; v.y *= w.y * r; v.z *= w.z * r; v.w *= w.w * r;
        }
        const float4 g = *reinterpret_cast<const float4*>(w_gate + i);
        dot = fmaf(v.x, g.x, fmaf(v.y, g.y, fmaf(v.z, g.z, fmaf(v.w, g.w, dot))));
        const float e[4] = {v.x, v.y, v.z, v.w};
        __half h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            h[k] = __float2half_rn(e[k]);
            l[k] = __float2half_rn(e[k] - __half2float(h[k]));
        }
        *reinterpret_cast<uint2*>(xh + (size_t) t * H + i) = make_uint2((uint32_t) __half_as_ushort(h[0]) | ((uint32_t) __half_as_ushort(h[1]) << 16),
                                                                        (uint32_t) __half_as_ushort(h[2]) | ((uint32_t) __half_as_ushort(h[3]) << 16));
        *reinterpret_cast<uint2*>(xl + (size_t) t * H + i) = make_uint2((uint32_t) __half_as_ushort(l[0]) | ((uint32_t) __half_as_ushort(l[1]) << 16),
                                                                        (uint32_t) __half_as_ushort(l[2]) | ((uint32_t) __half_as_ushort(l[3]) << 16));
    }
    dot = warp_sum(dot);
    __syncthreads();
    if ((tid & 31) == 0) ws[tid >> 5] = dot;
    __syncthreads();
    if (tid == 0) {
        float a = 0.f;
        for (int w = 0; w < 8; ++w) a += ws[w];
        logits[(size_t) t * ldl + E] = a;
    }
}

__global__ void k_router_split_w(const float* __restrict__ w, size_t n, __half* __restrict__ wh, __half* __restrict__ wl) {
    pdl_begin();
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = w[i] * 256.0f;
    const __half h = __float2half_rn(v);
    wh[i] = h;
    wl[i] = __float2half_rn(v - __half2float(h));
}

namespace fnxb {
int gemm_tma_launch(const __half* w, const __half* wl, const __half* x, const __half* xl, float* y, int ldy, int T, int rows, int K, int accumulate, float scale,
                    unsigned* err, cudaStream_t st);
static size_t rr_align(size_t v) { return (v + 255) & ~(size_t) 255; }
}  // namespace fnxb

extern "C" size_t fnx_router_rows_scratch_bytes(int T, int E, int H) {
    return 2 * rr_align((size_t) T * H * sizeof(__half)) + 2 * rr_align((size_t) E * H * sizeof(__half));
}

namespace fnxb {
// early: launch_dep's (the weights are read ahead)
int router_rows(const float* Wr, const float* x, const float* norm_w, float eps, int T, int E, int H, int K, float* logits, int* topi, float* topw, void* scratch,
                unsigned* err, bool early, cudaStream_t st) {
    FNX_REQUIRE(Wr && x && logits && topi && topw && err, "fnx_router_rows: null pointer");
    FNX_REQUIRE(T >= 1, "fnx_router_rows: %d rows", T);
    FNX_REQUIRE(E >= K && E <= RT_MAXE && K >= 1 && K <= 32, "fnx_router_rows: %d experts, top %d not supported", E, K);
    FNX_REQUIRE(H % 256 == 0 && H <= 4096, "fnx_router_rows: hidden %d not supported", H);
    static const bool gemm_off = []() { const char* e = getenv("FNX_PROMPT_GEMM"); return e && atoi(e) == 0; }();
    if (scratch && T >= 1024 && !gemm_off) {
        uint8_t* b = (uint8_t*) scratch;
        __half* xh = (__half*) b; b += rr_align((size_t) T * H * sizeof(__half));
        __half* xl = (__half*) b; b += rr_align((size_t) T * H * sizeof(__half));
        __half* wh = (__half*) b; b += rr_align((size_t) E * H * sizeof(__half));
        __half* wl = (__half*) b;
        FNX_CUDA_OK(launch_after(k_router_split_x, dim3(T), dim3(256), 0, st, x, norm_w, Wr + (size_t) E * H, H, eps, xh, xl, logits, E + 1, E));
        FNX_LAUNCH_OK("k_router_split_x");
        const size_t n = (size_t) E * H;
        FNX_CUDA_OK(launch_after(k_router_split_w, dim3((unsigned) ((n + 255) / 256)), dim3(256), 0, st, Wr, n, wh, wl));
        FNX_LAUNCH_OK("k_router_split_w");
        if (int rc = gemm_tma_launch(wh, wl, xh, xl, logits, E + 1, T, E, H, 0, 1.0f / 256.0f, err, st)) return rc;
    } else {
        FNX_TRY(router_logits(Wr, x, norm_w, eps, T, E, H, logits, err, nullptr, early, st));
    }
    FNX_CUDA_OK(launch_after(k_topk_rows, dim3((T + 7) / 8), dim3(256), 0, st, logits, T, E, K, topi, topw));
    FNX_LAUNCH_OK("k_topk_rows");
    return FNX_OK;
}
}  // namespace fnxb

extern "C" int fnx_router_rows(const float* Wr, const float* x, const float* norm_w, float eps, int T, int E, int H, int K, float* logits, int* topi,
                               float* topw, void* scratch, unsigned* err, fnx_stream st) {
    return router_rows(Wr, x, norm_w, eps, T, E, H, K, logits, topi, topw, scratch, err, false, as_stream(st));
}
