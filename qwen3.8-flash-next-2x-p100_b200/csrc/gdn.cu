// Gated DeltaNet core for a verify window, one launch.
//
// Replaces gdn_core / k_gdn_core (engine/src/kernels.hpp:97-99, engine/src/gdn_core.cuh:20-225; unfused statement
// engine/src/kernels.cu:422-506): conv4 + SiLU over the q|k|v channels, L2 norms of q and k, the gates, the delta
// rule on the fp32 state, the gated RMS norm of the output.  Differences by design:
//   - rows form a tree (parent[t]); row t starts from its parent's state and conv history, not from row t - 1's;
//   - the state after every row, and the history keeping it would leave, go to ring slot (*cur + 1 + t) % NS
//     instead of the snap / hsnap buffers, so that a commit is a change of *cur and copies nothing
//     (engine/src/engine_common.cu:710-754 copies the kept snapshot back);
//   - the four blocks that share a value head form a thread-block cluster and add up the head's square sums
//     through distributed shared memory, where the reference uses a global scratch buffer and atomic counters.
#include <cooperative_groups.h>

#include "gdn_core.h"
#include "nat_image.cuh"

namespace cg = cooperative_groups;

namespace fnxb {

constexpr int GDN_HS = 128, GDN_Q = 4, GDN_QC = GDN_HS / GDN_Q, GDN_THREADS = 2 * GDN_HS + GDN_QC, GDS_THREADS = 128;

// two f32 in a 64-bit register and the packed multiply-add on them (fma.rn.f32x2: each half rounded as the scalar fmaf is, so the
// products are those of the scalar form, at half the arithmetic instructions)
__device__ __forceinline__ uint64_t f2_pack(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t r, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// One block = a quarter (32 columns) of a value head; the four blocks of a head, and with an image the two heads of a 256-column
// block of it, form a cluster.  288 threads: one per conv channel the block needs (the head's q and k, its own v columns).  Four of the nine
// warps run the delta rule: a warp holds 8 columns of the state, lane = 8 rg + c: column c, key rows 16 j + 4 rg + i (j < 8, i < 4),
// so that a row's sums over the key rows are two shuffles inside the warp and nothing in the rows' chain is block-wide, and a warp's
// 16-byte reads of k and q fall on four different bank groups.  (Eight warps of 4 columns halve the chain's instructions, but their
// 16-byte pieces of the states' rows cost more than that: 36 us against 25 at 20 rows.)  The starting state, the history and the constants depend on no
// kernel of this window: they are loaded before the projections are waited for.
// Bound by latency at a few rows (the loads, the chain, the exchange over the cluster), by the states' 2 MB a row at many; one block
// barrier a row and every load after the wait before.
template <int CL>
__device__ __forceinline__ void gdn_body(const GdnArgs& p, int cur, float* sm) {
    cg::cluster_group cluster = cg::this_cluster();
    const int lv = blockIdx.x / GDN_Q, qq = blockIdx.x % GDN_Q, kh = lv % p.nk, tid = threadIdx.x, T = p.T, NS = p.NS;
    const int warp = tid >> 5, lane = tid & 31;
    const int ch = (2 * p.nk + p.nv) * GDN_HS;
    const size_t hsz = (size_t) 3 * ch, ssz = (size_t) p.nv * GDN_HS * GDN_HS;
    float* xq = sm;                              // [T][HS] q after conv and silu (its norm's factor is applied to the sums)
    float* xk = xq + (size_t) T * GDN_HS;        // [T][HS]
    float* vs = xk + (size_t) T * GDN_HS;        // [T][QC]
    float* os = vs + (size_t) T * GDN_QC;        // [T][QC] the rows' outputs
    float* gates = os + (size_t) T * GDN_QC;     // [T][2]
    float* fac = gates + 2 * T;                  // [T][2] 1 / |q|, 1 / |k|
    float* osum = fac + 2 * T;                   // [T][2] this block's square sums and maxima (read by the cluster)
    float* gath = osum + 2 * T;                  // [T][2 CL] the blocks' square sums and maxima
    float* xin = gath + 2 * CL * T;              // trees: [T + 3][2 HS + QC] conv inputs
    constexpr int NC = GDN_THREADS;
    int* anc = reinterpret_cast<int*>(xin + (size_t) (T + 3) * NC);   // trees: [T][3]
    auto slot_of = [&](int t) {   // the ring slot of row t's result (cur + 1 + t < 2 NS)
        const int v = cur + 1 + t;
        return v >= NS ? v - NS : v;
    };
    const int cc = (warp & 3) * 8 + (lane & 7), rg = lane >> 3;
    const size_t soff = (size_t) lv * GDN_HS * GDN_HS + (size_t) (4 * rg) * GDN_HS + qq * GDN_QC + cc;
    uint64_t s[16];   // pairs of key rows: s[2 j + h] = rows 16 j + 4 rg + 2 h, + 1
    auto load_state = [&](int slot) {
        const float* src = p.S_pool + (size_t) slot * ssz + soff;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) s[2 * j + h] = f2_pack(src[(size_t) (16 * j + 2 * h) * GDN_HS], src[(size_t) (16 * j + 2 * h + 1) * GDN_HS]);
    };
    if (warp < 4) load_state(cur);
    // this thread's channel: q, k or v element
    const int part = tid < GDN_HS ? 0 : tid < 2 * GDN_HS ? 1 : 2, el = part < 2 ? tid - part * GDN_HS : tid - 2 * GDN_HS;
    const int c = part == 0 ? kh * GDN_HS + el : part == 1 ? p.nk * GDN_HS + kh * GDN_HS + el : 2 * p.nk * GDN_HS + lv * GDN_HS + qq * GDN_QC + el;
    const float* hin = p.hist_pool + (size_t) cur * hsz;
    const float4 cw = *reinterpret_cast<const float4*>(p.convw + c * 4);
    float h0 = hin[c], h1 = hin[ch + c], h2 = hin[2 * ch + c];
    const float dtv = p.dt[lv], av = p.a[lv], nwv = p.nw[qq * GDN_QC + lane];
    pdl_wait();   // from here on: the projections
    pdl_launch_dependents();
    if (tid >= NC - 32 && lane < T) {
        const float* abt = p.ab + (size_t) lane * p.ldab;
        const float x = abt[lv] + dtv, be = abt[p.nv + lv];
        gates[2 * lane] = expf((x > 20.0f ? x : log1pf(expf(x))) * av);
        gates[2 * lane + 1] = 1.0f / (1.0f + expf(-be));
    }
    const bool writes = part == 2 || (lv < p.nk && qq == 0);   // one block per channel writes its history
    float* xout = part == 0 ? xq + el : part == 1 ? xk + el : vs + el;
    const int xstr = part < 2 ? GDN_HS : GDN_QC;
    auto put = [&](int t, float x3, float x2, float x1, float x0) {
        const float x = cw.x * x3 + cw.y * x2 + cw.z * x1 + cw.w * x0;
        xout[t * xstr] = x / (1.0f + expf(-x));
        if (writes) {
            float* hout = p.hist_pool + (size_t) slot_of(t) * hsz + c;
            hout[0] = x2;
            hout[ch] = x1;
            hout[2 * ch] = x0;
        }
    };
    const float* src = p.qkvz + c;
    if (!p.parent) {   // a chain: the channel's inputs pass through registers, eight rows' loads in flight
        for (int t0 = 0; t0 < T; t0 += 8) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = t0 + i < T ? src[(size_t) (t0 + i) * p.stride] : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (t0 + i >= T) break;
                put(t0 + i, h0, h1, h2, x[i]);
                h0 = h1;
                h1 = h2;
                h2 = x[i];
            }
        }
    } else {   // a tree: the inputs staged, rows 0..2 = the starting history (oldest first), row 3 + t = window row t
        xin[tid] = h0;
        xin[NC + tid] = h1;
        xin[2 * NC + tid] = h2;
        for (int t0 = 0; t0 < T; t0 += 16) {
            float x[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = t0 + i < T ? src[(size_t) (t0 + i) * p.stride] : 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (t0 + i < T) xin[(size_t) (3 + t0 + i) * NC + tid] = x[i];
        }
        // the three rows before each window row on its path, as rows of xin (past the root: the history)
        if (tid < T) {
            int a = tid;
            for (int k = 1; k <= 3; ++k) {
                if (a >= 0) a = p.parent[a];
                else --a;                      // a = -1 - (rows past the root)
                anc[tid * 3 + k - 1] = 3 + a;  // -1 -> row 2 (newest history), -2 -> row 1, -3 -> row 0
            }
        }
        __syncthreads();
        for (int t = 0; t < T; ++t) put(t, xin[anc[t * 3 + 2] * NC + tid], xin[anc[t * 3 + 1] * NC + tid], xin[anc[t * 3] * NC + tid], xin[(3 + t) * NC + tid]);
    }
    __syncthreads();
    // ---- the L2 norms of q and k: a warp per (row, vector)
    for (int i = warp; i < 2 * T; i += NC / 32) {
        const float4 v = *reinterpret_cast<const float4*>((i & 1 ? xk : xq) + (i >> 1) * GDN_HS + lane * 4);
        const float ss = warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w));
        if (lane == 0) fac[i] = rsqrtf(ss + 1e-6f);
    }
    __syncthreads();
    // ---- the delta rule
    if (warp < 4) {
        int have = -1;   // the row whose result the registers hold (-1: the starting state)
        const float scale = rsqrtf((float) GDN_HS);
#pragma unroll 1
        for (int t = 0; t < T; ++t) {
            if (p.parent) {
                const int par = p.parent[t];
                if (par != have) load_state(par < 0 ? cur : slot_of(par));
            }
            const float gv = gates[2 * t], bv = gates[2 * t + 1], fq = fac[2 * t], fk = fac[2 * t + 1];
            const float* kt = xk + t * GDN_HS + 4 * rg;
            const float* qt = xq + t * GDN_HS + 4 * rg;
            uint64_t kp[16], acc[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = 0ull;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(kt + 16 * j);
                kp[2 * j] = k2.x;
                kp[2 * j + 1] = k2.y;
                acc[(2 * j) & 3] = f2_fma(s[2 * j], k2.x, acc[(2 * j) & 3]);
                acc[(2 * j + 1) & 3] = f2_fma(s[2 * j + 1], k2.y, acc[(2 * j + 1) & 3]);
            }
            float a0, a1, a2, a3, a4, a5, a6, a7;
            f2_unpack(acc[0], a0, a1);
            f2_unpack(acc[1], a2, a3);
            f2_unpack(acc[2], a4, a5);
            f2_unpack(acc[3], a6, a7);
            float kv = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
            kv += __shfl_xor_sync(0xffffffffu, kv, 8);
            kv += __shfl_xor_sync(0xffffffffu, kv, 16);
            const float dk = (vs[t * GDN_QC + cc] - gv * (kv * fk)) * bv * fk;
            const uint64_t d2 = f2_pack(dk, dk), g2 = f2_pack(gv, gv);
            float* dst = p.S_pool + (size_t) slot_of(t) * ssz + soff;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = 0ull;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(qt + 16 * j);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 2 * j + h;
                    s[i] = f2_fma(kp[i], d2, f2_mul(g2, s[i]));
                    acc[i & 3] = f2_fma(s[i], h ? q2.y : q2.x, acc[i & 3]);
                    float lo, hi;
                    f2_unpack(s[i], lo, hi);
                    dst[(size_t) (16 * j + 2 * h) * GDN_HS] = lo;
                    dst[(size_t) (16 * j + 2 * h + 1) * GDN_HS] = hi;
                }
            }
            f2_unpack(acc[0], a0, a1);
            f2_unpack(acc[1], a2, a3);
            f2_unpack(acc[2], a4, a5);
            f2_unpack(acc[3], a6, a7);
            float at = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
            at += __shfl_xor_sync(0xffffffffu, at, 8);
            at += __shfl_xor_sync(0xffffffffu, at, 16);
            if (rg == 0) os[t * GDN_QC + cc] = at * fq * scale;
            have = t;
        }
    }
    // the gate inputs of the warp's output rows (warp, warp + 9, ...), fetched while the rule runs
    constexpr int OR = (FNX_MAX_ROWS + NC / 32 - 1) / (NC / 32);
    float u[OR];
#pragma unroll
    for (int j = 0; j < OR; ++j) {
        const int t = warp + j * (NC / 32);
        u[j] = t < T ? p.qkvz[(size_t) t * p.stride + ch + lv * GDN_HS + qq * GDN_QC + lane] : 0.f;
    }
    __syncthreads();
    // ---- the outputs times their norm weight and gate; their square sums and maxima
#pragma unroll
    for (int j = 0; j < OR; ++j) {
        const int t = warp + j * (NC / 32);
        if (t >= T) break;
        const float o = os[t * GDN_QC + lane];
        u[j] = o * nwv / (1.0f + expf(-u[j]));
        const float sq = warp_sum(o * o), mx = CL > GDN_Q ? warp_max(fabsf(u[j])) : 0.f;
        if (lane == 0) *reinterpret_cast<float2*>(osum + 2 * t) = make_float2(sq, mx);
    }
    cluster.sync();
    for (int i = tid; i < T * CL; i += NC) {   // every block's, one remote read per thread
        const int t = i / CL, r = i % CL;
        const float2 v = *reinterpret_cast<const float2*>(cluster.map_shared_rank(osum, r) + 2 * t);
        gath[t * 2 * CL + r] = v.x;
        gath[t * 2 * CL + CL + r] = v.y;
    }
    __syncthreads();
    const int hb = CL > GDN_Q ? (lv & 1) * GDN_Q : 0;   // the head's blocks in the cluster
#pragma unroll
    for (int j = 0; j < OR; ++j) {
        const int t = warp + j * (NC / 32);
        if (t >= T) break;
        const float* gt = gath + t * 2 * CL;
        const float r = rsqrtf(((gt[hb] + gt[hb + 1]) + (gt[hb + 2] + gt[hb + 3])) / (float) GDN_HS + p.eps), yv = u[j] * r;
        p.y[(size_t) t * p.nv * GDN_HS + lv * GDN_HS + qq * GDN_QC + lane] = yv;
        if (CL > GDN_Q) {   // the image: the block's 32 columns are a sub-block of it, eight lanes a cell of each level
            const int ob = GDN_Q - hb;
            const float ro = rsqrtf(((gt[ob] + gt[ob + 1]) + (gt[ob + 2] + gt[ob + 3])) / (float) GDN_HS + p.eps);
            const float* gm = gt + CL;
            const float am = fmaxf(fmaxf(fmaxf(gm[hb], gm[hb + 1]), fmaxf(gm[hb + 2], gm[hb + 3])) * r, fmaxf(fmaxf(gm[ob], gm[ob + 1]), fmaxf(gm[ob + 2], gm[ob + 3])) * ro);
            uint32_t w1, w2;
            float d;
            ni_code(yv, am, w1, w2, d);
            w1 <<= 8 * (lane & 3);
            w2 <<= 8 * (lane & 3);
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                w1 |= __shfl_xor_sync(0xffffffffu, w1, o);
                w2 |= __shfl_xor_sync(0xffffffffu, w2, o);
            }
            const int KB = p.nv * GDN_HS / 256, sb = (lv & 1) * 4 + qq;
            uint8_t* rec = p.img + (size_t) t * ni_row_bytes(KB) + (size_t) (lv >> 1) * NI_BYTES;
            uint8_t* cell = rec + (sb >> 1) * 64 + (lane >> 3) * 16 + (sb & 1) * 8 + (lane & 4);
            if ((lane & 3) == 0) *reinterpret_cast<uint32_t*>(cell) = w1;
            if ((lane & 3) == 1) *reinterpret_cast<uint32_t*>(cell + 256) = w2;
            if (sb == 0 && lane == 2) *reinterpret_cast<float4*>(rec + NI_SCALE) = make_float4(d, d * (1.0f / 256.0f), 0.f, 0.f);
        }
    }
    cluster.sync();   // no block may leave while a neighbour still reads its shared memory
}

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(GDN_THREADS, 2) k_gdn_core(const GdnArgs p, const int* __restrict__ curp) {
    extern __shared__ __align__(16) float sm[];
    gdn_body<CL>(p, *curp % p.NS, sm);
}

// Batched lanes: blockIdx.y = lane j, the rows [lane_row0[j], lane_row0[j + 1]) of sequence lane_seq[j], a chain from
// that sequence's state slot cur[seq] in its own rings (hist_pool + seq * hist_stride, S_pool + seq * s_stride)
// (gdn_core_segs, engine/src/kernels.cu:2112-2156).  Every block of a cluster has the same lane, so all of them take
// the same path.
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(GDN_THREADS, 2)
    k_gdn_core_lanes(const GdnArgs p0, size_t hist_stride, size_t s_stride, const int* __restrict__ cur, const int* __restrict__ lane_seq,
                     const int* __restrict__ lane_row0) {
    extern __shared__ __align__(16) float sm[];
    const int lane = blockIdx.y, row0 = lane_row0[lane], T = lane_row0[lane + 1] - row0, seq = lane_seq[lane];
    if (T <= 0 || seq < 0) {   // (a negative sequence: another rank's lane)
        pdl_wait();
        return;
    }
    GdnArgs p = p0;
    p.qkvz += (size_t) row0 * p.stride;
    p.ab += (size_t) row0 * p.ldab;
    p.hist_pool += seq * hist_stride;
    p.S_pool += seq * s_stride;
    p.y += (size_t) row0 * p.nv * GDN_HS;
    if (p.img) p.img += (size_t) row0 * ni_row_bytes(p.nv * GDN_HS / 256);
    p.T = T;
    p.parent = nullptr;
    gdn_body<CL>(p, cur[seq], sm);
}

// ------------------------------------------------------------------------------------------------ prompts
// A prompt's rows are a chain of which every row is kept, so the work splits by what depends on what (gdn_prompt,
// engine/src/kernels.cu:2158): conv + SiLU, the q / k norms and the gates of every row at once (k_gdn_pre); the delta rule, the
// only sequential part, with the state in registers from the first row to the last and the rows' q, k, v streamed through
// shared memory (k_gdn_scan); the gated RMS norm of every row at once (k_gdn_post).  Only the last row's state and the last
// three rows' conv inputs are written back.
constexpr int GDP_THREADS = 256;

// block = one row; thread = channels tid, tid + 256, ...  xq / xk [T][nk][HS], xv [T][nv][HS], gates [T][nv][2]
__global__ void __launch_bounds__(GDP_THREADS) k_gdn_pre(const float* __restrict__ qkvz, int stride, const float* __restrict__ ab, int ldab,
                                                         const float* __restrict__ hin, float* __restrict__ hout, const float* __restrict__ convw,
                                                         const float* __restrict__ dt, const float* __restrict__ a_, float* __restrict__ xq,
                                                         float* __restrict__ xk, float* __restrict__ xv, float* __restrict__ gates, int nk, int nv, int T) {
    __shared__ float red[GDP_THREADS / 32];
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ch = (2 * nk + nv) * GDN_HS;
    // row t - k of the chain: a row of this call, or the history the call starts from (rows 0..2, oldest first)
    auto xrow = [&](int r, int c) { return r >= 0 ? qkvz[(size_t) r * stride + c] : hin[(size_t) (3 + r) * ch + c]; };
    for (int c0 = 0; c0 < ch; c0 += GDP_THREADS) {
        const int c = c0 + tid;
        const float4 cw = *reinterpret_cast<const float4*>(convw + (size_t) c * 4);
        const float x3 = xrow(t - 3, c), x2 = xrow(t - 2, c), x1 = xrow(t - 1, c), x0 = xrow(t, c);
        const float x = cw.x * x3 + cw.y * x2 + cw.z * x1 + cw.w * x0;
        float v = x / (1.0f + expf(-x));
        if (t == T - 1) {   // the history the next call starts from
            hout[c] = x2;
            hout[ch + c] = x1;
            hout[2 * ch + c] = x0;
        }
        if (c < 2 * nk * GDN_HS) {
            // q and k heads: the L2 norm over the head's 128 channels = four warps of this pass (two heads per pass)
            const float sq = warp_sum(v * v);
            __syncthreads();
            if (lane == 0) red[warp] = sq;
            __syncthreads();
            const int w0 = warp & ~3;
            float ssum = 0.f;
            for (int w = 0; w < 4; ++w) ssum += red[w0 + w];
            v *= rsqrtf(ssum + 1e-6f);
            if (c < nk * GDN_HS) xq[(size_t) t * nk * GDN_HS + c] = v;
            else xk[(size_t) t * nk * GDN_HS + (c - nk * GDN_HS)] = v;
        } else {
            xv[(size_t) t * nv * GDN_HS + (c - 2 * nk * GDN_HS)] = v;
        }
    }
    if (tid < nv) {
        const float* abt = ab + (size_t) t * ldab;
        const float x = abt[tid] + dt[tid];
        gates[((size_t) t * nv + tid) * 2] = expf((x > 20.0f ? x : log1pf(expf(x))) * a_[tid]);
        gates[((size_t) t * nv + tid) * 2 + 1] = 1.0f / (1.0f + expf(-abt[nv + tid]));
    }
}

// block = (value head, column quarter) as in the window kernel: warp `part` holds key rows [32 part, +32) of the block's 32 value
// columns, lane = column.  Rows stream through two shared-memory tiles of GDS_ROWS rows.
constexpr int GDS_ROWS = 16;
__global__ void __launch_bounds__(GDS_THREADS) k_gdn_scan(const float* __restrict__ xq, const float* __restrict__ xk, const float* __restrict__ xv,
                                                          const float* __restrict__ gates, const float* __restrict__ S_in, float* __restrict__ S_out,
                                                          float* __restrict__ o, int nk, int nv, int T) {
    constexpr int ROWF = 2 * GDN_HS + GDN_QC + 2;   // floats of a staged row: k, q, the block's v, the two gates
    __shared__ __align__(16) float tile[2][GDS_ROWS][ROWF + 2];
    __shared__ float kred[2][4][GDN_QC], ared[GDS_ROWS][4][GDN_QC];
    const int lv = blockIdx.x / GDN_Q, qq = blockIdx.x % GDN_Q, kh = lv % nk, tid = threadIdx.x;
    const int part = tid >> 5, lane = tid & 31, col = qq * GDN_QC + lane;
    const size_t soff = (size_t) lv * GDN_HS * GDN_HS + (size_t) part * 32 * GDN_HS + col;
    uint64_t s[16];   // the thread's 32 state values, in pairs (rows 2 i, 2 i + 1)
#pragma unroll
    for (int r = 0; r < 32; r += 2) s[r / 2] = f2_pack(S_in[soff + (size_t) r * GDN_HS], S_in[soff + (size_t) (r + 1) * GDN_HS]);
    auto stage = [&](int buf, int t0) {
        const int nr = min(GDS_ROWS, T - t0);
        for (int i = tid; i < nr * (ROWF / 2); i += GDS_THREADS) {   // 8-byte pieces
            const int r = i / (ROWF / 2), e = (i % (ROWF / 2)) * 2, t = t0 + r;
            const float* src;
            if (e < GDN_HS) src = xk + ((size_t) t * nk + kh) * GDN_HS + e;
            else if (e < 2 * GDN_HS) src = xq + ((size_t) t * nk + kh) * GDN_HS + (e - GDN_HS);
            else if (e < 2 * GDN_HS + GDN_QC) src = xv + ((size_t) t * nv + lv) * GDN_HS + qq * GDN_QC + (e - 2 * GDN_HS);
            else src = gates + ((size_t) t * nv + lv) * 2;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(&tile[buf][r][e])), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const float scale = rsqrtf((float) GDN_HS);
    stage(0, 0);
    int buf = 0;
    for (int t0 = 0; t0 < T; t0 += GDS_ROWS, buf ^= 1) {
        const int nr = min(GDS_ROWS, T - t0);
        if (t0 + GDS_ROWS < T) {
            stage(buf ^ 1, t0 + GDS_ROWS);   // (its last readers passed the barrier that ended the previous tile)
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
#pragma unroll 1
        for (int r0 = 0; r0 < nr; ++r0) {
            const float* row = tile[buf][r0];
            const float* kt = row + part * 32;
            const float* qt = row + GDN_HS + part * 32;
            const float gv = row[2 * GDN_HS + GDN_QC], bv = row[2 * GDN_HS + GDN_QC + 1];
            // (the row's k and q for this warp's 32 key rows: eight 16-byte broadcast reads each, as pairs)
            uint64_t kp[16], qp[16];
#pragma unroll
            for (int r = 0; r < 32; r += 4) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(kt + r), b = *reinterpret_cast<const ulonglong2*>(qt + r);
                kp[r / 2] = a.x; kp[r / 2 + 1] = a.y;
                qp[r / 2] = b.x; qp[r / 2 + 1] = b.y;
            }
            // eight running sums in four pairs (row r of the 32 goes to sum r % 8): four independent chains of packed products
            uint64_t kacc[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) kacc[i] = f2_pack(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < 16; r += 4)
#pragma unroll
                for (int i = 0; i < 4; ++i) kacc[i] = f2_fma(s[r + i], kp[r + i], kacc[i]);
            float k0, k1, k2, k3, k4, k5, k6, k7;
            f2_unpack(kacc[0], k0, k1);
            f2_unpack(kacc[1], k2, k3);
            f2_unpack(kacc[2], k4, k5);
            f2_unpack(kacc[3], k6, k7);
            float* kr = &kred[r0 & 1][0][0];
            kr[part * GDN_QC + lane] = ((k0 + k1) + (k2 + k3)) + ((k4 + k5) + (k6 + k7));
            __syncthreads();
            const float kvs = (kr[lane] + kr[GDN_QC + lane]) + (kr[2 * GDN_QC + lane] + kr[3 * GDN_QC + lane]);
            const float delta = (row[2 * GDN_HS + lane] - gv * kvs) * bv;
            const uint64_t d2 = f2_pack(delta, delta), g2 = f2_pack(gv, gv);
            uint64_t aacc[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) aacc[i] = f2_pack(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < 16; r += 4)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[r + i] = f2_fma(kp[r + i], d2, f2_mul(g2, s[r + i]));
                    aacc[i] = f2_fma(s[r + i], qp[r + i], aacc[i]);
                }
            float a0, a1, a2, a3, a4, a5, a6, a7;
            f2_unpack(aacc[0], a0, a1);
            f2_unpack(aacc[1], a2, a3);
            f2_unpack(aacc[2], a4, a5);
            f2_unpack(aacc[3], a6, a7);
            ared[r0][part][lane] = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
        }
        __syncthreads();   // the tile's sums are complete; its buffer may be refilled two tiles on
        for (int i = tid; i < nr * GDN_QC; i += GDS_THREADS) {
            const int r0 = i / GDN_QC, c = i % GDN_QC;
            o[((size_t) (t0 + r0) * nv + lv) * GDN_HS + qq * GDN_QC + c] = ((ared[r0][0][c] + ared[r0][1][c]) + (ared[r0][2][c] + ared[r0][3][c])) * scale;
        }
    }
#pragma unroll
    for (int r = 0; r < 32; r += 2) {
        float x, y;
        f2_unpack(s[r / 2], x, y);
        S_out[soff + (size_t) r * GDN_HS] = x;
        S_out[soff + (size_t) (r + 1) * GDN_HS] = y;
    }
}

// block = one row, warp = a quarter (32 columns) of a value head at a time: y = o * rsqrt(mean(o^2) + eps) * nw * sigmoid(z)
__global__ void __launch_bounds__(GDP_THREADS) k_gdn_post(const float* __restrict__ o, const float* __restrict__ qkvz, int stride, const float* __restrict__ nw,
                                                          float* __restrict__ y, int nk, int nv, float eps) {
    __shared__ float red[GDP_THREADS / 32];
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ch = (2 * nk + nv) * GDN_HS;
    for (int c0 = 0; c0 < nv * GDN_HS; c0 += GDP_THREADS) {
        const int c = c0 + tid, col = c % GDN_HS;
        const float ov = o[(size_t) t * nv * GDN_HS + c];
        const float zv = qkvz[(size_t) t * stride + ch + c];
        const float sq = warp_sum(ov * ov);
        __syncthreads();
        if (lane == 0) red[warp] = sq;
        __syncthreads();
        const int w0 = warp & ~3;
        const float ms = ((red[w0] + red[w0 + 1]) + (red[w0 + 2] + red[w0 + 3])) / (float) GDN_HS;
        y[(size_t) t * nv * GDN_HS + c] = ov * rsqrtf(ms + eps) * nw[col] / (1.0f + expf(-zv));
    }
}

static size_t gdn_smem_bytes(int T, int CL, bool tree) {
    return sizeof(float) * ((size_t) 2 * T * GDN_HS + (size_t) 2 * T * GDN_QC + 6 * T + 2 * CL * T + (tree ? (size_t) (T + 3) * (2 * GDN_HS + GDN_QC) + 3 * T : 0));
}

// an image needs the two heads of its 256-column blocks in one cluster
int gdn_window(const GdnArgs& p, const int* cur, bool early, cudaStream_t st) {
    const int CL = p.img ? 2 * GDN_Q : GDN_Q;
    auto kernel = p.img ? k_gdn_core<2 * GDN_Q> : k_gdn_core<GDN_Q>;
    if (int rc = set_smem_limit((const void*) kernel, 112 * 1024)) return rc;
    const cudaError_t le = launch_dep(early, kernel, dim3(p.nv * GDN_Q), dim3(GDN_THREADS), gdn_smem_bytes(p.T, CL, p.parent != nullptr), st, p, cur);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_gdn_core: launch failed: %s", cudaGetErrorString(le));
}
int gdn_window_lanes(const GdnArgs& p, size_t hist_seq_stride, size_t s_seq_stride, const int* cur, const int* lane_seq, const int* lane_row0, int n_lanes, int max_rows,
                     bool early, cudaStream_t st) {
    const int CL = p.img ? 2 * GDN_Q : GDN_Q;
    auto kernel = p.img ? k_gdn_core_lanes<2 * GDN_Q> : k_gdn_core_lanes<GDN_Q>;
    if (int rc = set_smem_limit((const void*) kernel, 112 * 1024)) return rc;
    const cudaError_t le = launch_dep(early, kernel, dim3(p.nv * GDN_Q, n_lanes), dim3(GDN_THREADS), gdn_smem_bytes(max_rows, CL, false), st, p, hist_seq_stride, s_seq_stride, cur,
                                      lane_seq, lane_row0);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_gdn_core_lanes: launch failed: %s", cudaGetErrorString(le));
}

}  // namespace fnxb

using namespace fnxb;

extern "C" int fnx_gdn_core(const float* qkvz, int ldx, const float* ab, int ldab, float* hist_pool, const float* convw, const float* dt, const float* a,
                            const float* nw, float* S_pool, const int* cur, int NS, const int* parent, float* y, int nk, int nv, int hs,
                            int T, float eps, fnx_stream st) {
    FNX_REQUIRE(qkvz && ab && hist_pool && convw && dt && a && nw && S_pool && cur && y, "fnx_gdn_core: null pointer");
    FNX_REQUIRE(hs == GDN_HS, "fnx_gdn_core: head dim %d (this build: %d)", hs, GDN_HS);
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS && NS >= T + 1, "fnx_gdn_core: %d rows need at least %d state slots, have %d", T, T + 1, NS);
    FNX_REQUIRE(nk >= 1 && nv >= nk && nv % nk == 0, "fnx_gdn_core: %d key heads, %d value heads", nk, nv);
    return gdn_window(GdnArgs{qkvz, ldx, ab, ldab, hist_pool, convw, dt, a, nw, S_pool, NS, parent, y, nullptr, nk, nv, T, eps}, cur, false, as_stream(st));
}

extern "C" size_t fnx_gdn_prompt_scratch_bytes(int T, int nk, int nv, int hs) {
    return sizeof(float) * ((size_t) T * (2 * nk + 2 * nv) * hs + (size_t) T * nv * 2 + (size_t) 3 * (2 * nk + nv) * hs) + 1024;
}

extern "C" int fnx_gdn_prompt(const float* qkvz, int ldx, const float* ab, int ldab, float* hist_pool, const float* convw, const float* dt, const float* a,
                              const float* nw, float* S_pool, int cur_host, int NS, float* y, int nk, int nv, int hs, int T, float eps, void* scratch,
                              fnx_stream st) {
    FNX_REQUIRE(qkvz && ab && hist_pool && convw && dt && a && nw && S_pool && y && scratch, "fnx_gdn_prompt: null pointer");
    FNX_REQUIRE(hs == GDN_HS, "fnx_gdn_prompt: head dim %d (this build: %d)", hs, GDN_HS);
    FNX_REQUIRE(T >= 1 && NS >= 2 && cur_host >= 0 && cur_host < NS, "fnx_gdn_prompt: %d rows, slot %d of %d", T, cur_host, NS);
    FNX_REQUIRE(nk >= 1 && nv >= nk && nv % nk == 0 && nv <= GDP_THREADS && ((2 * nk + nv) * GDN_HS) % GDP_THREADS == 0, "fnx_gdn_prompt: %d key heads, %d value heads", nk, nv);
    const int ch = (2 * nk + nv) * GDN_HS, out_slot = (cur_host + T) % NS;
    const size_t hsz = (size_t) 3 * ch, ssz = (size_t) nv * GDN_HS * GDN_HS;
    float* xq = (float*) scratch;
    float* xk = xq + (size_t) T * nk * GDN_HS;
    float* xv = xk + (size_t) T * nk * GDN_HS;
    float* o = xv + (size_t) T * nv * GDN_HS;
    float* gates = o + (size_t) T * nv * GDN_HS;
    cudaStream_t s = as_stream(st);
    // the history the call starts from is read from a copy: the slot it leaves its own in may be the same one
    float* hin = gates + (size_t) T * nv * 2;
    FNX_CUDA_OK(cudaMemcpyAsync(hin, hist_pool + (size_t) cur_host * hsz, hsz * sizeof(float), cudaMemcpyDeviceToDevice, s));
    k_gdn_pre<<<T, GDP_THREADS, 0, s>>>(qkvz, ldx, ab, ldab, hin, hist_pool + (size_t) out_slot * hsz, convw, dt, a, xq, xk, xv, gates, nk,
                                         nv, T);
    FNX_LAUNCH_OK("k_gdn_pre");
    k_gdn_scan<<<nv * GDN_Q, GDS_THREADS, 0, s>>>(xq, xk, xv, gates, S_pool + (size_t) cur_host * ssz, S_pool + (size_t) out_slot * ssz, o, nk, nv, T);
    FNX_LAUNCH_OK("k_gdn_scan");
    k_gdn_post<<<T, GDP_THREADS, 0, s>>>(o, qkvz, ldx, nw, y, nk, nv, eps);
    FNX_LAUNCH_OK("k_gdn_post");
    return FNX_OK;
}

extern "C" int fnx_gdn_core_lanes(const float* qkvz, int ldx, const float* ab, int ldab, float* hist_pool, size_t hist_seq_stride, const float* convw,
                                  const float* dt, const float* a, const float* nw, float* S_pool, size_t s_seq_stride, const int* cur, int NS,
                                  const int* lane_seq, const int* lane_row0, int n_lanes, int max_lane_rows, float* y, int nk, int nv, int hs, float eps,
                                  fnx_stream st) {
    FNX_REQUIRE(qkvz && ab && hist_pool && convw && dt && a && nw && S_pool && cur && lane_seq && lane_row0 && y, "fnx_gdn_core_lanes: null pointer");
    FNX_REQUIRE(hs == GDN_HS, "fnx_gdn_core_lanes: head dim %d (this build: %d)", hs, GDN_HS);
    FNX_REQUIRE(n_lanes >= 1 && n_lanes <= FNX_MAX_ROWS && max_lane_rows >= 1 && NS >= max_lane_rows + 1, "fnx_gdn_core_lanes: %d lanes of up to %d rows, %d state slots",
                n_lanes, max_lane_rows, NS);
    FNX_REQUIRE(nk >= 1 && nv >= nk && nv % nk == 0, "fnx_gdn_core_lanes: %d key heads, %d value heads", nk, nv);
    return gdn_window_lanes(GdnArgs{qkvz, ldx, ab, ldab, hist_pool, convw, dt, a, nw, S_pool, NS, nullptr, y, nullptr, nk, nv, max_lane_rows, eps}, hist_seq_stride,
                            s_seq_stride, cur, lane_seq, lane_row0, n_lanes, max_lane_rows, false, as_stream(st));
}
