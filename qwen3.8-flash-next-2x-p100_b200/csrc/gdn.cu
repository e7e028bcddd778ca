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

#include <type_traits>

#include "gdn_core.h"
#include "nat_image.cuh"

namespace cg = cooperative_groups;

namespace fnxb {

constexpr int GDN_HS = 128, GDN_Q = 4, GDN_QC = GDN_HS / GDN_Q, GDN_THREADS = 256, GDS_THREADS = 128;

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
// block of it, form a cluster.  Warps 0 .. 3 run the delta rule: a lane holds a column, its warp every fourth group of four key rows, so that a state's rows
// leave in whole lines; a row's sums over the key rows are exchanged once, behind one barrier of the four warps, and what the row gives out and what the next one
// takes from the state are summed as the state is updated.  The first four rows' conv and norms are everybody's; warps 4 .. 7 go on with the rest, four
// rows at a time, ahead of the rule.  The starting state, the history, the constants and a tree's paths depend on no kernel of this window: they are loaded before
// the projections are waited for.
// Bound by latency at a few rows (the loads, the chain, the exchange over the cluster); at many by the rule.  By its clocks, 32 value heads (a block an SM), a row's 0.72 us between 12
// and 32 rows are 1,000 cycles of the rule and 0.2 us ahead of it and behind it; of the rule's some 590 lie in the update with the states' stores (16 KB at an SM's 32 bytes a
// cycle; 250 in a copy without the stores, whose row takes 880), some 400 in the totals, their exchange and the next row's loads, 45 in the wait for the conv.
// us a launch, 1, 5, 8 and 20 rows and a tree of 20, in the form before (columns eight a warp, sums by shuffles, all of the conv ahead of the rule) and here: 4.5 8.8 11.6 24.6
// 28.2, 4.3 8.0 10.6 18.7 19.4.  Tried here: the states out of shared memory by tensor copies (20 rows 20 to 23), eight warps for the rule and eight for the conv (19.0), an SM
// to each block (16 clusters of eight do not fit at once: 35).
constexpr int GDN_BATCH = 4, GDN_CHANS = 2 * GDN_HS + GDN_QC;

__host__ __device__ constexpr bool gdn_staged(int T, bool tree) { return tree || T > GDN_BATCH; }

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
    float* os = vs + (size_t) T * GDN_QC;        // [T][4][QC] the rows' outputs, a warp's key rows each
    float* ug = os + (size_t) 4 * T * GDN_QC;    // [T][QC] their gates' inputs
    float* sk = ug + (size_t) T * GDN_QC;        // [2][4][QC] S' k of the row that is next, a warp's key rows each
    float* gates = sk + 8 * GDN_QC;              // [T][2]
    float* fac = gates + 2 * T;                  // [T][2] 1 / |q|, 1 / |k|
    float* osum = fac + 2 * T;                   // [T][2] this block's square sums and maxima (read by the cluster)
    float* xin = gates + ((6 * T + 3) & ~3);     // staged inputs: [T + 3][channels], rows 0..2 = the starting history (oldest first), row 3 + t = row t
    int* anc = reinterpret_cast<int*>(xin + (size_t) (T + 3) * GDN_CHANS);   // trees: [T][4] the last three rows before each on its path, as rows of xin
    auto slot_of = [&](int t) {   // the ring slot of row t's result (cur + 1 + t < 2 NS)
        const int v = cur + 1 + t;
        return v >= NS ? v - NS : v;
    };
    const int rg = warp & 3;
    const size_t soff = (size_t) lv * GDN_HS * GDN_HS + (size_t) (4 * rg) * GDN_HS + qq * GDN_QC + lane;
    uint64_t s[16];   // pairs of key rows: s[2 j + h] = rows 16 j + 4 rg + 2 h, + 1
    auto load_state = [&](int slot) {
        const float* src = p.S_pool + (size_t) slot * ssz + soff;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) s[2 * j + h] = f2_pack(src[(size_t) (16 * j + 2 * h) * GDN_HS], src[(size_t) (16 * j + 2 * h + 1) * GDN_HS]);
    };
    if (warp < 4) load_state(cur);
    // the thread's channel: an element of q (warps 0 .. 3) or k; warp 4 has the v columns besides
    const int el = tid & (GDN_HS - 1);
    const int cA = (tid < GDN_HS ? 0 : p.nk * GDN_HS) + kh * GDN_HS + el, cQ = kh * GDN_HS + el, cV = 2 * p.nk * GDN_HS + lv * GDN_HS + qq * GDN_QC + lane;
    const float* hin = p.hist_pool + (size_t) cur * hsz;
    const float4 wA = *reinterpret_cast<const float4*>(p.convw + cA * 4);
    float a0 = hin[cA], a1 = hin[ch + cA], a2 = hin[2 * ch + cA];
    float4 wV = make_float4(0.f, 0.f, 0.f, 0.f);
    float v0 = 0.f, v1 = 0.f, v2 = 0.f;
    if (warp == 4) {
        wV = *reinterpret_cast<const float4*>(p.convw + cV * 4);
        v0 = hin[cV];
        v1 = hin[ch + cV];
        v2 = hin[2 * ch + cV];
    }
    const float dtv = p.dt[lv], av = p.a[lv], nwv = p.nw[qq * GDN_QC + lane];
    if (p.parent) {
        if (tid < T) {
            int a = tid;
            for (int k = 0; k < 3; ++k) {
                if (a >= 0) a = p.parent[a];
                else --a;                  // a = -1 - (rows past the root)
                anc[tid * 4 + k] = 3 + a;  // -1 -> row 2 (newest history), -2 -> row 1, -3 -> row 0
            }
        }
        __syncthreads();
    }
    pdl_wait();   // from here on: the projections
    pdl_launch_dependents();
    auto copy4 = [](float* dst, const float* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
    float xA[GDN_BATCH], xV[GDN_BATCH];
#pragma unroll
    for (int i = 0; i < GDN_BATCH; ++i) {
        xA[i] = i < T ? p.qkvz[(size_t) i * p.stride + cA] : 0.f;
        xV[i] = i < T && warp == 4 ? p.qkvz[(size_t) i * p.stride + cV] : 0.f;
    }
    if (warp == 7 && lane < T) {
        const float* abt = p.ab + (size_t) lane * p.ldab;
        const float x = abt[lv] + dtv, be = abt[p.nv + lv];
        gates[2 * lane] = expf((x > 20.0f ? x : log1pf(expf(x))) * av);
        gates[2 * lane + 1] = 1.0f / (1.0f + expf(-be));
    }
    if (warp >= 4)   // the rows after the first batch
        for (int t = GDN_BATCH; t < T; ++t) {
            const float* src = p.qkvz + (size_t) t * p.stride;
            float* dst = xin + (size_t) (3 + t) * GDN_CHANS;
            copy4(dst + el, src + cQ);
            copy4(dst + tid, src + cA);
            if (warp == 4) copy4(dst + 2 * GDN_HS + lane, src + cV);
        }
    for (int t = warp; t < T; t += GDN_THREADS / 32) copy4(ug + t * GDN_QC + lane, p.qkvz + (size_t) t * p.stride + ch + lv * GDN_HS + qq * GDN_QC + lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // (one block per channel writes its history)
    const bool own = lv < p.nk && qq == 0;
    // (the products in the order that the compiler gave them when it chose: a row's bits stay what they were)
    auto put = [&](int t, const float4& w, float* out, int c, bool writes, float x3, float x2, float x1, float x0) {
        const float x = fmaf(w.w, x0, fmaf(w.z, x1, fmaf(w.x, x3, w.y * x2)));
        *out = x / (1.0f + expf(-x));
        if (writes) {
            float* hout = p.hist_pool + (size_t) slot_of(t) * hsz + c;
            hout[0] = x2;
            hout[ch] = x1;
            hout[2 * ch] = x0;
        }
    };
    auto put_path = [&](int t, const float4& w, float* out, int c, bool writes, const float* col) {   // from staged inputs
        int4 at = make_int4(t + 2, t + 1, t, 0);
        if (p.parent) at = *reinterpret_cast<const int4*>(anc + t * 4);
        put(t, w, out, c, writes, col[at.z * GDN_CHANS], col[at.y * GDN_CHANS], col[at.x * GDN_CHANS], col[(3 + t) * GDN_CHANS]);
    };
    if (gdn_staged(T, p.parent != nullptr)) {   // (a thread's own columns: read back by itself, and by the others behind the barrier below)
        float* col = xin + tid;
        col[0] = a0;
        col[GDN_CHANS] = a1;
        col[2 * GDN_CHANS] = a2;
#pragma unroll
        for (int i = 0; i < GDN_BATCH; ++i)
            if (i < T) col[(3 + i) * GDN_CHANS] = xA[i];
        if (warp == 4) {
            col = xin + 2 * GDN_HS + lane;
            col[0] = v0;
            col[GDN_CHANS] = v1;
            col[2 * GDN_CHANS] = v2;
#pragma unroll
            for (int i = 0; i < GDN_BATCH; ++i)
                if (i < T) col[(3 + i) * GDN_CHANS] = xV[i];
        }
    }
    float* outA = (tid < GDN_HS ? xq : xk) + el;
    if (p.parent) {
#pragma unroll 2
        for (int t = 0; t < min(T, GDN_BATCH); ++t) {
            put_path(t, wA, outA + t * GDN_HS, cA, own, xin + tid);
            if (warp == 4) put_path(t, wV, vs + t * GDN_QC + lane, cV, true, xin + 2 * GDN_HS + lane);
        }
    } else {
#pragma unroll
        for (int i = 0; i < GDN_BATCH; ++i) {
            if (i >= T) break;
            put(i, wA, outA + i * GDN_HS, cA, own, a0, a1, a2, xA[i]);
            a0 = a1;
            a1 = a2;
            a2 = xA[i];
            if (warp == 4) {
                put(i, wV, vs + i * GDN_QC + lane, cV, true, v0, v1, v2, xV[i]);
                v0 = v1;
                v1 = v2;
                v2 = xV[i];
            }
        }
    }
    // the L2 norms of n rows' q and k by w of nw warps: eight lanes a vector, four 16-byte pieces a lane
    auto norms = [&](int r0, int n, int w, int nw) {
        for (int i0 = 4 * w; i0 < 2 * n; i0 += 4 * nw) {
            const int i = min(i0 + (lane >> 3), 2 * n - 1), row = r0 + (i >> 1);
            const float* v = (i & 1 ? xk : xq) + row * GDN_HS + (lane & 7) * 4;
            float ss[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 x = *reinterpret_cast<const float4*>(v + 32 * k);
                ss[k] = (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
            }
            float sum = (ss[0] + ss[2]) + (ss[1] + ss[3]);
#pragma unroll
            for (int o = 4; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if ((lane & 7) == 0) fac[2 * row + (i & 1)] = rsqrtf(sum + 1e-6f);
        }
    };
    __syncthreads();
    if (warp < 4) {
        // ---- the delta rule.  A row's output and the next row's S' k are sums over the same state: both are taken as it is updated.
        norms(0, min(T, GDN_BATCH), 0, 1);   // (each of the four warps for itself: the same values)
        __syncwarp();
        uint64_t ak[4], aq[4];   // sums in pairs
        auto zero = [](uint64_t (&a)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = 0ull;
        };
        auto total = [](const uint64_t (&a)[4]) {
            float a0, a1, a2, a3, a4, a5, a6, a7;
            f2_unpack(a[0], a0, a1);
            f2_unpack(a[1], a2, a3);
            f2_unpack(a[2], a4, a5);
            f2_unpack(a[3], a6, a7);
            return ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
        };
        auto sums_with = [&](const float* k) {
            zero(ak);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(k + 16 * j);
                ak[(2 * j) & 3] = f2_fma(s[2 * j], k2.x, ak[(2 * j) & 3]);
                ak[(2 * j + 1) & 3] = f2_fma(s[2 * j + 1], k2.y, ak[(2 * j + 1) & 3]);
            }
        };
        const float* kt = xk + 4 * rg;
        const float* qt = xq + 4 * rg;
        if (p.parent && p.parent[0] >= 0) load_state(slot_of(p.parent[0]));
        sums_with(kt);
        sk[rg * GDN_QC + lane] = total(ak);
#pragma unroll 1
        for (int t = 0; t < T; ++t) {
            const bool last = t + 1 == T;
            if (!last && (t + 1) % GDN_BATCH == 0) asm volatile("bar.sync %0, %1;" ::"r"(2 + (t + 1) / GDN_BATCH), "n"(GDN_THREADS) : "memory");   // the next batch is ready
            const float gv = gates[2 * t], bv = gates[2 * t + 1], fk = fac[2 * t + 1], v = vs[t * GDN_QC + lane];
            const float* sums = sk + (t & 1) * 4 * GDN_QC + lane;
            const float* kn = last ? kt : kt + GDN_HS;   // (the last row's sums with its own k are dropped)
            // k, q and the next k are loaded two steps ahead, before the stores that the compiler would keep them behind
            constexpr int AHEAD = 2;
            ulonglong2 k1[AHEAD], q1[AHEAD], n1[AHEAD];
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) {
                k1[j] = *reinterpret_cast<const ulonglong2*>(kt + 16 * j);
                q1[j] = *reinterpret_cast<const ulonglong2*>(qt + 16 * j);
                n1[j] = *reinterpret_cast<const ulonglong2*>(kn + 16 * j);
            }
            const int par = p.parent && !last ? anc[4 * t + 4] - 3 : t;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const float kv = (sums[0] + sums[GDN_QC]) + (sums[2 * GDN_QC] + sums[3 * GDN_QC]);
            const float dk = (v - gv * (kv * fk)) * bv * fk;
            const uint64_t d2 = f2_pack(dk, dk), g2 = f2_pack(gv, gv);
            float* dst = p.S_pool + (size_t) slot_of(t) * ssz + soff;
            zero(ak);
            zero(aq);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 k = k1[j % AHEAD], q = q1[j % AHEAD], n = n1[j % AHEAD];
                if (j + AHEAD < 8) {
                    k1[j % AHEAD] = *reinterpret_cast<const ulonglong2*>(kt + 16 * (j + AHEAD));
                    q1[j % AHEAD] = *reinterpret_cast<const ulonglong2*>(qt + 16 * (j + AHEAD));
                    n1[j % AHEAD] = *reinterpret_cast<const ulonglong2*>(kn + 16 * (j + AHEAD));
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 2 * j + h;
                    s[i] = f2_fma(h ? k.y : k.x, d2, f2_mul(g2, s[i]));
                    aq[i & 3] = f2_fma(s[i], h ? q.y : q.x, aq[i & 3]);
                    ak[i & 3] = f2_fma(s[i], h ? n.y : n.x, ak[i & 3]);
                    float lo, hi;
                    f2_unpack(s[i], lo, hi);
                    dst[(16 * j + 2 * h) * GDN_HS] = lo;
                    dst[(16 * j + 2 * h + 1) * GDN_HS] = hi;
                }
            }
            if (par != t) {   // a tree: the next row leaves from another row's state
                load_state(par < 0 ? cur : slot_of(par));
                sums_with(kn);
            }
            sk[((t + 1) & 1) * 4 * GDN_QC + rg * GDN_QC + lane] = total(ak);
            os[(t * 4 + rg) * GDN_QC + lane] = total(aq);
            kt += GDN_HS;
            qt += GDN_HS;
        }
    } else if (T > GDN_BATCH) {
        // ---- the batches after the first, ahead of the rule
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        const float4 wQ = *reinterpret_cast<const float4*>(p.convw + cQ * 4);
#pragma unroll 1
        for (int t0 = GDN_BATCH; t0 < T; t0 += GDN_BATCH) {
#pragma unroll 1
            for (int t = t0; t < min(T, t0 + GDN_BATCH); ++t) {   // (rolled: the rule's loop runs beside it)
                put_path(t, wA, xk + t * GDN_HS + el, cA, own, xin + tid);
                put_path(t, wQ, xq + t * GDN_HS + el, cQ, own, xin + el);
                if (warp == 4) put_path(t, wV, vs + t * GDN_QC + lane, cV, true, xin + 2 * GDN_HS + lane);
            }
            asm volatile("bar.sync 2, 128;" ::: "memory");
            norms(t0, min(GDN_BATCH, T - t0), 7 - warp, 4);
            asm volatile("bar.arrive %0, %1;" ::"r"(2 + t0 / GDN_BATCH), "n"(GDN_THREADS) : "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // (a thread reads the gate inputs that it copied)
    __syncthreads();
    // ---- the outputs times their norm weight and gate, their square sums and maxima, and the cluster's: row warp + 8 j
    auto results = [&](auto rows) {
        constexpr int N = decltype(rows)::value;
        const float scale = rsqrtf((float) GDN_HS);
        float u[N];
        float2 g[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int t = min(warp + 8 * j, T - 1);
            const float* ot = os + 4 * t * GDN_QC + lane;
            const float o = ((ot[0] + ot[GDN_QC]) + (ot[2 * GDN_QC] + ot[3 * GDN_QC])) * fac[2 * t] * scale;
            u[j] = o * nwv / (1.0f + expf(-ug[t * GDN_QC + lane]));
            g[j] = make_float2(o * o, fabsf(u[j]));
        }
#pragma unroll
        for (int d = 16; d; d >>= 1)
#pragma unroll
            for (int j = 0; j < N; ++j) {
                g[j].x += __shfl_xor_sync(0xffffffffu, g[j].x, d);
                if (CL > GDN_Q) g[j].y = fmaxf(g[j].y, __shfl_xor_sync(0xffffffffu, g[j].y, d));
            }
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (lane == 0 && warp + 8 * j < T) *reinterpret_cast<float2*>(osum + 2 * (warp + 8 * j)) = g[j];
        cluster.sync();
        // every block's sums of the warp's rows, a lane each: lanes [0, 4) and [4, 8) one head's
#pragma unroll
        for (int j = 0; j < N; ++j) g[j] = *reinterpret_cast<const float2*>(cluster.map_shared_rank(osum, lane % CL) + 2 * min(warp + 8 * j, T - 1));
#pragma unroll
        for (int j = 0; j < N; ++j) {
            g[j].x += __shfl_xor_sync(0xffffffffu, g[j].x, 1);
            g[j].x += __shfl_xor_sync(0xffffffffu, g[j].x, 2);
            g[j].x = rsqrtf(g[j].x / (float) GDN_HS + p.eps);
            if (CL > GDN_Q) {
                g[j].y = fmaxf(g[j].y, __shfl_xor_sync(0xffffffffu, g[j].y, 1));
                g[j].y = fmaxf(g[j].y, __shfl_xor_sync(0xffffffffu, g[j].y, 2)) * g[j].x;
                g[j].y = fmaxf(g[j].y, __shfl_xor_sync(0xffffffffu, g[j].y, 4));
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (the neighbours' shared memory is read)
        const int hb = CL > GDN_Q ? (lv & 1) * GDN_Q : 0;   // the head's blocks in the cluster
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int t = warp + 8 * j;
            const float yv = u[j] * __shfl_sync(0xffffffffu, g[j].x, hb);
            if (t >= T) break;
            p.y[(size_t) t * p.nv * GDN_HS + lv * GDN_HS + qq * GDN_QC + lane] = yv;
            if (CL > GDN_Q) {   // the image: the block's 32 columns are a sub-block of it, eight lanes a cell of each level
                uint32_t w1, w2;
                float d;
                ni_code(yv, g[j].y, w1, w2, d);
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
    };
    if constexpr (CL > GDN_Q) results(std::integral_constant<int, 1>{});   // (GDN_PAIR_ROWS at most)
    else if (T <= 8) results(std::integral_constant<int, 1>{});
    else results(std::integral_constant<int, FNX_MAX_ROWS / 8>{});
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // no block may leave while a neighbour still reads its shared memory
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
// engine/src/kernels.cu:2158): conv + SiLU, the q / k norms, the gates and what of the rule does not involve the state, for every group
// of eight rows at once (k_gdn_pre); the delta rule, the only sequential part, with the state in registers from the first row to the last
// (k_gdn_scan); the gated RMS norm of every row at once (k_gdn_post).  Only the last row's state and the last three rows' conv inputs are
// written back.
//
// Row by row, the rule is  S <- g S,  d = beta (v - S' k),  S <- S + k d',  o = S' q / sqrt(128).  Over the rows i = 0 .. 7 of a group
// that starts from S, with b_i = g_0 .. g_i and r_ij = g_(j+1) .. g_i:
//   (I + L) d = w,  w_i = beta_i v_i - beta_i b_i (S' k_i),  L_ij = beta_i r_ij (k_i . k_j), j < i
//   o_i = (b_i (S' q_i) + sum_(j <= i) r_ij (q_i . k_j) d_j) / sqrt(128)
//   S  <- b_7 S + sum_j r_7j k_j d_j'
// so the state is read for all eight rows at once and updated once; (I + L)^-1, which does not involve it, is applied to the k of the update
// beforehand:  sum_j r_7j k_j d_j' = sum_l c_l w_l',  c_l = sum_j r_7j ((I + L)^-1)_jl k_j.  All in f32.
constexpr int GDP_THREADS = 256;
constexpr int GDP_ROWS = 8;
// a group's coefficients for a value head: beta, beta b, b / sqrt(128) [8 each]; b_7; what of o comes from w [8][8]
constexpr int GC_BV = 0, GC_BK = 8, GC_BQ = 16, GC_BC = 24, GC_M = 28, GC_FLOATS = 92;

// grid (groups, key heads + pairs of value heads): a key head's q and k, its dots, and its value heads' coefficients and c; or 256 channels
// of v.  Rows past T become zeros (their coefficients leave the state as it is).  xq / xk [8 groups][nk][HS], xv / xc [..][nv][HS].
// Bound by instructions (the conv's exponentials and divisions; of a key head's the dots of the pairs j <= i alone, a row's norm over a warp in nine shuffles for all
// eight rows) and the chain of a block's four barriers, which the gates' loads and exponentials no longer lie in; a row's inputs are read by one block, eight rows and three before them at a time.
// Six blocks an SM, by 40 registers a thread: 333, 3,001 and 38,912 rows 10.9, 73.6, 916 us, at 64 registers 12.3, 91.6, 1,183, at 32 (with spills) 11.8, 74.9, 925.  One by one: with all
// pairs' dots 11.8, 78.2, 970; with 40 shuffles for the norms 11.7, 77.4, 960; with the gates behind the dots 11.2, 76.1, 956; with two loops for the gates' products 11.2, 75.4,
// 935; with none of these and no bound on the registers 13.4, 98.5, 1,243.  The conv and the norms alone take 750 of the 916, the bytes 490.
__global__ void __launch_bounds__(GDP_THREADS, 6) k_gdn_pre(const float* __restrict__ qkvz, int stride, const float* __restrict__ ab, int ldab,
                                                         const float* __restrict__ hin, float* __restrict__ hout, const float* __restrict__ convw,
                                                         const float* __restrict__ dt, const float* __restrict__ a_, float* __restrict__ xq,
                                                         float* __restrict__ xk, float* __restrict__ xv, float* __restrict__ xc, float* __restrict__ coef, int nk, int nv,
                                                         int T) {
    pdl_begin();
    constexpr int R = GDP_ROWS, HS = GDN_HS, LD = HS + 16;   // (16 banks between neighbouring rows)
    __shared__ __align__(16) float qs[R][LD], ks[R][LD];
    __shared__ float red[GDP_THREADS / 32][R], kk[R][R], qk[R][R], sg[2][R], sb[2][R], Lm[2][R][R], Qm[2][R][R], Ti[2][R][R];
    const int t0 = blockIdx.x * R, y = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ch = (2 * nk + nv) * HS, el = tid & (HS - 1), hf = tid / HS;
    const int c = y < nk ? hf * nk * HS + y * HS + el : 2 * nk * HS + (y - nk) * GDP_THREADS + tid;
    const float4 cw = *reinterpret_cast<const float4*>(convw + (size_t) c * 4);
    float x[R + 3], v[R];   // rows t0 - 3 ..: of this call, or the history it starts from (rows 0..2, oldest first)
    if (t0 >= 3 && t0 + R <= T) {
        const float* src = qkvz + (size_t) (t0 - 3) * stride + c;
#pragma unroll
        for (int i = 0; i < R + 3; ++i) x[i] = src[(size_t) i * stride];
    } else {
#pragma unroll
        for (int i = 0; i < R + 3; ++i) {
            const int r = t0 - 3 + i;
            x[i] = r < 0 ? hin[(size_t) (3 + r) * ch + c] : r < T ? qkvz[(size_t) r * stride + c] : 0.f;
        }
    }
    auto gates = [&](int lv) {   // a value head's: one half block's head each, eight rows
        if (el < R && lv < nv) {
            const int t = t0 + el;
            const float* abt = ab + (size_t) t * ldab;
            float g = 1.f, b = 0.f;
            if (t < T) {
                const float p = abt[lv] + dt[lv];
                g = expf((p > 20.0f ? p : log1pf(expf(p))) * a_[lv]);
                b = 1.0f / (1.0f + expf(-abt[nv + lv]));
            }
            sg[hf][el] = g;
            sb[hf][el] = b;
        }
    };
    if (y < nk) gates(y + hf * nk);   // (their loads' way is that of the rows')
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const float s = cw.x * x[i] + cw.y * x[i + 1] + cw.z * x[i + 2] + cw.w * x[i + 3];
        v[i] = t0 + i < T ? s / (1.0f + expf(-s)) : 0.f;
    }
    if (t0 + R >= T) {   // the history the next call starts from: rows T - 3 .. T - 1
#pragma unroll
        for (int i = 1; i < R + 3; ++i) {
            const int k = t0 - 3 + i - (T - 3);
            if (k >= 0 && k < 3) hout[(size_t) k * ch + c] = x[i];
        }
    }
    if (y >= nk) {
        float* dst = xv + (size_t) t0 * nv * HS + (y - nk) * GDP_THREADS + tid;
#pragma unroll
        for (int i = 0; i < R; ++i) dst[(size_t) i * nv * HS] = v[i];
        return;
    }
    {   // the squares' sums over the warp, all rows at once: at each of three steps a lane keeps the half of its rows that its lane number names
        float sq[R];
#pragma unroll
        for (int i = 0; i < R; ++i) sq[i] = v[i] * v[i];
#pragma unroll
        for (int o = 16, n = R / 2; n >= 1; o >>= 1, n >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float keep = up ? sq[i + n] : sq[i], give = up ? sq[i] : sq[i + n];
                sq[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], 2);
        sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], 1);
        static_assert(R == 8, "lanes 16, 8 and 4 name the row");
        if ((lane & 3) == 0) red[warp][lane >> 2] = sq[0];
    }
    __syncthreads();
    {
        float* dst = (hf ? xk : xq) + ((size_t) t0 * nk + y) * HS + el;
        float (*own)[LD] = hf ? ks : qs;
        const int w0 = warp & ~3;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float n = v[i] * rsqrtf(((red[w0][i] + red[w0 + 1][i]) + red[w0 + 2][i]) + red[w0 + 3][i] + 1e-6f);
            dst[(size_t) i * nk * HS] = n;
            own[i][el] = n;
        }
    }
    __syncthreads();
    if (tid < 4 * R * (R + 1) / 2) {   // four threads a pair of rows j <= i (the others' have no part in anything)
        const int pr = tid >> 2, i = (pr >= 1) + (pr >= 3) + (pr >= 6) + (pr >= 10) + (pr >= 15) + (pr >= 21) + (pr >= 28), j = pr - i * (i + 1) / 2, e0 = (tid & 3) * 4;
        const unsigned live = tid < 128 ? 0xffffffffu : 0xffffu;   // four warps and half of the fifth
        static_assert(4 * R * (R + 1) / 2 == 128 + 16, "the lanes above");
        float dk = 0.f, dq = 0.f;
#pragma unroll
        for (int m = 0; m < HS / 16; ++m) {
            const float4 a = *reinterpret_cast<const float4*>(&ks[i][e0 + 16 * m]), b = *reinterpret_cast<const float4*>(&qs[i][e0 + 16 * m]),
                         k = *reinterpret_cast<const float4*>(&ks[j][e0 + 16 * m]);
            dk = fmaf(a.x, k.x, fmaf(a.y, k.y, fmaf(a.z, k.z, fmaf(a.w, k.w, dk))));
            dq = fmaf(b.x, k.x, fmaf(b.y, k.y, fmaf(b.z, k.z, fmaf(b.w, k.w, dq))));
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            dk += __shfl_xor_sync(live, dk, o);
            dq += __shfl_xor_sync(live, dq, o);
        }
        if ((tid & 3) == 0) {
            kk[i][j] = dk;
            qk[i][j] = dq;
        }
    }
    const float scale = rsqrtf((float) HS);
    const int ti = (el >> 3) & 7, tj = el & 7;
    for (int lv0 = y; lv0 < nv; lv0 += 2 * nk) {   // the key head's value heads, one a half block
        const int lv = lv0 + hf * nk;
        const bool on = lv < nv;
        if (lv0 != y) gates(lv);
        __syncthreads();
        auto prod = [&](int a, int b) {   // g_a .. g_b
            float p = 1.f;
            for (int l = a; l <= b; ++l) p *= sg[hf][l];
            return p;
        };
        if (on && el < 32) {   // a warp: two entries of the matrices a lane, then column `el` of the inverse
            const int j = el & 7;
            float pr[2] = {1.f, 1.f};   // g_(j + 1) .. g_i of both in one pass, the gates' loads all at once: a value head's chain is every further one's wait
#pragma unroll
            for (int l = 1; l < R; ++l) {
                const float g = l > j ? sg[hf][l] : 1.f;
                if (l <= (el >> 3)) pr[0] *= g;
                if (l <= (el >> 3) + 4) pr[1] *= g;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = (el >> 3) + 4 * h;
                const float r = j <= i ? pr[h] : 0.f;
                Lm[hf][i][j] = j < i ? sb[hf][i] * r * kk[i][j] : 0.f;
                Qm[hf][i][j] = j <= i ? scale * r * qk[i][j] : 0.f;
            }
            __syncwarp();
            if (el < R) {
                float t[R];
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    float a = i == el ? 1.f : 0.f;
#pragma unroll
                    for (int j = 0; j < i; ++j) a = fmaf(-Lm[hf][i][j], t[j], a);
                    t[i] = i < el ? 0.f : a;
                    Ti[hf][i][el] = t[i];
                }
            }
        }
        __syncthreads();
        if (on) {
            float* dst = coef + ((size_t) blockIdx.x * nv + lv) * GC_FLOATS;
            if (el < 64) {
                float m = 0.f;   // (rows after ti have no part in it: what is not finite in them stays there)
#pragma unroll
                for (int j = 0; j < R; ++j) m = fmaf(Qm[hf][ti][j], j <= ti ? Ti[hf][j][tj] : 0.f, m);
                dst[GC_M + el] = m;
            } else if (el < 64 + GC_M) {
                const int u = el - 64, i = u & 7;
                dst[u] = u < GC_BK ? sb[hf][i] : u < GC_BQ ? sb[hf][i] * prod(0, i) : u < GC_BC ? scale * prod(0, i) : u == GC_BC ? prod(0, R - 1) : 0.f;
            }
            float cl[R], e = 1.f;
#pragma unroll
            for (int l = 0; l < R; ++l) cl[l] = 0.f;
#pragma unroll
            for (int j = R - 1; j >= 0; --j) {   // e = r_7j
                const float k = e * ks[j][el];
#pragma unroll
                for (int l = 0; l <= j; ++l) cl[l] = fmaf(Ti[hf][j][l], k, cl[l]);
                e *= sg[hf][j];
            }
            float* cd = xc + ((size_t) t0 * nv + lv) * HS + el;
#pragma unroll
            for (int l = 0; l < R; ++l) cd[(size_t) l * nv * HS] = cl[l];
        }
        __syncthreads();
    }
}

// block = (value head, 16 columns), two to an SM so that one's loads and barriers pass while the other works: a warp holds 32 key rows
// of the state in registers, lane = 8 of them (lane / 8) x two columns.  Bound by instructions (some 430 a warp and group) and the
// shared memory's rate: k, q and c are broadcast, two columns a lane halve their loads; then by the chain partial sums -> sums -> w ->
// state between two barriers.  Row by row that chain took 560 cycles a row.  Groups come through three stages of shared memory.
constexpr int GDS_COLS = 16, GDS_STAGES = 3, GDS_PARTS = 2 * GDS_THREADS / 32, GDS_PART = 2 * GDP_ROWS * GDS_COLS + GDS_COLS;   // (the parts 16 banks apart)
constexpr int GDS_K = 0, GDS_QO = GDP_ROWS * GDN_HS, GDS_CO = 2 * GDS_QO, GDS_V = 3 * GDS_QO, GDS_C = GDS_V + GDP_ROWS * GDS_COLS, GDS_STAGE = GDS_C + GC_FLOATS;   // floats
constexpr int GDS_SMEM = (GDS_STAGES * GDS_STAGE + GDS_PARTS * GDS_PART + 4 * GDP_ROWS * GDS_COLS) * (int) sizeof(float);
__global__ void __launch_bounds__(GDS_THREADS, 2) k_gdn_scan(const float* __restrict__ xq, const float* __restrict__ xk, const float* __restrict__ xv,
                                                             const float* __restrict__ xc, const float* __restrict__ coef, const float* __restrict__ S_in,
                                                             float* __restrict__ S_out, float* __restrict__ o, int nk, int nv, int T) {
    constexpr int R = GDP_ROWS, HS = GDN_HS, C = GDS_COLS, SL = HS / C;
    extern __shared__ __align__(16) float gds[];
    float* red = gds + GDS_STAGES * GDS_STAGE;             // [parts][k sums, q sums of 8 rows][columns]
    float* ws = red + GDS_PARTS * GDS_PART;                // [8][columns]
    float2* w2 = reinterpret_cast<float2*>(ws + R * C);    // [2][8][columns / 2]: a lane's two columns, the one whose sums it keeps first
    const int lv = blockIdx.x / SL, col0 = blockIdx.x % SL * C, kh = lv % nk, tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, cp = lane & 7, up = lane >> 4, ng = (T + R - 1) / R;
    const int key0 = warp * 32 + (lane >> 3) * 8, keep = cp + 8 * up, part = warp * 2 + ((lane >> 3) & 1);
    const int row = tid / C, col = tid % C;                // of the sums that the thread completes
    const size_t soff = (size_t) lv * HS * HS + (size_t) key0 * HS + col0;
    uint64_t s[2][4];   // the thread's 16 state values: its column `keep` and the other, key rows (2 i, 2 i + 1)
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[c][i] = f2_pack(S_in[soff + (size_t) (2 * i) * HS + (keep ^ (8 * c))], S_in[soff + (size_t) (2 * i + 1) * HS + (keep ^ (8 * c))]);
    // the thread's 16-byte pieces of a stage: a piece of two rows of k, q and c each, and a few of v and the coefficients
    const int pr = tid >> 5, pe = lane * 4;
    const uint32_t tile_s = smem_u32(gds) + tid * 16;
    const float* gk = xk + ((size_t) pr * nk + kh) * HS + pe;
    const float* gq = xq + ((size_t) pr * nk + kh) * HS + pe;
    const float* gc = xc + ((size_t) pr * nv + lv) * HS + pe;
    const float* gv = tid < R * C / 4 ? xv + ((size_t) (tid / (C / 4)) * nv + lv) * HS + col0 + tid % (C / 4) * 4 : coef + (size_t) lv * GC_FLOATS + (tid - R * C / 4) * 4;
    const size_t kstep = (size_t) R * nk * HS, cstep = (size_t) R * nv * HS, vstep = tid < R * C / 4 ? cstep : (size_t) nv * GC_FLOATS;
    const bool has_v = tid < R * C / 4 + GC_FLOATS / 4;
    auto cp16 = [](uint32_t dst, const float* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); };
    auto stage = [&](int g) {
        if (g < ng) {
            const uint32_t d = tile_s + g % GDS_STAGES * (GDS_STAGE * 4);
            cp16(d, gk); cp16(d + 2048, gk + (size_t) 4 * nk * HS);
            cp16(d + GDS_QO * 4, gq); cp16(d + GDS_QO * 4 + 2048, gq + (size_t) 4 * nk * HS);
            cp16(d + GDS_CO * 4, gc); cp16(d + GDS_CO * 4 + 2048, gc + (size_t) 4 * nv * HS);
            if (has_v) cp16(d + GDS_V * 4, gv);
            gk += kstep; gq += kstep; gc += cstep; gv += vstep;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    static_assert(GDS_THREADS == GDP_ROWS * GDS_COLS && GDS_THREADS * 4 == 4 * GDN_HS && GDS_C == GDS_V + GDP_ROWS * GDS_COLS, "the pieces above");
#pragma unroll
    for (int g = 0; g < GDS_STAGES - 1; ++g) stage(g);
    asm volatile("cp.async.wait_group %0;" ::"n"(GDS_STAGES - 2) : "memory");
    __syncthreads();
    float* od = o + ((size_t) row * nv + lv) * HS + col0 + col;
    const size_t ostep = (size_t) R * nv * HS;
#pragma unroll 1
    for (int g = 0; g < ng; ++g, od += ostep) {
        const float* tl = gds + g % GDS_STAGES * GDS_STAGE;
        float* rp = red + part * GDS_PART + keep;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(tl + GDS_K + i * HS + key0), k1 = *reinterpret_cast<const ulonglong2*>(tl + GDS_K + i * HS + key0 + 4);
            const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(tl + GDS_QO + i * HS + key0), q1 = *reinterpret_cast<const ulonglong2*>(tl + GDS_QO + i * HS + key0 + 4);
            float ks[2], qs[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint64_t ka = f2_fma(s[c][3], k1.y, f2_fma(s[c][2], k1.x, f2_fma(s[c][1], k0.y, f2_mul(s[c][0], k0.x))));
                const uint64_t qa = f2_fma(s[c][3], q1.y, f2_fma(s[c][2], q1.x, f2_fma(s[c][1], q0.y, f2_mul(s[c][0], q0.x))));
                float lo, hi;
                f2_unpack(ka, lo, hi);
                ks[c] = lo + hi;
                f2_unpack(qa, lo, hi);
                qs[c] = lo + hi;
            }
            // another eight key rows' sums of the column this lane keeps
            rp[i * C] = ks[0] + __shfl_xor_sync(0xffffffffu, ks[1], 16);
            rp[(R + i) * C] = qs[0] + __shfl_xor_sync(0xffffffffu, qs[1], 16);
        }
        __syncthreads();
        stage(g + GDS_STAGES - 1);   // (into the slot of the group before: its last readers passed the barrier above)
        const float* cf = tl + GDS_C;
        float ksw = 0.f, qsw = 0.f;
#pragma unroll
        for (int p = 0; p < GDS_PARTS; ++p) {
            ksw += red[p * GDS_PART + row * C + col];
            qsw += red[p * GDS_PART + (R + row) * C + col];
        }
        {
            const float w = cf[GC_BV + row] * tl[GDS_V + row * C + col] - cf[GC_BK + row] * ksw;
            const int h = col >> 3;
            ws[row * C + col] = w;
            (&w2[row * 8 + (col & 7)].x)[h] = w;
            (&w2[(R + row) * 8 + (col & 7)].x)[h ^ 1] = w;
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(GDS_STAGES - 2) : "memory");   // the next group is in
        __syncthreads();
        const float bc = cf[GC_BC];
        const uint64_t bc2 = f2_pack(bc, bc);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int p = 0; p < 4; ++p) s[c][p] = f2_mul(bc2, s[c][p]);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float2 w = w2[(up * R + i) * 8 + cp];
            const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(tl + GDS_CO + i * HS + key0), c1 = *reinterpret_cast<const ulonglong2*>(tl + GDS_CO + i * HS + key0 + 4);
            const uint64_t wx = f2_pack(w.x, w.x), wy = f2_pack(w.y, w.y);
            s[0][0] = f2_fma(c0.x, wx, s[0][0]); s[0][1] = f2_fma(c0.y, wx, s[0][1]); s[0][2] = f2_fma(c1.x, wx, s[0][2]); s[0][3] = f2_fma(c1.y, wx, s[0][3]);
            s[1][0] = f2_fma(c0.x, wy, s[1][0]); s[1][1] = f2_fma(c0.y, wy, s[1][1]); s[1][2] = f2_fma(c1.x, wy, s[1][2]); s[1][3] = f2_fma(c1.y, wy, s[1][3]);
        }
        {
            const float4 m0 = *reinterpret_cast<const float4*>(cf + GC_M + row * R), m1 = *reinterpret_cast<const float4*>(cf + GC_M + row * R + 4);
            const float m[R] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            float a = cf[GC_BQ + row] * qsw;
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (j <= row) a = fmaf(m[j], ws[j * C + col], a);   // (m is 0 beyond, w need not be finite there)
            if (g * R + row < T) *od = a;
        }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float x, y;
            f2_unpack(s[c][i], x, y);
            S_out[soff + (size_t) (2 * i) * HS + (keep ^ (8 * c))] = x;
            S_out[soff + (size_t) (2 * i + 1) * HS + (keep ^ (8 * c))] = y;
        }
}

// block = one row, warp = a value head at a time, four columns a lane: y = o * rsqrt(mean(o^2) + eps) * nw * sigmoid(z).  Bound by its reads and
// writes; four heads' loads are in flight together (a quarter of a head a warp, with two barriers per 256 columns: 44 us for 3,001 rows, 27 now).
// VEC: the caller's rows lie on 16-byte boundaries.
template <bool VEC>
__device__ __forceinline__ float4 gdp_load4(const float* p) {
    return VEC ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
template <bool VEC>
__global__ void __launch_bounds__(GDP_THREADS) k_gdn_post(const float* __restrict__ o, const float* __restrict__ qkvz, int stride, const float* __restrict__ nw,
                                                          float* __restrict__ y, int nk, int nv, float eps) {
    pdl_begin();
    constexpr int HEADS = 4, WARPS = GDP_THREADS / 32;
    static_assert(GDN_HS == 128, "four columns a lane");
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* orow = o + (size_t) t * nv * GDN_HS + lane * 4;
    const float* zrow = qkvz + (size_t) t * stride + (2 * nk + nv) * GDN_HS + lane * 4;
    float* yrow = y + (size_t) t * nv * GDN_HS + lane * 4;
    const float4 w = gdp_load4<VEC>(nw + lane * 4);
    for (int h0 = warp; h0 < nv; h0 += HEADS * WARPS) {
        float4 a[HEADS], z[HEADS];
#pragma unroll
        for (int j = 0; j < HEADS; ++j) {
            const int h = min(h0 + j * WARPS, nv - 1);
            a[j] = gdp_load4<true>(orow + (size_t) h * GDN_HS);
            z[j] = gdp_load4<VEC>(zrow + (size_t) h * GDN_HS);
        }
#pragma unroll
        for (int j = 0; j < HEADS; ++j) {
            const int h = h0 + j * WARPS;
            const float r = rsqrtf(warp_sum(a[j].x * a[j].x + a[j].y * a[j].y + (a[j].z * a[j].z + a[j].w * a[j].w)) / (float) GDN_HS + eps);
            if (h < nv) {
                float4 v;
                v.x = a[j].x * r * w.x / (1.0f + expf(-z[j].x));
                v.y = a[j].y * r * w.y / (1.0f + expf(-z[j].y));
                v.z = a[j].z * r * w.z / (1.0f + expf(-z[j].z));
                v.w = a[j].w * r * w.w / (1.0f + expf(-z[j].w));
                float* d = yrow + (size_t) h * GDN_HS;
                if (VEC) *reinterpret_cast<float4*>(d) = v;
                else { d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w; }
            }
        }
    }
}

static constexpr size_t gdn_smem_bytes(int T, bool tree) {
    return sizeof(float) * ((size_t) 2 * T * GDN_HS + (size_t) 6 * T * GDN_QC + 8 * GDN_QC + ((6 * T + 3) & ~3) +
                            (gdn_staged(T, tree) ? (size_t) (T + 3) * GDN_CHANS + 4 * T : 0));
}
constexpr int GDN_SMEM = 112 * 1024;
// The clusters are placed by load balancing.  The blocks start while the projection's leave (two of these or one and one of those to an SM), and by the default
// policy, which spreads a cluster over SMs, one or two of the 32 clusters of eight of two lanes (33 fit at once) then wait for the first ones' end.
// Windows of twelve layers, us, by the default policy and by this one: lanes of 1 and 2 rows 624 and 603, 2 and 2 668 and 647; a tree of 20 1,389 and 1,382; none slower.
static_assert(gdn_smem_bytes(FNX_MAX_ROWS, true) <= GDN_SMEM, "the most rows fit, two blocks an SM");
static_assert(FNX_MAX_ROWS <= 32 && FNX_MAX_ROWS % 8 == 0 && 2 + (FNX_MAX_ROWS - 1) / GDN_BATCH < 16, "a lane a row's gates, eight warps of results, named barriers");

// An image needs the two heads of its 256-column blocks in one cluster: clusters of eight, whose warps finish a row each.  A kernel for the image takes 1.4 us; more rows, or
// very many clusters whose blocks wait for one another in eights, cost more than that.  Windows, us, in clusters of eight and in two kernels: of twelve layers with 32 value heads,
// 1 and 8 rows (16 clusters) 499 and 505, 832 and 841, lanes of 1 and 2 rows and of 2 and 2 (32) 603 and 614, 647 and 655, eight of one (128) 928 and 929; of eight DeltaNet layers with 64
// value heads, lanes of 4 and 4 rows (64) 548 and 560, four, six and eight of one (128, 192, 256) 511 and 518, 630 and 628, 720 and 697; with 16, 8 rows (8) 497 and 503.
// (A form of the clusters of eight for more rows: chains of 9 to 24 rows 3 to 10 us faster, of 1 to 5 up to 3 us slower, with 128 value heads 4 to 10 slower.)
constexpr int GDN_PAIR_ROWS = 8, GDN_PAIR_CLUSTERS = 128;
static_assert(GDN_PAIR_ROWS <= 8, "clusters of eight give a row to each of a block's warps");
static bool gdn_apart(const GdnArgs& p, int n_lanes, int rows) { return p.img && (rows > GDN_PAIR_ROWS || p.nv / 2 * n_lanes > GDN_PAIR_CLUSTERS); }
int gdn_window(const GdnArgs& p0, const int* cur, bool early, cudaStream_t st) {
    GdnArgs p = p0;
    const bool apart = gdn_apart(p, 1, p.T);
    if (apart) p.img = nullptr;
    auto kernel = p.img ? k_gdn_core<2 * GDN_Q> : k_gdn_core<GDN_Q>;
    FNX_TRY(set_smem_limit((const void*) kernel, GDN_SMEM, true));
    const cudaError_t le = launch_dep(early, kernel, dim3(p.nv * GDN_Q), dim3(GDN_THREADS), gdn_smem_bytes(p.T, p.parent != nullptr), st, p, cur);
    if (le != cudaSuccess) return fail(FNX_E_CUDA, "k_gdn_core: launch failed: %s", cudaGetErrorString(le));
    return apart ? nat_rows_image(p.y, p.nv * GDN_HS, p.T, p.nv * GDN_HS, nullptr, p0.img, st) : FNX_OK;
}
int gdn_window_lanes(const GdnArgs& p0, size_t hist_seq_stride, size_t s_seq_stride, const int* cur, const int* lane_seq, const int* lane_row0, int n_lanes, int max_rows,
                     int rows, bool early, cudaStream_t st) {
    GdnArgs p = p0;
    const bool apart = gdn_apart(p, n_lanes, rows);
    if (apart) p.img = nullptr;
    auto kernel = p.img ? k_gdn_core_lanes<2 * GDN_Q> : k_gdn_core_lanes<GDN_Q>;
    FNX_TRY(set_smem_limit((const void*) kernel, GDN_SMEM, true));
    const cudaError_t le = launch_dep(early, kernel, dim3(p.nv * GDN_Q, n_lanes), dim3(GDN_THREADS), gdn_smem_bytes(max_rows, false), st, p, hist_seq_stride, s_seq_stride, cur,
                                      lane_seq, lane_row0);
    if (le != cudaSuccess) return fail(FNX_E_CUDA, "k_gdn_core_lanes: launch failed: %s", cudaGetErrorString(le));
    return apart ? nat_rows_image(p.y, p.nv * GDN_HS, rows, p.nv * GDN_HS, nullptr, p0.img, st) : FNX_OK;
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
    const size_t ng = ((size_t) T + GDP_ROWS - 1) / GDP_ROWS;
    return sizeof(float) * (ng * GDP_ROWS * (2 * nk + 3 * nv) * hs + ng * nv * GC_FLOATS + (size_t) 3 * (2 * nk + nv) * hs) + 1024;
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
    const int ng = (T + GDP_ROWS - 1) / GDP_ROWS;
    const size_t Tp = (size_t) ng * GDP_ROWS;
    float* xq = (float*) (((uintptr_t) scratch + 15) & ~(uintptr_t) 15);   // (16-byte pieces; the spare bytes of the scratch leave room to align)
    float* xk = xq + Tp * nk * GDN_HS;
    float* xv = xk + Tp * nk * GDN_HS;
    float* xc = xv + Tp * nv * GDN_HS;
    float* o = xc + Tp * nv * GDN_HS;
    float* coef = o + (size_t) T * nv * GDN_HS;
    cudaStream_t s = as_stream(st);
    // the history the call starts from is read from a copy where the slot that it leaves its own in is the same one
    const float* hin = hist_pool + (size_t) cur_host * hsz;
    if (out_slot == cur_host) {
        float* copy = coef + (size_t) ng * nv * GC_FLOATS;
        FNX_CUDA_OK(cudaMemcpyAsync(copy, hin, hsz * sizeof(float), cudaMemcpyDeviceToDevice, s));
        hin = copy;
    }
    FNX_CUDA_OK(launch_after(k_gdn_pre, dim3(ng, nk + nv * GDN_HS / GDP_THREADS), dim3(GDP_THREADS), 0, s, qkvz, ldx, ab, ldab, hin, hist_pool + (size_t) out_slot * hsz, convw, dt, a, xq, xk, xv, xc,
                                                                               coef, nk, nv, T));
    FNX_LAUNCH_OK("k_gdn_pre");
    FNX_TRY(set_smem_limit((const void*) k_gdn_scan, GDS_SMEM));
    // (not ahead of its predecessor's end: blocks that fill the SMs as these come free sit three to some and one to others, 600 us instead of 440 for 3,001 rows)
    FNX_CUDA_OK(launch_dep(false, k_gdn_scan, dim3(nv * (GDN_HS / GDS_COLS)), dim3(GDS_THREADS), GDS_SMEM, s, xq, xk, xv, xc, coef, S_pool + (size_t) cur_host * ssz, S_pool + (size_t) out_slot * ssz, o, nk, nv, T));
    FNX_LAUNCH_OK("k_gdn_scan");
    const bool vec = ldx % 4 == 0 && (((uintptr_t) qkvz | (uintptr_t) nw | (uintptr_t) y) & 15) == 0;
    FNX_CUDA_OK(launch_after(vec ? k_gdn_post<true> : k_gdn_post<false>, dim3(T), dim3(GDP_THREADS), 0, s, o, qkvz, ldx, nw, y, nk, nv, eps));
    FNX_LAUNCH_OK("k_gdn_post");
    return FNX_OK;
}

extern "C" int fnx_gdn_core_lanes(const float* qkvz, int ldx, const float* ab, int ldab, float* hist_pool, size_t hist_seq_stride, const float* convw,
                                  const float* dt, const float* a, const float* nw, float* S_pool, size_t s_seq_stride, const int* cur, int NS,
                                  const int* lane_seq, const int* lane_row0, int n_lanes, int max_lane_rows, float* y, int nk, int nv, int hs, float eps,
                                  fnx_stream st) {
    FNX_REQUIRE(qkvz && ab && hist_pool && convw && dt && a && nw && S_pool && cur && lane_seq && lane_row0 && y, "fnx_gdn_core_lanes: null pointer");
    FNX_REQUIRE(hs == GDN_HS, "fnx_gdn_core_lanes: head dim %d (this build: %d)", hs, GDN_HS);
    FNX_REQUIRE(n_lanes >= 1 && n_lanes <= FNX_MAX_ROWS && max_lane_rows >= 1 && max_lane_rows <= FNX_MAX_ROWS && NS >= max_lane_rows + 1,
                "fnx_gdn_core_lanes: %d lanes of up to %d rows, %d state slots", n_lanes, max_lane_rows, NS);
    FNX_REQUIRE(nk >= 1 && nv >= nk && nv % nk == 0, "fnx_gdn_core_lanes: %d key heads, %d value heads", nk, nv);
    return gdn_window_lanes(GdnArgs{qkvz, ldx, ab, ldab, hist_pool, convw, dt, a, nw, S_pool, NS, nullptr, y, nullptr, nk, nv, max_lane_rows, eps}, hist_seq_stride,
                            s_seq_stride, cur, lane_seq, lane_row0, n_lanes, max_lane_rows, 0, false, as_stream(st));
}
