// Attention of a decode window over its sequences' caches, split over positions: the window form of attn / k_attn_part + k_attn_local +
// k_attn_combine (engine/src/kernels.hpp:238, engine/src/kernels.cu:558-667, 786-803), on the 5th-generation tensor cores.
//
// What bounds it: the K and V rows, read once for all of the window's rows (a KV head's eight query heads x up to sixteen rows =
// 128 score rows = tensor-memory lanes).  An SM's share of the memory's rate is 64 positions of one KV head (64 KB) in about 2,850
// cycles; the products of such a step take about 1,550 (scores 2 x 16 tcgen05.mma M128 N64 K16, sums 4 x M128 N256 K16), its softmax
// about as long as one of them, and they overlap.  The mma.sync form before it re-read the queries' operands from shared memory in every
// warp and ran its phases one after another.
//
//   scores  = Q K^T with Q = Qhi + Qlo, two f16 halves of the f32 queries (Qhi in shared memory, Qlo in tensor memory), so that only
//             K's own f16 rounding remains;
//   weights = exp(score - running max), rounded to f16 (their sum is taken over the rounded values), left in tensor memory over
//             their scores: the next product's A operand;
//   sums   += weights V, accumulated in f32 tensor memory across the steps.
//
// Split s of S takes the 64-position chunks s, s + S, ... in order.  Chunks are cut at absolute positions and S is fixed, so what a row's
// partial of a split sums, and in which order, depends on the row's own position only: a row verified alone and the same row verified
// among drafts give the same bits.  A block walks its items (lane, split, KV head, 128-row tile); the loader runs ahead of the item that
// is computed, across items.
#include "attn_core.cuh"
#include "attn_tc.cuh"
#include "attn_win.h"
#include "nat_image.cuh"

namespace fnxb {

constexpr int AW_M = 128, AW_N = ATC_N, AW_HD = ATC_HD;
constexpr int AW_SOFT = 256;                    // warps 0-7: two threads per score row (a half of the step's positions, of the row's dims)
constexpr int AW_LOAD = 128;                    // warps 8-11: the loader (one thread; all of them for the chunk that a context ends in)
constexpr int AW_THREADS = AW_SOFT + AW_LOAD + 32;   // warp 12: the products
constexpr int AW_RING = 5;                      // tiles of 64 positions, K and V in turn
constexpr int AW_BOX = AW_N * 128;              // a box of 64 dims: 64 positions x 128 bytes, 128-byte swizzle
constexpr int AW_TILE = (AW_HD / 64) * AW_BOX;  // 32 KB
constexpr int AW_QBOX = AW_M * 128;             // Qhi: four such boxes of 128 rows
constexpr int AW_SBO = 8 * 128;                 // between 8-row groups
constexpr int AW_HEAD = 3072;                   // barriers, tables, the halves' exchange
constexpr int AW_SMEM = AW_HEAD + AW_RING * AW_TILE + 4 * AW_QBOX;
static_assert(AW_SMEM <= 227 * 1024, "the tiles fit one block's shared memory");
// tensor memory columns: the sums, the queries' low halves, two steps' scores
constexpr uint32_t AW_O = 0, AW_QLO = 256, AW_S = 384;
constexpr int AW_TMEM_COLS = 512;

struct AwShared {
    uint64_t full[AW_RING], empty[AW_RING];
    uint64_t bar_s[2], bar_p[2], bar_o, bar_q;
    uint32_t tmem;
    volatile int gave_up;
    unsigned see[32];                   // one sequence: per window row the rows it sees
    int first[FNX_MAX_ROWS + 1];        // lanes: their first items
    int pos[FNX_MAX_ROWS];
    float xch[2][2][AW_M];              // [step parity][half][row]
};
static_assert(sizeof(AwShared) <= AW_HEAD, "the head fits");

__device__ __forceinline__ bool aw_wait(uint64_t* bar, unsigned parity, AwShared& S) { return ta_wait_for(bar, parity, S.gave_up); }

struct AwItem {
    int lane, row0, nr, kvh, s, n, ctx, pos0;   // rows [row0, row0 + nr) of the window; n steps
    long long seq_row;                          // the sequence's first cache row
};

// grid: one block an SM.  Five rows over 32,768 positions, with the merge: 53 -> 27 us (2.5 TB/s of cache rows); 20 rows in 4 lanes over
// 131,072: 4.0 TB/s in the steps, whose 2,850 cycles are the memory's share.  A short context is bound by the item's own chain (queries in,
// scores, weights, sums, results out: about 8 us).
__global__ void __launch_bounds__(AW_THREADS, 1) k_attn_win(const AttnWin a, float* __restrict__ acc_out, AttPartial* __restrict__ mz_out, int S,
                                                           const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v) {
    extern __shared__ __align__(1024) uint8_t smem[];
    AwShared& sh = *reinterpret_cast<AwShared*>(smem);
    uint8_t* ring = smem + AW_HEAD;
    uint8_t* Qs = ring + AW_RING * AW_TILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (smem_u32(smem) & 1023u) {   // the swizzled tiles need their 1,024-byte boundary
        pdl_wait();
        if (tid == 0 && a.err) atomicOr(a.err, (unsigned) FNX_ERR_TIMEOUT);
        return;
    }
    const int qpk = a.nq / a.nkv, RT = min(AW_M / qpk, (int) FNX_MAX_ROWS);   // window rows of a tile
    const int nl = a.lane_seq ? a.n_lanes : 1;
    if (tid < 32) {   // the lanes' items
        int items = 0, pos = 0;
        if (lane < nl) {
            const int seq = a.lane_seq ? a.lane_seq[lane] : 0, rows = a.lane_seq ? a.lane_row0[lane + 1] - a.lane_row0[lane] : a.T;
            if (rows > 0 && seq >= 0) {
                pos = a.pos[seq];
                items = min(S, (pos + rows + AW_N - 1) / AW_N) * a.nkv * ((rows + RT - 1) / RT);
            }
            sh.pos[lane] = pos;
        }
        int sum = items;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        sh.first[lane + 1] = sum;
        if (lane == 0) sh.first[0] = 0;
    } else if (tid < 64) {   // one sequence: the window rows on each row's path to the root
        const int t = lane;
        const int p = t < a.T && !a.lane_seq ? (a.parent ? a.parent[t] : t - 1) : -1;
        unsigned m = 0;
        int at = t < a.T ? t : -1;
        for (int i = 0; i < FNX_MAX_ROWS; ++i) {
            if (at >= 0) m |= 1u << at;
            const int up = __shfl_sync(0xffffffffu, p, at & 31);
            at = at >= 0 ? up : -1;
        }
        sh.see[t] = m;
    } else if (tid == 64) {
        for (int i = 0; i < AW_RING; ++i) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.bar_s[i], 1);
            mbar_init(&sh.bar_p[i], AW_SOFT / 32);
        }
        mbar_init(&sh.bar_o, 1);
        mbar_init(&sh.bar_q, AW_SOFT / 32);
        sh.gave_up = 0;
        fence_barrier_init();
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(AW_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ta_fence_before();
    __syncthreads();
    ta_fence_after();
    const uint32_t tmem = sh.tmem;
    const int total = sh.first[nl];
    const float inv_kv = __fdividef(1.0f, (float) a.nkv), inv_s = __fdividef(1.0f, (float) S);
    int cur = 0;
    auto item_of = [&](int it) {
        AwItem x;
        while (it >= sh.first[cur + 1]) ++cur;
        x.lane = cur;
        const int r0 = a.lane_seq ? a.lane_row0[cur] : 0, rows = a.lane_seq ? a.lane_row0[cur + 1] - r0 : a.T, tiles = (rows + RT - 1) / RT;
        // (quotients below 2^20: exact in f32 with the half added)
        const int local = it - sh.first[cur], rest = (int) (((float) local + 0.5f) * __fdividef(1.0f, (float) tiles)), tile = local - rest * tiles;
        x.s = (int) (((float) rest + 0.5f) * inv_kv);
        x.kvh = rest - x.s * a.nkv;
        x.pos0 = sh.pos[cur];
        x.ctx = x.pos0 + rows;
        x.row0 = r0 + tile * RT;
        x.nr = min(RT, rows - tile * RT);
        x.n = (int) (((float) ((x.ctx + AW_N - 1) / AW_N - x.s + S - 1) + 0.5f) * inv_s);
        x.seq_row = a.lane_seq ? (long long) a.lane_seq[cur] * (long long) a.seq_rows : 0;
        return x;
    };
    if (warp >= 8 && warp < 12) {
        // ---------------------------------------------------------------------------------------- the loader
        const int lt = tid - AW_SOFT;
        bool ok = true, waited = false;
        int n = 0;   // tiles so far
        for (int it = blockIdx.x; it < total; it += gridDim.x) {
            const AwItem x = item_of(it);
            for (int j = 0; j < x.n; ++j) {
                const int p0 = (x.s + j * S) * AW_N, np = min(AW_N, x.ctx - p0);
                const bool whole = np == AW_N;
                if (!waited && p0 + np > x.pos0) {   // the window's own rows: what the kernel before this one wrote
                    pdl_wait();
                    waited = true;
                }
                if (whole) {
                    if (lt == 0) {
#pragma unroll
                        for (int kv = 0; kv < 2; ++kv) {
                            const int slot = (n + kv) % AW_RING;
                            if (ok && n + kv >= AW_RING) ok = aw_wait(&sh.empty[slot], (unsigned) (((n + kv) / AW_RING - 1) & 1), sh);
                            if (!ok) break;
                            mbar_expect_tx(&sh.full[slot], AW_TILE);
#pragma unroll
                            for (int c = 0; c < AW_HD / 64; ++c)
                                ta_tma_3d(smem_u32(ring + slot * AW_TILE + c * AW_BOX), kv ? &map_v : &map_k, c * 64, x.kvh, (int) (x.seq_row + p0), &sh.full[slot]);
                        }
                    }
                    n += 2;
                    continue;
                }
                // the chunk that the context ends in: 16-byte pieces where the swizzle puts them, the rows past the context zero (every loader
                // takes the barriers, whatever the wait saw; the first alone keeps count of the slots' phases)
                if (lt == 0)
                    for (int kv = 0; kv < 2; ++kv)
                        if (ok && n + kv >= AW_RING) ok = aw_wait(&sh.empty[(n + kv) % AW_RING], (unsigned) (((n + kv) / AW_RING - 1) & 1), sh);
                asm volatile("bar.sync 5, %0;" ::"n"(AW_LOAD) : "memory");
                if (!sh.gave_up) {
                    uint8_t* kd = ring + n % AW_RING * AW_TILE;
                    uint8_t* vd = ring + (n + 1) % AW_RING * AW_TILE;
#pragma unroll
                    for (int i0 = 0; i0 < AW_N * (AW_HD / 8) / AW_LOAD; ++i0) {
                        const int i = lt + i0 * AW_LOAD, rest = i >> 5, r = (rest & 15) * 4 + (i & 3), d8 = (rest >> 4) * 8 + ((i >> 2) & 7);
                        const uint32_t off = (uint32_t) ((d8 >> 3) * AW_BOX + r * 128 + (((d8 & 7) ^ (r & 7)) * 16));
                        if (r < np) {
                            const size_t go = ((size_t) (x.seq_row + p0 + r) * a.nkv + x.kvh) * AW_HD + d8 * 8;
                            cp_async16(kd + off, a.kc + go);
                            cp_async16(vd + off, a.vc + go);
                        } else {
                            *reinterpret_cast<uint4*>(kd + off) = make_uint4(0, 0, 0, 0);
                            *reinterpret_cast<uint4*>(vd + off) = make_uint4(0, 0, 0, 0);
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    fence_proxy_async();   // (the products read it through the async proxy)
                }
                asm volatile("bar.sync 5, %0;" ::"n"(AW_LOAD) : "memory");
                if (lt == 0 && ok) {
                    mbar_arrive(&sh.full[n % AW_RING]);
                    mbar_arrive(&sh.full[(n + 1) % AW_RING]);
                }
                n += 2;
            }
        }
        if (!waited) pdl_wait();
    } else if (warp == 12) {
        // ---------------------------------------------------------------------------------------- the products
        // f32 accumulate, f16 x f16, M = 128; S: both operands K-major, N = 64; O: B (V) MN-major, N = 256
        constexpr uint32_t IDESC_S = (1u << 4) | ((uint32_t) (AW_N >> 3) << 17) | ((uint32_t) (AW_M >> 4) << 24);
        constexpr uint32_t IDESC_O = (1u << 4) | (1u << 16) | ((uint32_t) (AW_HD >> 3) << 17) | ((uint32_t) (AW_M >> 4) << 24);
        const uint32_t q_s = smem_u32(Qs), ring_s = smem_u32(ring);
        bool ok = true;
        int g = 0, nit = 0;   // steps and items so far
        // (the products' operands reach the uniform registers cheaply only under elect.sync: 38 and 56 cycles an issue instead of 76)
        auto scores = [&](int step) {
            const int n = 2 * step, slot = n % AW_RING;
            const uint32_t k_s = ring_s + slot * AW_TILE, tm_s = tmem + AW_S + (uint32_t) (step & 1) * AW_N;
            if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.full[slot], (unsigned) ((n / AW_RING) & 1), sh));
            if (ok && ta_elect()) {
                ta_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < AW_HD / 16; ++k16)
                    ta_mma(tm_s, ta_desc_sw(q_s + (k16 >> 2) * AW_QBOX + (k16 & 3) * 32, 16, AW_SBO), ta_desc_sw(k_s + (k16 >> 2) * AW_BOX + (k16 & 3) * 32, 16, AW_SBO),
                           IDESC_S, k16 != 0);
#pragma unroll
                for (int k16 = 0; k16 < AW_HD / 16; ++k16)
                    ta_mma_ta(tm_s, tmem + AW_QLO + k16 * 8, ta_desc_sw(k_s + (k16 >> 2) * AW_BOX + (k16 & 3) * 32, 16, AW_SBO), IDESC_S, 1);
                ta_commit(&sh.empty[slot]);
                ta_commit(&sh.bar_s[step & 1]);
            }
            __syncwarp();
        };
        for (int it = blockIdx.x; it < total; it += gridDim.x, ++nit) {
            const AwItem x = item_of(it);
            if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.bar_q, (unsigned) (nit & 1), sh));
            scores(g);
            for (int j = 0; j < x.n; ++j, ++g) {
                if (j + 1 < x.n) scores(g + 1);   // (while the softmax of this step runs)
                const int n = 2 * g + 1, slot = n % AW_RING;
                const uint32_t v_s = ring_s + slot * AW_TILE, tm_p = tmem + AW_S + (uint32_t) (g & 1) * AW_N;
                if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.full[slot], (unsigned) ((n / AW_RING) & 1), sh));
                if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.bar_p[g & 1], (unsigned) ((g >> 1) & 1), sh));
                if (ok && ta_elect()) {
                    ta_fence_after();
#pragma unroll
                    for (int k16 = 0; k16 < AW_N / 16; ++k16)
                        ta_mma_ta(tmem + AW_O, tm_p + k16 * 8, ta_desc_sw(v_s + k16 * 2 * AW_SBO, AW_BOX, AW_SBO), IDESC_O, (j | k16) != 0);
                    ta_commit(&sh.empty[slot]);
                    ta_commit(&sh.bar_o);
                }
                __syncwarp();
            }
        }
        pdl_wait();
    } else {
        // ---------------------------------------------------------------------------------------- queries, softmax, results
        pdl_wait();
        if (tid == 0) pdl_launch_dependents();
        const int r = (warp & 3) * 32 + lane, half = warp >> 2;   // the thread's score row, its half
        const uint32_t lane_base = (uint32_t) (32 * (warp & 3)) << 16;
        const unsigned pair_bar = 1u + (unsigned) (warp & 3);     // the row group's two warps
        const int qinv = (65536 + qpk - 1) / qpk;                 // q / qpk = q qinv >> 16 for q < 128
        const float scale2 = 0.0625f * 1.4426950408889634f;       // 1 / sqrt(256) x log2 e: the scores in the base-2 domain
        bool ok = true;
        int g = 0;
        for (int it = blockIdx.x; it < total; it += gridDim.x) {
            const AwItem x = item_of(it);
            const int NQ = x.nr * qpk;
            const bool live_warp = (warp & 3) * 32 < NQ, live = r < NQ;   // (dead rows hold whatever they hold: rows do not mix)
            const int tq = (min(r, NQ - 1) * qinv) >> 16, t = x.row0 + tq, h = x.kvh * qpk + min(r, NQ - 1) - tq * qpk;
            // A warp takes whole rows (1 KB of a query, 8 dims a lane), so the low halves reach their rows' lanes by way of shared memory: the
            // half of Qs that holds no high halves (yet), or for the last 64 rows of a full tile their own place before the high halves take it.
            // (Rolled: each line runs once or twice an item, and fetching straight-line code for it took 15,000 cycles.)
            const int nph = NQ > 64 ? 3 : 1;
#pragma unroll 1
            for (int ph = 0; ph < nph; ++ph) {
                const int q0 = nph == 3 && ph == 0 ? 64 : 0, q1 = q0 ? NQ : min(NQ, 64);       // these rows
                const bool put_hi = ph != 1, put_lo = ph != 2;
                const int to = (nph == 1 ? 64 : q0 ? -64 : 0) * 128;                            // their low halves' place, from their own
                uint8_t* piece = Qs + (lane >> 3) * AW_QBOX;
#pragma unroll 4
                for (int q = q0 + warp; q < q1; q += 8) {
                    const int qr = (q * qinv) >> 16;
                    const float4* src = reinterpret_cast<const float4*>(a.qg + (size_t) (x.row0 + qr) * a.ldq + (size_t) (x.kvh * qpk + q - qr * qpk) * 2 * AW_HD + lane * 8);
                    const float4 v0 = src[0], v1 = src[1];
                    const float f[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const __half2 hh = __floats2half2_rn(f[2 * k], f[2 * k + 1]);
                        const float2 back = __half22float2(hh);
                        const __half2 ll = __floats2half2_rn(f[2 * k] - back.x, f[2 * k + 1] - back.y);
                        hi[k] = *reinterpret_cast<const uint32_t*>(&hh);
                        lo[k] = *reinterpret_cast<const uint32_t*>(&ll);
                    }
                    uint8_t* at = piece + q * 128 + (((lane & 7) ^ (q & 7)) * 16);
                    if (put_hi) *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    if (put_lo) *reinterpret_cast<uint4*>(at + to) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
                if (!put_lo) break;
                asm volatile("bar.sync 6, %0;" ::"n"(AW_SOFT) : "memory");
                if ((warp & 3) * 32 >= q0 && (warp & 3) * 32 < q1) {
#pragma unroll 1
                    for (int d0 = 0; d0 < 2; ++d0) {   // 64 dims at a time
                        float lf[32];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 w = *reinterpret_cast<const float4*>(Qs + (half * 2 + d0) * AW_QBOX + r * 128 + to + ((i ^ (r & 7)) * 16));
                            lf[4 * i] = w.x; lf[4 * i + 1] = w.y; lf[4 * i + 2] = w.z; lf[4 * i + 3] = w.w;
                        }
                        ta_st32(tmem + AW_QLO + lane_base + (uint32_t) (half * 64 + d0 * 32), lf);
                    }
                    ta_wait_st();
                }
                if (ph + 1 < nph) asm volatile("bar.sync 6, %0;" ::"n"(AW_SOFT) : "memory");
            }
            fence_proxy_async();
            ta_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.bar_q);
            const int my_row = x.row0 - (a.lane_seq ? a.lane_row0[x.lane] : 0) + tq;   // within the sequence's rows
            const unsigned see = a.lane_seq ? (2u << my_row) - 1u : sh.see[my_row];
            float m_run = -INFINITY, z_half = 0.f;
            for (int j = 0; j < x.n; ++j, ++g) {
                const int b = g & 1, p0 = (x.s + j * S) * AW_N;
                if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.bar_s[b], (unsigned) ((g >> 1) & 1), sh));   // (warps without live rows keep step)
                ta_fence_after();
                if (live_warp) {   // (both warps of a row group, or neither)
                    const uint32_t tm_s = tmem + AW_S + (uint32_t) b * AW_N + lane_base;
                    float s[32];
                    float mx = -INFINITY;
                    if (ok) {
                        ta_ld32(tm_s + 32 * half, s);
                        // the positions that the row sees, as bits: all before the window, then its path's
                        const int w = p0 + 32 * half - x.pos0;
                        const unsigned vis = w <= -32 ? ~0u : w < 0 ? (see << -w) | ((1u << -w) - 1u) : w < 32 ? see >> w : 0u;
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            s[i] = (vis >> i) & 1u ? s[i] * scale2 : -INFINITY;
                            mx = fmaxf(mx, s[i]);
                        }
                    }
                    sh.xch[b][half][r] = mx;
                    asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");   // (every thread takes it, whatever its waits saw)
                    if (ok) {
                        const float mn = fmaxf(m_run, fmaxf(mx, sh.xch[b][half ^ 1][r]));
                        const float ms = mn == -INFINITY ? 0.f : mn;   // (a row that sees nothing yet: weights of 0)
                        float sum = 0.f;
                        uint32_t pk[16];
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const __half2 hh = __floats2half2_rn(ta_ex2(s[i] - ms), ta_ex2(s[i + 1] - ms));
                            const float2 back = __half22float2(hh);
                            sum += back.x;
                            sum += back.y;
                            pk[i / 2] = *reinterpret_cast<const uint32_t*>(&hh);
                        }
                        const float f = m_run == -INFINITY ? 0.f : ta_ex2(m_run - ms);
                        z_half = z_half * f + sum;
                        m_run = mn;
                        ta_st16(tm_s + 16 * half, pk);   // over the scores, which both of the row's threads have read
                        // the sums of the step before are complete (no phase is skipped), and rescaled where some row's maximum has moved: deep
                        // into a long context that is rare
                        if (j >= 1) {
                            ok = __all_sync(0xffffffffu, aw_wait(&sh.bar_o, (unsigned) ((g - 1) & 1), sh));
                            ta_fence_after();
                            if (ok && __any_sync(0xffffffffu, f != 1.0f)) {
#pragma unroll 1
                                for (int c32 = 0; c32 < AW_HD / 64; ++c32) {
                                    float o[32];
                                    ta_ld32(tmem + AW_O + lane_base + 128 * half + c32 * 32, o);
#pragma unroll
                                    for (int i = 0; i < 32; ++i) o[i] *= f;
                                    ta_st32(tmem + AW_O + lane_base + 128 * half + c32 * 32, o);
                                }
                            }
                        }
                        ta_wait_st();
                    }
                    ta_fence_before();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.bar_p[b]);
            }
            // the item's partial (the sums of the step before have the other parity's exchange to themselves)
            if (live_warp) {
                if (ok) ok = __all_sync(0xffffffffu, aw_wait(&sh.bar_o, (unsigned) ((g - 1) & 1), sh));
                ta_fence_after();
                float* zx = &sh.xch[g & 1][0][0];
                zx[half * AW_M + r] = z_half;
                asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
                const size_t slot = ((size_t) t * a.nq + h) * S + x.s;
                if (live && half == 0) mz_out[slot] = ok ? AttPartial{m_run, zx[r] + zx[AW_M + r]} : AttPartial{0.f, __int_as_float(0x7fc00000)};
                if (ok) {
                    // 32 dims at a time through the queries' place, so that whole lines leave
                    uint8_t* mine = Qs + warp * 4096;
                    const int w0 = (warp & 3) * 32;
#pragma unroll 1
                    for (int c32 = 0; c32 < AW_HD / 64; ++c32) {
                        float o[32];
                        ta_ld32(tmem + AW_O + lane_base + 128 * half + c32 * 32, o);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            *reinterpret_cast<float4*>(mine + lane * 128 + ((i ^ (lane & 7)) * 16)) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int q = i * 4 + (lane >> 3), c = lane & 7;
                            if (w0 + q < NQ) {
                                const int qr = ((w0 + q) * qinv) >> 16, qh = x.kvh * qpk + w0 + q - qr * qpk;
                                *reinterpret_cast<float4*>(acc_out + ((size_t) ((x.row0 + qr) * a.nq + qh) * S + x.s) * AW_HD + half * (AW_HD / 2) + c32 * 32 + c * 4) =
                                    *reinterpret_cast<const float4*>(mine + q * 128 + ((c ^ (q & 7)) * 16));
                            }
                        }
                        __syncwarp();
                    }
                }
                ta_fence_before();
            }
            asm volatile("bar.sync 6, %0;" ::"n"(AW_SOFT) : "memory");   // (the next item's queries go where other warps' results pass)
        }
    }
    ta_fence_before();
    __syncthreads();
    if (tid == 0 && sh.gave_up && a.err) atomicOr(a.err, (unsigned) FNX_ERR_TIMEOUT);
    if (warp == 12) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(AW_TMEM_COLS) : "memory");
}

// The merge of the splits of (head, row): out = sum_s 2^(m_s - m) acc_s / sum_s 2^(m_s - m) z_s * sigmoid(gate).  Bound by latency: one
// round of loads (every thread's partial sums, four dims of every sixteenth live split, and their maxima) and one exchange; the
// one-dim-a-thread form before it took three rounds behind two barriers (7.3 us after five rows over 32,768 positions).  Groups and
// their order do not depend on how many splits are live: a dead one adds 0.
// TG of the sixteen groups at a time (their sums, and so the bits, are the same): all of them, or four, in blocks of a quarter the size, where
// there are more (head, row) pairs than the SMs hold of the large blocks (two each): 64 heads, 32 rows over 3,000 positions, both kernels: 73 us
// with the large blocks, 53 with these; 16 heads, 32 rows: 37 and 31; 8 heads, 32 rows over 131,000 positions (256 pairs): 76 and 80.
constexpr int AM_GROUPS = 16, AM_BATCH = 5;
template <int TG>
__global__ void __launch_bounds__(TG * 64) k_attn_merge(const float* __restrict__ acc_in, const AttPartial* __restrict__ mz_in, const float* __restrict__ qg, int ldq,
                                                              float* __restrict__ out, uint8_t* __restrict__ img, int T, int nq, int S, const int* __restrict__ pos,
                                                              const int* __restrict__ lane_seq, const int* __restrict__ lane_row0, int n_lanes) {
    __shared__ __align__(16) float part[AM_GROUPS][AW_HD];
    __shared__ __align__(16) float row[AW_HD];
    const int tid = threadIdx.x, lane = tid & 31, d4 = tid & 63, g = tid >> 6, h = blockIdx.x, t = blockIdx.y;
    int live = S;
    bool skip = false;
    if (lane_seq) {
        int j = 0;
        while (j + 1 < n_lanes && t >= lane_row0[j + 1]) ++j;
        const int seq = lane_seq[j];
        skip = seq < 0;   // another rank's lane
        if (!skip) live = min(S, (pos[seq] + lane_row0[j + 1] - lane_row0[j] + AW_N - 1) / AW_N);
    } else live = min(S, (*pos + T + AW_N - 1) / AW_N);
    const float gate = tid < AW_HD && !skip ? qg[(size_t) t * ldq + (size_t) h * 2 * AW_HD + AW_HD + tid] : 0.f;
    pdl_wait();
    pdl_launch_dependents();
    if (skip) return;
    const size_t base = ((size_t) t * nq + h) * S;
    float4 v[AM_BATCH];
    float m[AM_BATCH];
    auto fetch = [&](int gg, int s0) {
#pragma unroll
        for (int i = 0; i < AM_BATCH; ++i) {
            const int s = s0 + gg + i * AM_GROUPS;
            m[i] = -INFINITY;
            if (s < live) {
                m[i] = mz_in[base + s].m;
                v[i] = *reinterpret_cast<const float4*>(acc_in + (base + s) * AW_HD + d4 * 4);
            }
        }
    };
    fetch(g, 0);
    AttPartial p[8];   // (up to 256 splits)
    float mx = -INFINITY, z = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        p[i] = AttPartial{-INFINITY, 0.f};
        if (lane + 32 * i < live) p[i] = mz_in[base + lane + 32 * i];
        mx = fmaxf(mx, p[i].m);
    }
    mx = warp_max(mx);
#pragma unroll
    for (int i = 0; i < 8; ++i) z += p[i].m == -INFINITY ? 0.f : exp2f(p[i].m - mx) * p[i].z;
    z = warp_sum(z);
#pragma unroll 1
    for (int r = 0; r < AM_GROUPS / TG; ++r) {
        const int gg = g + r * TG;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < live; s0 += AM_BATCH * AM_GROUPS) {
            if (s0 || r) fetch(gg, s0);
#pragma unroll
            for (int i = 0; i < AM_BATCH; ++i)
                if (m[i] != -INFINITY) {
                    const float w = exp2f(m[i] - mx);
                    sum.x = fmaf(w, v[i].x, sum.x);
                    sum.y = fmaf(w, v[i].y, sum.y);
                    sum.z = fmaf(w, v[i].z, sum.z);
                    sum.w = fmaf(w, v[i].w, sum.w);
                }
        }
        *reinterpret_cast<float4*>(&part[gg][d4 * 4]) = sum;
    }
    __syncthreads();
    if (tid >= AW_HD) return;
    float tot = part[0][tid];
#pragma unroll
    for (int k = 1; k < AM_GROUPS; ++k) tot += part[k][tid];
    const float y = tot / z * sigmoidf_(gate);
    if (!img) {
        out[((size_t) t * nq + h) * AW_HD + tid] = y;
        return;
    }
    row[tid] = y;
    asm volatile("bar.sync 1, %0;" ::"n"(AW_HD) : "memory");
    if (tid >= 32) return;
    const float4 a = *reinterpret_cast<const float4*>(&row[lane * 8]), b = *reinterpret_cast<const float4*>(&row[lane * 8 + 4]);
    const float y8[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    ni_quant(img, nq, y8, 0.f, t, h, lane);
}

int attn_window_setup() {
    CUtensorMap map;
    FNX_TRY(attn_kv_map(&map, reinterpret_cast<const __half*>(256), 1, 64));
    return set_smem_limit((const void*) k_attn_win, AW_SMEM);
}

int attn_window(const AttnWin& a, void* scratch, float* out, uint8_t* img, bool early, cudaStream_t st) {
    FNX_REQUIRE(a.hd == AW_HD, "attention: head dim %d (this build: %d)", a.hd, AW_HD);
    FNX_REQUIRE(a.nkv >= 1 && a.nq % a.nkv == 0 && a.nq / a.nkv <= ATT_MAXQ, "attention: %d q heads over %d KV heads", a.nq, a.nkv);
    FNX_REQUIRE(a.T >= 1 && a.T <= FNX_MAX_ROWS && a.n_lanes <= FNX_MAX_ROWS, "attention: %d rows", a.T);
    const int S = sm_count() / a.nkv < 1 ? 1 : sm_count() / a.nkv;
    if (S > 256) return fail(FNX_E_ARG, "attention: %d splits", S);
    if (a.ldq % 4 || ((uintptr_t) a.qg & 15) || ((uintptr_t) a.kc & 15) || ((uintptr_t) a.vc & 15)) return fail(FNX_E_ARG, "attention: rows and caches must be 16-byte aligned");
    float* acc = (float*) (((uintptr_t) scratch + 15) & ~(uintptr_t) 15);   // (16-byte pieces; the scratch may lie on any 8-byte boundary)
    AttPartial* mz = (AttPartial*) (acc + (size_t) a.T * a.nq * S * AW_HD);
    // (nominal extents, as far as a copy's row number reaches: the kernel asks only for whole chunks below a context's end)
    CUtensorMap map_k, map_v;
    FNX_TRY(attn_kv_map(&map_k, a.kc, a.nkv, 1ll << 31));
    FNX_TRY(attn_kv_map(&map_v, a.vc, a.nkv, 1ll << 31));
    FNX_TRY(set_smem_limit((const void*) k_attn_win, AW_SMEM));
    cudaError_t le = launch_dep(early, k_attn_win, dim3(sm_count()), dim3(AW_THREADS), (size_t) AW_SMEM, st, a, acc, mz, S, map_k, map_v);
    if (le != cudaSuccess) return fail(FNX_E_CUDA, "k_attn_win: launch failed: %s", cudaGetErrorString(le));
    // (the merge reads positions, lane tables and gates ahead of its wait: all of them older than the kernel before it)
    const bool many = (long long) a.T * a.nq > 2 * sm_count();
    le = launch_dep(true, many ? k_attn_merge<4> : k_attn_merge<AM_GROUPS>, dim3(a.nq, a.T), dim3((many ? 4 : AM_GROUPS) * 64), 0, st, (const float*) acc, (const AttPartial*) mz,
                    a.qg, a.ldq, out, img, a.T, a.nq, S, a.pos, a.lane_seq, a.lane_row0, a.n_lanes);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_attn_merge: launch failed: %s", cudaGetErrorString(le));
}

}  // namespace fnxb
