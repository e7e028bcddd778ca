// Prompt attention on the 5th-generation tensor cores: the chunk's query rows against the sequence's K/V cache, causal,
// for models whose KV head serves eight query heads of 256 dims (the benchmark's shape).  The counterpart of the reference's
// attn_prompt (engine/src/kernels.hpp:252); same arithmetic as the mma.sync form it stands in for (fnx_attn_prompt's other
// path): f16 queries, f32 scores, an online softmax over steps of 64 positions with f16 weights, f32 sums, the sigmoid gate.
//
// One block = 16 chunk rows x the 8 query heads of one KV head = 128 score rows (tensor-memory lanes), so a K/V tile is
// fetched once for 128 rows.  Per step of 64 positions:
//   S = Q K^T        16 x tcgen05.mma M128 N64 K16   (Q, K in shared memory, 128-byte swizzle; two S in tensor memory, so that the next
//                    step's scores are made while this one's softmax runs)
//   softmax          two threads per row: tcgen05.ld of their 32 scores each, running max / sum, weights rounded to f16 and left in tensor
//                    memory over their scores (the A operand of the next product); the row of O is rescaled in tensor memory only when
//                    some row of the warp moved its maximum
//   O += P V         4 x tcgen05.mma M128 N256 K16   (V as it lies in the cache: dims contiguous = an MN-major B operand)
// K and V tiles run through a ring of five 32 KB slots, filled by tensor copies (cp.async.bulk.tensor, 64 dims x 64 positions a box, 128-byte
// swizzle) as far ahead as slots are free; only a step that the context ends in is fetched by 16-byte async copies, so that nothing past the
// context is ever read.
// What bounds it: a step's products take 1,130 cycles, its 64 KB from L2 about 1,700 of an SM's share, its softmax 1,300; they overlap.
// With one score tile and the phases one after another a step took 4,350 cycles.  Every wait is bounded.
#include <cstdlib>
#include <cstring>

#include "attn_tc.cuh"

namespace fnxb {

constexpr int TA_M = 128;          // score rows per block: 16 positions x 8 heads
constexpr int TA_POS = 16;
constexpr int TA_QPK = 8;
constexpr int TA_N = ATC_N;        // positions per step
constexpr int TA_HD = ATC_HD;
constexpr int TA_SOFT = 256;       // warps 0-7: two threads per score row (a half of the step's positions, of the row's dims)
constexpr int TA_LOAD = 128;       // warps 8-11: the loader (one thread; all of them for the step that the context ends in)
constexpr int TA_THREADS = TA_SOFT + TA_LOAD + 32;   // warp 12: the products
constexpr int TA_RING = 5;         // tiles of 64 positions, K and V in turn
constexpr int TA_BOX = TA_N * 128; // a box of 64 dims: 64 positions x 128 bytes (the 16-byte piece c of position n lies at piece c ^ (n % 8))
constexpr int TA_TILE = (TA_HD / 64) * TA_BOX;   // 32 KB
constexpr int TA_QBOX = TA_M * 128;
constexpr int TA_SBO = 8 * 128;    // between 8-row groups
constexpr int TA_HEAD = 3072;      // barriers, the halves' exchange
constexpr int TA_SMEM = TA_HEAD + TA_RING * TA_TILE + 4 * TA_QBOX;
static_assert(TA_SMEM <= 227 * 1024, "the tiles fit one block's shared memory");
constexpr uint32_t TA_O = 0, TA_S = 256;   // tensor memory columns: the sums, two steps' scores
constexpr int TA_TMEM_COLS = 512;

struct TaShared {
    uint64_t full[TA_RING], empty[TA_RING], bar_s[2], bar_p[2], bar_o, bar_q;
    uint32_t tmem;
    volatile int gave_up;
    float xch[2][2][TA_M];              // [step parity][half][row]
};
static_assert(sizeof(TaShared) <= TA_HEAD, "the head fits");

__device__ __forceinline__ bool ta_wait(uint64_t* bar, unsigned parity, TaShared& S) { return ta_wait_for(bar, parity, S.gave_up); }

// grid (16-row tiles of the chunk, latest first; KV heads)
__global__ void __launch_bounds__(TA_THREADS, 1) k_attn_prompt_tc(const float* __restrict__ qg, int ldq, const __half* __restrict__ kc,
                                                                 const __half* __restrict__ vc, float* __restrict__ out, int T, int nq, int nkv,
                                                                 const int* __restrict__ pos0p, unsigned* __restrict__ err,
                                                                 const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v) {
    pdl_wait();   // (as in the DeltaNet scan, the successor starts at the end)
    extern __shared__ __align__(1024) uint8_t smem[];
    TaShared& sh = *reinterpret_cast<TaShared*>(smem);
    uint8_t* ring = smem + TA_HEAD;
    uint8_t* Qs = ring + TA_RING * TA_TILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = (int) gridDim.x - 1 - (int) blockIdx.x, kvh = blockIdx.y;
    const int t0 = tile * TA_POS, nr = min(TA_POS, T - t0), pos0 = *pos0p;
    const int ctx = pos0 + t0 + nr;                // the tile's rows see positions [0, ctx): a chain's rows see nothing past themselves
    const int nsteps = (ctx + TA_N - 1) / TA_N;
    if (tid == 0) {
        for (int i = 0; i < TA_RING; ++i) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.bar_s[i], 1);
            mbar_init(&sh.bar_p[i], TA_SOFT / 32);
        }
        mbar_init(&sh.bar_o, 1);
        mbar_init(&sh.bar_q, TA_SOFT / 32);
        sh.gave_up = smem_u32(smem) & 1023u ? 1 : 0;   // (the swizzled tiles need their 1,024-byte boundary)
        fence_barrier_init();
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(TA_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ta_fence_before();
    __syncthreads();
    ta_fence_after();
    const uint32_t tmem = sh.tmem;
    bool ok = !sh.gave_up;
    if (warp >= 8 && warp < 12) {
        // ---------------------------------------------------------------------------------------- the loader
        const int lt = tid - TA_SOFT;
        for (int j = 0; j < nsteps; ++j) {
            const int p0 = j * TA_N, np = min(TA_N, ctx - p0), n = 2 * j;
            if (lt == 0)
                for (int kv = 0; kv < 2; ++kv) {
                    const int slot = (n + kv) % TA_RING;
                    if (ok && n + kv >= TA_RING) ok = ta_wait(&sh.empty[slot], (unsigned) (((n + kv) / TA_RING - 1) & 1), sh);
                    if (!ok || np < TA_N) continue;
                    mbar_expect_tx(&sh.full[slot], TA_TILE);
#pragma unroll
                    for (int c = 0; c < TA_HD / 64; ++c) ta_tma_3d(smem_u32(ring + slot * TA_TILE + c * TA_BOX), kv ? &map_v : &map_k, c * 64, kvh, p0, &sh.full[slot]);
                }
            if (np == TA_N) continue;
            // the step the context ends in (the last): 16-byte pieces where the swizzle puts them, the rows past the context zero
            asm volatile("bar.sync 5, %0;" ::"n"(TA_LOAD) : "memory");
            if (!sh.gave_up) {
                uint8_t* kd = ring + n % TA_RING * TA_TILE;
                uint8_t* vd = ring + (n + 1) % TA_RING * TA_TILE;
#pragma unroll 4
                for (int i0 = 0; i0 < TA_N * (TA_HD / 8) / TA_LOAD; ++i0) {
                    const int i = lt + i0 * TA_LOAD, rest = i >> 5, r = (rest & 15) * 4 + (i & 3), d8 = (rest >> 4) * 8 + ((i >> 2) & 7);
                    const uint32_t off = (uint32_t) ((d8 >> 3) * TA_BOX + r * 128 + (((d8 & 7) ^ (r & 7)) * 16));
                    if (r < np) {
                        const size_t go = ((size_t) (p0 + r) * nkv + kvh) * TA_HD + d8 * 8;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(kd + off)), "l"(kc + go) : "memory");
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(vd + off)), "l"(vc + go) : "memory");
                    } else {
                        *reinterpret_cast<uint4*>(kd + off) = make_uint4(0, 0, 0, 0);
                        *reinterpret_cast<uint4*>(vd + off) = make_uint4(0, 0, 0, 0);
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                fence_proxy_async();   // (the products read it through the async proxy)
            }
            asm volatile("bar.sync 5, %0;" ::"n"(TA_LOAD) : "memory");
            if (lt == 0 && ok) {
                mbar_arrive(&sh.full[n % TA_RING]);
                mbar_arrive(&sh.full[(n + 1) % TA_RING]);
            }
        }
    } else if (warp == 12) {
        // ---------------------------------------------------------------------------------------- the products
        // f32 accumulate, f16 x f16, M = 128; S: both operands K-major, N = 64; O: B (V) MN-major, N = 256
        constexpr uint32_t IDESC_S = (1u << 4) | ((uint32_t) (TA_N >> 3) << 17) | ((uint32_t) (TA_M >> 4) << 24);
        constexpr uint32_t IDESC_O = (1u << 4) | (1u << 16) | ((uint32_t) (TA_HD >> 3) << 17) | ((uint32_t) (TA_M >> 4) << 24);
        const uint32_t q_s = smem_u32(Qs), ring_s = smem_u32(ring);
        if (ta_elect()) {
            auto scores = [&](int j) {
                const int n = 2 * j, slot = n % TA_RING;
                const uint32_t k_s = ring_s + slot * TA_TILE, tm_s = tmem + TA_S + (uint32_t) (j & 1) * TA_N;
                if (ok) ok = ta_wait(&sh.full[slot], (unsigned) ((n / TA_RING) & 1), sh);
                if (!ok) return;
                ta_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < TA_HD / 16; ++k16)
                    ta_mma(tm_s, ta_desc_sw(q_s + (k16 >> 2) * TA_QBOX + (k16 & 3) * 32, 16, TA_SBO), ta_desc_sw(k_s + (k16 >> 2) * TA_BOX + (k16 & 3) * 32, 16, TA_SBO), IDESC_S,
                           k16 != 0);
                ta_commit(&sh.empty[slot]);
                ta_commit(&sh.bar_s[j & 1]);
            };
            ok = ok && ta_wait(&sh.bar_q, 0u, sh);
            scores(0);
            for (int j = 0; j < nsteps; ++j) {
                if (j + 1 < nsteps) scores(j + 1);   // (while the softmax of this step runs; the scores two steps back are weights already used)
                const int n = 2 * j + 1, slot = n % TA_RING;
                const uint32_t v_s = ring_s + slot * TA_TILE, tm_p = tmem + TA_S + (uint32_t) (j & 1) * TA_N;
                ok = ok && ta_wait(&sh.full[slot], (unsigned) ((n / TA_RING) & 1), sh) && ta_wait(&sh.bar_p[j & 1], (unsigned) ((j >> 1) & 1), sh);
                if (!ok) break;
                ta_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < TA_N / 16; ++k16)
                    ta_mma_ta(tmem + TA_O, tm_p + k16 * 8, ta_desc_sw(v_s + k16 * 2 * TA_SBO, TA_BOX, TA_SBO), IDESC_O, (j | k16) != 0);
                ta_commit(&sh.empty[slot]);
                ta_commit(&sh.bar_o);
            }
            // the last arrivals, before the shared memory goes (the score threads wait for bar_o)
            if (ok) ta_wait(&sh.empty[(2 * nsteps - 1) % TA_RING], (unsigned) (((2 * nsteps - 1) / TA_RING) & 1), sh);
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------------------------------------- queries, softmax, results
        // the queries as f16: row r = head (r / 16), chunk row t0 + r % 16; a warp takes whole rows, rows past the chunk's end are zero
#pragma unroll 4
        for (int r = warp; r < TA_M; r += TA_SOFT / 32) {
            uint4 pk = make_uint4(0, 0, 0, 0);
            if ((r & 15) < nr) {
                const float4* src = reinterpret_cast<const float4*>(qg + (size_t) (t0 + (r & 15)) * ldq + (size_t) (kvh * TA_QPK + (r >> 4)) * 2 * TA_HD + lane * 8);
                const float4 a = src[0], b = src[1];
                const __half2 h0 = __floats2half2_rn(a.x, a.y), h1 = __floats2half2_rn(a.z, a.w), h2 = __floats2half2_rn(b.x, b.y), h3 = __floats2half2_rn(b.z, b.w);
                pk = make_uint4(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1), *reinterpret_cast<const uint32_t*>(&h2),
                                *reinterpret_cast<const uint32_t*>(&h3));
            }
            *reinterpret_cast<uint4*>(Qs + (lane >> 3) * TA_QBOX + r * 128 + (((lane & 7) ^ (r & 7)) * 16)) = pk;
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.bar_q);
        const int r = (warp & 3) * 32 + lane, half = warp >> 2, pi = min(r & 15, nr - 1);   // the thread's row, its half, its chunk row (past the end: the last one's mask)
        const int my_pos = pos0 + t0 + pi;
        const uint32_t lane_base = (uint32_t) (32 * (warp & 3)) << 16;
        const unsigned pair_bar = 1u + (unsigned) (warp & 3);   // the named barrier of the row group's two warps
        // scores in the base-2 domain: exp(x - m) = exp2(x log2 e - m log2 e)
        const float scale2 = 0.0625f * 1.4426950408889634f;   // 1 / sqrt(256) x log2 e
        float m_run = -INFINITY, z_half = 0.f;
        for (int j = 0; j < nsteps; ++j) {
            const int b = j & 1, p0 = j * TA_N;
            const uint32_t tm_s = tmem + TA_S + (uint32_t) b * TA_N + lane_base;
            if (ok) ok = __all_sync(0xffffffffu, ta_wait(&sh.bar_s[b], (unsigned) ((j >> 1) & 1), sh));
            ta_fence_after();
            float s[32];
            float mx = -INFINITY;
            if (ok) {
                ta_ld32(tm_s + 32 * half, s);
                // a step wholly before the tile's first row is visible to every row
                if (p0 + TA_N <= pos0 + t0 + 1) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx = fmaxf(mx, s[i]);
                } else {
                    const int c0 = p0 + 32 * half;
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        s[i] = c0 + i <= my_pos ? s[i] : -INFINITY;
                        mx = fmaxf(mx, s[i]);
                    }
                }
                mx *= scale2;
            }
            sh.xch[b][half][r] = mx;
            asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");   // (every thread takes it, whatever its waits saw)
            if (ok) {
                const float mn = fmaxf(m_run, fmaxf(mx, sh.xch[b][half ^ 1][r]));   // (position 0 is visible to every row: never -inf)
                float sum0 = 0.f, sum1 = 0.f;
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const __half2 h = __floats2half2_rn(ta_ex2(fmaf(s[i], scale2, -mn)), ta_ex2(fmaf(s[i + 1], scale2, -mn)));
                    const float2 back = __half22float2(h);
                    sum0 += back.x;
                    sum1 += back.y;
                    pk[i / 2] = *reinterpret_cast<const uint32_t*>(&h);
                }
                const float f = m_run == -INFINITY ? 0.f : ta_ex2(m_run - mn);
                z_half = z_half * f + (sum0 + sum1);
                m_run = mn;
                ta_st16(tm_s + 16 * half, pk);   // over the scores, which both of the row's threads have read
                // the sums of the step before are complete (no phase is skipped), and rescaled where some row's maximum has moved: deep into a long
                // context that is rare
                if (j >= 1) {
                    ok = __all_sync(0xffffffffu, ta_wait(&sh.bar_o, (unsigned) ((j - 1) & 1), sh));
                    ta_fence_after();
                    if (ok && __any_sync(0xffffffffu, f != 1.0f)) {
#pragma unroll 1
                        for (int c32 = 0; c32 < TA_HD / 64; ++c32) {
                            float o[32];
                            ta_ld32(tmem + TA_O + lane_base + 128 * half + c32 * 32, o);
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] *= f;
                            ta_st32(tmem + TA_O + lane_base + 128 * half + c32 * 32, o);
                        }
                    }
                }
                ta_wait_st();
            }
            ta_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.bar_p[b]);
        }
        if (ok) ok = __all_sync(0xffffffffu, ta_wait(&sh.bar_o, (unsigned) ((nsteps - 1) & 1), sh));
        ta_fence_after();
        float* zx = &sh.xch[nsteps & 1][0][0];   // (the last step used the other parity)
        zx[half * TA_M + r] = z_half;
        asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
        if (ok) {
            // out = O / z * sigmoid(gate), 32 dims at a time through the queries' place (every product that reads it is done), so that whole
            // lines move
            uint8_t* mine = Qs + warp * 4096;
            const int w0 = (warp & 3) * 32;
            const float iz = 1.0f / (zx[r] + zx[TA_M + r]);
#pragma unroll 1
            for (int c32 = 0; c32 < TA_HD / 64; ++c32) {
                float o[32];
                ta_ld32(tmem + TA_O + lane_base + 128 * half + c32 * 32, o);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<float4*>(mine + lane * 128 + ((i ^ (lane & 7)) * 16)) = make_float4(o[4 * i] * iz, o[4 * i + 1] * iz, o[4 * i + 2] * iz, o[4 * i + 3] * iz);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int q = i * 4 + (lane >> 3), c = lane & 7, row = w0 + q;
                    if ((row & 15) < nr) {
                        const int t = t0 + (row & 15), h = kvh * TA_QPK + (row >> 4), d = 128 * half + c32 * 32 + c * 4;
                        const float4 g = *reinterpret_cast<const float4*>(qg + (size_t) t * ldq + (size_t) h * 2 * TA_HD + TA_HD + d);
                        const float4 v = *reinterpret_cast<const float4*>(mine + q * 128 + ((c ^ (q & 7)) * 16));
                        *reinterpret_cast<float4*>(out + ((size_t) t * nq + h) * TA_HD + d) =
                            make_float4(v.x * sigmoidf_(g.x), v.y * sigmoidf_(g.y), v.z * sigmoidf_(g.z), v.w * sigmoidf_(g.w));
                    }
                }
                __syncwarp();
            }
        }
    }
    ta_fence_before();
    __syncthreads();
    if (tid == 0 && sh.gave_up && err) atomicOr(err, (unsigned) FNX_ERR_TIMEOUT);
    if (warp == 12) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TA_TMEM_COLS) : "memory");
}

bool attn_prompt_tc_fits(int nq, int nkv, int hd) { return hd == TA_HD && nkv >= 1 && nq == nkv * TA_QPK; }

int attn_prompt_tc_launch(const float* qg, int ldq, const __half* kc, const __half* vc, float* out, int T, int nq, int nkv, const int* pos0, unsigned* err,
                          cudaStream_t st) {
    if (int rc = set_smem_limit((const void*) k_attn_prompt_tc, TA_SMEM)) return rc;
    // (nominal position extent: the kernel asks only for whole steps below a context's end)
    CUtensorMap map_k, map_v;
    FNX_TRY(attn_kv_map(&map_k, kc, nkv, 1 << 24));
    FNX_TRY(attn_kv_map(&map_v, vc, nkv, 1 << 24));
    FNX_CUDA_OK(launch_after(k_attn_prompt_tc, dim3((T + TA_POS - 1) / TA_POS, nkv), dim3(TA_THREADS), TA_SMEM, st, qg, ldq, kc, vc, out, T, nq, nkv, pos0, err, map_k, map_v));
    FNX_LAUNCH_OK("fnx_attn_prompt (tensor-core form)");
    return FNX_OK;
}

}  // namespace fnxb
