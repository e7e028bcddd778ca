// Prompt products x W^T from weights in the engine's own layout (nat_tile.h): the prompt's projections of few rows (a rule in moe_prefill.cu) and its expert
// products at every length, on tcgen05.mma with the weights as the A operand in tensor memory.
//
// Replaces the reference's grouped expert GEMMs for prompts, moe_gate_up_mma / moe_down_mma (engine/src/kernels.hpp:328-330,
// engine/src/moe_mma.cuh:301).
//
// What it cannot do without, for 256 features x 64 columns: at a few rows an expert, the weights' bytes (377 cycles of an SM's share of
// DRAM); at many, the products (8 x M128 N64 K16, 300 cycles) and the decode (16 warps x some 85 instructions, 340 cycles).  So nothing may pass
// through shared memory that need not: f16 weight tiles written there by the decode and read back by the tensor core took 500 cycles
// on their own, and 256-row tiles another 1,000 of products over rows that mostly were not there (thirteen rows an expert in a prompt
// of 640).  Here
//   - sixteen decode warps own a 16-row tile row each: 2,176-byte half tiles by their lanes' own async copies, three blocks ahead across
//     items; nibbles to f16 with one shift, four masks and eight half operations a word of eight; a lane's words are columns of
//     tcgen05.st's 16x128b shape, so 64 columns leave as one store of sixteen registers;
//   - two warps gather the job's live rows (a row of B only reaches its own column of D: the others stay what they are);
//   - one warp issues the products, one thread each, two accumulators (gate and up, or 2 x 128 features) double-buffered in tensor memory;
//   - four warps write the item before.
// Tensor memory: columns [0, 256) two pairs of accumulators, [256, 512) two stages of two 128 x 128 weight tiles.  Jobs have at most 64 rows, and
// the products' N is a job's own rows in sixteens (six rows a job: 178 us with N = 64, 166).  Jobs of 128 rows halve the decode, but leave one
// accumulator pair, whose results (6 us an item) then lie in the next item's way: 388 us for 512 jobs of 116 rows, 339 for 1,024 of 58.
// Measured, gate|up and down of a layer of a prompt (512 experts, ten picks a row: 512 jobs of up to 64 rows are fourteen items of 256 features x 2,048 columns an SM), us: 307 rows
// (six an expert) 147 + 79, 2,970 (58) 261 + 149, 38,912 (760, 64 a job) 2,423 + 1,430; with the weights' stores of shape 16x256b 151 + 82, 266 + 153, 2,497 + 1,432 (before these, jobs alone of six, 58 and 760 rows an
// expert: 187 + 101, 200 + 126 and 2,172 + 1,334 with four stages of rows, N = 64 and two instructions a word more, 162 + 92, 179 + 115 and 1,940 + 1,244 without).  By its clocks a down
// chunk of 128 columns takes 1,430 cycles at 333 rows and 1,630 at 20,000: a decode warp waits 200 of them for a free stage and works the rest (13 instructions a word, half and integer-logic ones at two cycles each on pipes that overlap by half), the issuing thread waits
// 410 to 530 for the weights.  DRAM would allow 88.
#include <type_traits>

#include "attn_tc.cuh"
#include "nat_tile.h"
#include "prompt_nat.cuh"

namespace fnxb {

constexpr int PN_KC = 128;             // columns a stage (64: every stage's waits and arrivals cost a few hundred cycles: 285 against 194 us for 513 jobs)
constexpr int PN_DECODE = 16;          // warps
constexpr int PN_EPI = 4, PN_LOAD = 2;
constexpr int PN_W_MMA = PN_EPI, PN_W_LOAD = PN_W_MMA + 1, PN_W_DECODE = 8;   // (warp 7 idles: the decode warps start at a multiple of four)
constexpr int PN_THREADS = (PN_W_DECODE + PN_DECODE) * 32;
constexpr int PN_AST = 256 / PN_KC;    // stages of A (tensor memory)
constexpr int PN_HEAD = 1024;
constexpr uint32_t PN_A = 256;         // tensor memory: first column of the weight stages
constexpr int PN_SLOTS = 3;            // half tiles in flight a decode warp
// Stages of B (shared memory).  The rows come from L2 in 16-byte pieces, a chunk some 1,000 cycles after it was asked for, and pace everything where few
// chunks are on the way: 512 jobs of 58 rows, gate|up 240 us with two stages, 198 with three, 190 with four, 179 with seven and a half tile less a warp.
constexpr int PN_BST = 7, PN_LAG = 3;  // (of which in flight)
constexpr int PN_BBOX = PN_N * 128, PN_BBYTES = PN_KC / 64 * PN_BBOX;   // 64 rows x 64 columns, 128-byte swizzle
constexpr int PN_SMEM = PN_HEAD + PN_BST * PN_BBYTES + PN_DECODE * PN_SLOTS * NAT_HALF_BYTES;
constexpr uint32_t PN_ACC = 2 * PN_N;  // tensor-memory columns of an accumulator pair
static_assert(PN_SMEM <= 227 * 1024, "fits one block's shared memory");

struct PnShared {
    uint64_t full[PN_AST], empty[PN_AST];     // weights of a chunk in tensor memory
    uint64_t bfull[PN_BST], bempty[PN_BST];   // rows of a chunk in shared memory
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem;
    volatile int gave_up;
};
static_assert(sizeof(PnShared) <= PN_HEAD, "the head fits");

__device__ __forceinline__ bool pn_wait(uint64_t* bar, unsigned parity, PnShared& S) { return ta_wait_for(bar, parity, S.gave_up); }

// sixteen tensor-memory lanes x 32 columns: register 2 b = column 4 b + q of lane g, 2 b + 1 the same of lane g + 8.  (The shape 16x256b, a fragment as mma.sync has it, takes
// twice as long: 131 cycles a warp's store against 67 with sixteen warps at it.)
__device__ __forceinline__ void pn_st_tile(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
                 "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ uint32_t pn_h2(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 pn_as_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// (a & b) ^ c in one instruction: with two constants the compiler makes two of it, and the integer-logic pipe is what bounds the decode
__device__ __forceinline__ uint32_t pn_and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// The eight weights of a word times the sub-block's scale (in both halves of f): out[0], out[1] = columns (0, 2), (1, 3), out[2], out[3] =
// (4, 6), (5, 7).  A nibble t at bits 0..3 of a half 0x6400 | .. is 1024 + (t + 8): twice that less 2,064 is 2 t, and one multiply-add makes
// (2 t + 1) f of it; at bits 4..7 it is 1024 + 16 (t + 8) = 8 (143 + m).  All exact but the one rounding of m f, as in the other forms of these
// products.  (Thirteen instructions a word; with the low nibbles moved up a bit, so that 1,039 + m was left to subtract, fifteen.)
// WIDE: the same for scales that may be infinite, where (2 t) f + f would be NaN.  A warp asks once a block of 256 columns (pn_wide): with a form of fourteen
// instructions that holds for all scales, prompts of up to 204 rows took 2 to 3% longer, others 1.5%.
template <bool WIDE>
__device__ __forceinline__ void pn_decode8(uint32_t w, __half2 f, uint32_t& o0, uint32_t& o1, uint32_t& o2, uint32_t& o3) {
    const uint32_t s = w >> 8;
    const uint32_t a = pn_and_xor(w, 0x000F000Fu, 0x64086408u), c = pn_and_xor(w, 0x00F000F0u, 0x64806480u);
    const uint32_t b = pn_and_xor(s, 0x000F000Fu, 0x64086408u), d = pn_and_xor(s, 0x00F000F0u, 0x64806480u);
    const __half2 two = pn_as_h2(0x40004000u), k1 = pn_as_h2(0xE808E808u), one = pn_as_h2(0x3C003C00u);   // 2, -2,064, 1
    const __half2 k8 = pn_as_h2(0x30003000u), k2 = pn_as_h2(0xD878D878u);       // 1 / 8, -143
    const __half2 ta = __hfma2(pn_as_h2(a), two, k1), tb = __hfma2(pn_as_h2(b), two, k1);
    o0 = pn_h2(WIDE ? __hmul2(__hadd2(ta, one), f) : __hfma2(ta, f, f));
    o1 = pn_h2(WIDE ? __hmul2(__hadd2(tb, one), f) : __hfma2(tb, f, f));
    o2 = pn_h2(__hmul2(__hfma2(pn_as_h2(c), k8, k2), f));
    o3 = pn_h2(__hmul2(__hfma2(pn_as_h2(d), k8, k2), f));
}
// whether one of a warp's scales d (two rows' in a word; z = d & d << 1) may overflow f16 times 31: 512 and up, infinities and NaN
__device__ __forceinline__ bool pn_wide(uint32_t z) { return __any_sync(0xffffffffu, (z & 0x40004000u) != 0u); }
// a row's two scales d (1 + 2 s) of sub-blocks 2 Q and 2 Q + 1 (the nibbles of byte Q of sn); d in both halves.  The byte goes into both halves
// 0x6400 | .., the low one keeps its low nibble (1024 + s), the high one its high nibble (1024 + 16 s); 1 + 2 s is exact, and its product with d rounds once, as
// from f32
__device__ __forceinline__ void pn_scales(uint32_t sn, int Q, __half2 d, __half2& f0, __half2& f1) {
    uint32_t t;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(t) : "r"(sn), "r"(0x64u), "r"(0x4040u + 0x0101u * Q));
    const __half2 s2 = __hfma2(pn_as_h2(t & 0xFFF0FF0Fu), pn_as_h2(0x30004000u), pn_as_h2(0xD7F0E7FFu));   // (2, 1 / 8) x - (2,047, 127)
    const __half2 f = __hmul2(s2, d);
    f0 = __low2half2(f);
    f1 = __high2half2(f);
}

struct PnItem {
    int w, n, start, slab;
};

// MODE 1: gate|up, 0: down, 2: dense (any number of 16-row groups, sums)
template <int MODE>
__global__ void __launch_bounds__(PN_THREADS, 1) k_prompt_nat(const PnParams p) {
    pdl_begin();
    extern __shared__ __align__(1024) uint8_t smem[];
    PnShared& sh = *reinterpret_cast<PnShared*>(smem);
    uint8_t* Bs = smem + PN_HEAD;
    uint8_t* ring = Bs + PN_BST * PN_BBYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < PN_AST; ++i) {
            mbar_init(&sh.full[i], PN_DECODE);
            mbar_init(&sh.empty[i], 1);
        }
        for (int i = 0; i < PN_BST; ++i) {
            mbar_init(&sh.bfull[i], PN_LOAD);
            mbar_init(&sh.bempty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_empty[i], PN_EPI);
        }
        sh.gave_up = smem_u32(smem) & 1023u ? 1 : 0;   // (the swizzled tiles need their 1,024-byte boundary)
        fence_barrier_init();
    }
    if (warp == PN_W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ta_fence_before();
    __syncthreads();
    ta_fence_after();
    const uint32_t tmem = sh.tmem;
    const int KB = p.K / 256, nchunk = p.K / PN_KC;
    const int slabs = MODE == 1 ? p.rows / 128 : (p.rows + 255) / 256;
    const int njobs = MODE != 2 ? *p.njobs : (p.T + p.per - 1) / p.per, total = njobs * slabs;
    auto job_of = [&](int it) {
        const int j = it / slabs;
        PnItem x;
        x.slab = it - j * slabs;
        if (MODE != 2) {
            const PnJob jb = p.jobs[j];
            x.w = jb.w; x.n = jb.n; x.start = jb.start;
        } else {
            x.w = 0; x.start = j * p.per; x.n = min(p.per, p.T - x.start);
        }
        return x;
    };
    bool ok = !sh.gave_up;
    if (warp >= PN_W_DECODE) {
        // ---------------------------------------------------------------------------------------- decode
        // tensor-memory lanes 32 (warp % 4) + 16 h of tile `mat`
        const int dw = warp - PN_W_DECODE, lq = dw & 3, h = (dw >> 2) & 1, mat = dw >> 3;
        const uint32_t t_lane = tmem + ((uint32_t) (32 * lq + 16 * h) << 16) + PN_A + mat * (PN_KC / 2);
        uint8_t* my = ring + dw * PN_SLOTS * NAT_HALF_BYTES;
        const uint32_t my_s = smem_u32(my);
        const int n16 = (MODE == 1 ? 2 : 1) * (p.rows / 16);
        // the item's half tiles of this warp (null: past the matrix's last row)
        auto expert_of = [&](int it) { return it < total && MODE != 2 ? p.jobs[it / slabs].w : 0; };
        auto base_of = [&](int it, int e) -> const uint8_t* {
            const int slab = it % slabs, i = MODE == 1 ? mat * (p.rows / 16) + slab * 8 + lq * 2 + h : slab * 16 + mat * 8 + lq * 2 + h;
            if (MODE == 2 && i >= n16) return nullptr;
            const uint8_t* W = MODE == 2 ? p.W : e >= p.E ? p.Wsh : p.W + (size_t) (e - p.e_base) * p.stride;
            return W + nat_half_at((size_t) i, (size_t) n16, 0, (size_t) KB, MODE == 1) + lane * 16;
        };
        // the copies' cursor
        int fit = blockIdx.x, fkb = 0, fslot = 0;
        const uint8_t* src = fit < total ? base_of(fit, expert_of(fit)) : nullptr;
        int e_next = expert_of(fit + gridDim.x);   // (one item ahead: its load is not waited for)
        auto fetch = [&]() {
            if (fit < total) {
                if (src) {
                    const uint32_t dst = my_s + fslot * NAT_HALF_BYTES + lane * 16;
#pragma unroll
                    for (int j = 0; j < 4; ++j) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * 512), "l"(src + j * 512) : "memory");
                    if (lane < 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + NAT_META), "l"(src + NAT_META) : "memory");
                    src += NAT_TILE_BYTES;
                }
                if (++fkb == KB) {
                    fkb = 0;
                    fit += gridDim.x;
                    if (fit < total) {
                        src = base_of(fit, e_next);
                        e_next = expert_of(fit + gridDim.x);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            fslot = fslot + 1 == PN_SLOTS ? 0 : fslot + 1;
        };
#pragma unroll
        for (int i = 0; i < PN_SLOTS; ++i) fetch();
        int c = 0, slot = 0;   // chunks so far
        for (int it = blockIdx.x; it < total; it += gridDim.x) {
            for (int kb = 0; kb < KB; ++kb) {
                asm volatile("cp.async.wait_group %0;" ::"n"(PN_SLOTS - 1) : "memory");
                __syncwarp();   // (the scales came in by other lanes' copies)
                uint32_t w[2][8];
                const uint8_t* t = my + slot * NAT_HALF_BYTES;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint4 v = *reinterpret_cast<const uint4*>(t + j * 512 + lane * 16);
                    w[j >> 1][(j & 1) * 4] = v.x; w[j >> 1][(j & 1) * 4 + 1] = v.y; w[j >> 1][(j & 1) * 4 + 2] = v.z; w[j >> 1][(j & 1) * 4 + 3] = v.w;
                }
                const uint4 m = *reinterpret_cast<const uint4*>(t + NAT_META + (lane >> 2) * 16);
                const __half2 d = pn_as_h2(m.z), d0 = __low2half2(d), d1 = __high2half2(d);
                __syncwarp();   // every lane has the slot
                fetch();
                slot = slot + 1 == PN_SLOTS ? 0 : slot + 1;
                auto decode = [&](auto wide) {
                    constexpr bool WIDE = decltype(wide)::value;
#pragma unroll
                    for (int st = 0; st < PN_AST; ++st, ++c) {
#pragma unroll
                        for (int q2 = 0; q2 < PN_KC / 64; ++q2) {
                            const int Q = PN_KC / 64 * st + q2;
                            uint32_t o[16];
                            __half2 f00, f01, f10, f11;
                            pn_scales(m.x, Q, d0, f00, f01);
                            pn_scales(m.y, Q, d1, f10, f11);
                            pn_decode8<WIDE>(w[0][2 * Q], f00, o[0], o[2], o[4], o[6]);
                            pn_decode8<WIDE>(w[1][2 * Q], f10, o[1], o[3], o[5], o[7]);
                            pn_decode8<WIDE>(w[0][2 * Q + 1], f01, o[8], o[10], o[12], o[14]);
                            pn_decode8<WIDE>(w[1][2 * Q + 1], f11, o[9], o[11], o[13], o[15]);
                            if (q2 == 0) {
                                if (ok && c >= PN_AST) ok = __all_sync(0xffffffffu, pn_wait(&sh.empty[st], (unsigned) ((c / PN_AST - 1) & 1), sh));
                                ta_fence_after();
                            }
                            pn_st_tile(t_lane + st * PN_KC + q2 * 32, o);
                        }
                        ta_wait_st();
                        ta_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.full[st]);
                    }
                };
                if (pn_wide(m.z & (m.z << 1))) decode(std::true_type{});
                else decode(std::false_type{});
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp >= PN_W_LOAD && warp < PN_W_LOAD + PN_LOAD) {
        // ---------------------------------------------------------------------------------------- the rows
        // thread: piece lt % 8 of the rows lt / 8 + 8 j, in both boxes of a stage.  Jobs and entries are loaded an item ahead, and a chunk
        // is reported before the wait for the next one's stage, so that neither latency lies in the products' way.
        constexpr int RJ = PN_N / (4 * PN_LOAD);
        const int lt = tid - PN_W_LOAD * 32, piece = lt & 7, r0 = lt >> 3;
        const uint32_t b_s = smem_u32(Bs) + r0 * 128 + ((piece ^ (r0 & 7)) * 16);   // (r0 + 8 j has the same low bits)
        int c = 0, st = 0, lst = 0;   // chunks so far; the next one's stage, the next reported one's
        unsigned bpar = 1;            // (a stage's first use finds it free)
        auto landed = [&]() {
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.bfull[lst]);
            lst = lst + 1 == PN_BST ? 0 : lst + 1;
        };
        PnItem x = job_of(min((int) blockIdx.x, total - 1)), nx;
        int e[RJ];   // the item's entries
        auto entries = [&](const PnItem& y) {
#pragma unroll
            for (int j = 0; j < RJ; ++j) e[j] = MODE != 2 ? p.order[y.start + min(r0 + 4 * PN_LOAD * j, y.n - 1)] : y.start + r0 + 4 * PN_LOAD * j;
        };
        entries(x);
        for (int it = blockIdx.x; it < total; it += gridDim.x) {
            uint32_t src[RJ];   // in units of 16 bytes
            const int live = (x.n - r0 + 4 * PN_LOAD - 1) / (4 * PN_LOAD);   // of the thread's rows
#pragma unroll
            for (int j = 0; j < RJ; ++j) {
                int row = e[j];
                if (MODE == 1) row = row >= p.TKp ? row - p.TKp : row / p.Kp;
                src[j] = (uint32_t) row * (uint32_t) (p.K / 8) + piece;
            }
            const bool more = it + (int) gridDim.x < total;
            if (more) nx = job_of(it + gridDim.x);
            const __half* xk = p.x;
            for (int k = 0; k < nchunk; ++k, ++c, xk += PN_KC) {
                if (c >= PN_LAG) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(PN_LAG - 1) : "memory");
                    landed();
                }
                if (ok && c >= PN_BST) ok = __all_sync(0xffffffffu, pn_wait(&sh.bempty[st], bpar, sh));
                if (ok) {
                    const uint32_t dst = b_s + st * PN_BBYTES;
#pragma unroll
                    for (int j = 0; j < RJ; ++j)
                        if (j < live) {
                            const __half* g = xk + (size_t) src[j] * 8;
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * (512 * PN_LOAD)), "l"(g) : "memory");
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + PN_BBOX + j * (512 * PN_LOAD)), "l"(g + 64) : "memory");
                        }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (++st == PN_BST) {
                    st = 0;
                    bpar ^= 1;
                }
                if (k == 0 && more) entries(nx);
            }
            x = nx;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        for (int i = max(0, c - PN_LAG); i < c; ++i) landed();
    } else if (warp == PN_W_MMA) {
        // ---------------------------------------------------------------------------------------- the products
        const uint32_t b_s = smem_u32(Bs);
        // (one thread all through: among sixteen decoding warps every instruction of this one is paid five or six times)
        if (ta_elect()) {
            int c = 0, nit = 0, st = 0;
            unsigned bpar = 0;
            int n = job_of(min((int) blockIdx.x, total - 1)).n;
            for (int it = blockIdx.x; it < total && ok; it += gridDim.x, ++nit) {
                const int buf = nit & 1;
                const uint32_t acc = tmem + buf * PN_ACC;
                // N: the job's rows, in sixteens
                const uint32_t idesc = (1u << 4) | ((uint32_t) ((n + 15) >> 4) << 18) | ((uint32_t) (128 >> 4) << 24);
                if (it + (int) gridDim.x < total) n = job_of(it + gridDim.x).n;   // (used an item later)
                if (nit >= 2) ok = pn_wait(&sh.acc_empty[buf], (unsigned) ((nit / 2 - 1) & 1), sh);
                for (int k = 0; k < nchunk && ok; ++k, ++c) {
                    ok = pn_wait(&sh.bfull[st], bpar, sh) && pn_wait(&sh.full[c % PN_AST], (unsigned) ((c / PN_AST) & 1), sh);
                    if (!ok) break;
                    ta_fence_after();
                    const uint32_t a_t = tmem + PN_A + (c % PN_AST) * PN_KC, b = b_s + st * PN_BBYTES;
#pragma unroll
                    for (int k16 = 0; k16 < PN_KC / 16; ++k16) {
                        const uint64_t bd = ta_desc_sw(b + (k16 >> 2) * PN_BBOX + (k16 & 3) * 32, 16, 1024);
                        ta_mma_ta(acc, a_t + k16 * 8, bd, idesc, (k | k16) != 0);
                        ta_mma_ta(acc + PN_N, a_t + PN_KC / 2 + k16 * 8, bd, idesc, (k | k16) != 0);
                    }
                    ta_commit(&sh.empty[c % PN_AST]);
                    ta_commit(&sh.bempty[st]);
                    if (k == nchunk - 1) ta_commit(&sh.acc_full[buf]);
                    if (++st == PN_BST) {
                        st = 0;
                        bpar ^= 1;
                    }
                }
            }
            if (ok && c > 0) {   // the last arrivals, before the shared memory goes
                pn_wait(&sh.empty[(c - 1) % PN_AST], (unsigned) (((c - 1) / PN_AST) & 1), sh);
                pn_wait(&sh.bempty[(c - 1) % PN_BST], (unsigned) (((c - 1) / PN_BST) & 1), sh);
            }
        }
        __syncwarp();
    } else if (warp < PN_EPI) {
        // ---------------------------------------------------------------------------------------- the results
        const int lq = warp & 3;
        const uint32_t lane_base = (uint32_t) (32 * lq) << 16;
        const int ldo = MODE == 1 ? p.rows : p.ldo;
        int nit = 0;
        for (int it = blockIdx.x; it < total; it += gridDim.x, ++nit) {
            const PnItem x = job_of(it);
            const int buf = nit & 1;
            int e[PN_N / 32];   // the item's output rows
#pragma unroll
            for (int j = 0; j < PN_N / 32; ++j) {
                e[j] = x.start + min(lane + 32 * j, x.n - 1);
                if (MODE != 2) e[j] = p.order[e[j]];
            }
            if (ok) ok = __all_sync(0xffffffffu, pn_wait(&sh.acc_full[buf], (unsigned) ((nit / 2) & 1), sh));
            ta_fence_after();
            if (ok) {
                const uint32_t acc = tmem + buf * PN_ACC + lane_base;
                const int f = MODE == 1 ? x.slab * 128 + lq * 32 + pn_slot(lane) : x.slab * 256 + lq * 32 + lane;
                const bool in0 = f < p.rows, in1 = f + 128 < p.rows;
#pragma unroll 1
                for (int c0 = 0; c0 < x.n; c0 += 16) {
                    int mine = e[0];
#pragma unroll
                    for (int j = 1; j < PN_N / 32; ++j)
                        if (c0 >= 32 * j) mine = e[j];
                    float g[16], u[16], old0[MODE == 2 ? 16 : 1], old1[MODE == 2 ? 16 : 1];
                    if (MODE == 2) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const size_t o = (size_t) __shfl_sync(0xffffffffu, mine, (c0 & 16) + i) * ldo + f;
                            old0[i] = p.accumulate && in0 && c0 + i < x.n ? p.out[o] : 0.f;
                            old1[i] = p.accumulate && in1 && c0 + i < x.n ? p.out[o + 128] : 0.f;
                        }
                    }
                    ta_ld16(acc + c0, g);
                    ta_ld16(acc + PN_N + c0, u);
                    ta_wait_ld(g, u);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const size_t o = (size_t) __shfl_sync(0xffffffffu, mine, (c0 & 16) + i) * ldo + f;
                        if (c0 + i < x.n) {
                            // (rounded to f16: the hardware's exponential and division are far inside that)
                            if (MODE == 1) p.outh[o] = __float2half_rn(__fdividef(g[i], 1.0f + __expf(-g[i])) * u[i]);
                            else if (MODE == 0) {
                                __stcs(p.out + o, g[i]);
                                __stcs(p.out + o + 128, u[i]);
                            } else {
                                if (in0) p.out[o] = old0[i] + g[i];
                                if (in1) p.out[o + 128] = old1[i] + u[i];
                            }
                        }
                    }
                }
            }
            ta_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
        }
    }
    ta_fence_before();
    __syncthreads();
    if (tid == 0 && sh.gave_up) atomicOr(p.err, (unsigned) FNX_ERR_TIMEOUT);
    if (warp == PN_W_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------------------------------------------------------ jobs of few rows
// The expert products where an expert has up to four rows on average: mma.sync with the decoded fragments in registers as the A
// operand, so that neither tensor memory nor the waits between its writers and readers are in the way.  Bound by the decode's instructions
// (integer-logic and half pipes, two cycles each; half of either busy).  An item is a job and 16 tiles of 32 features (gate|up: 16 gate
// and the 16 up of the same features), a warp each; the job's rows go through three shared-memory chunks of 256 columns, a warp's tiles
// through two slots of its own.  A layer's experts of a prompt (512 of them, ten picks a row; job lists, rows' copy
// and combine included), us: 32, 64, 100, 150 and 204 rows 117, 168, 194, 222 and 257 here, 126, 175, 201, 224 and 243 by k_prompt_nat; two groups of eight rows a
// job won 1% between four and five rows an expert and lost beyond.
// The rows' columns lie in fours as (0, 2, 1, 3), the order of a decoded word's pairs.
constexpr int PW_WARPS = 16, PW_THREADS = PW_WARPS * 32, PW_BST = 3;
constexpr int PW_N = PROMPT_FEW_ROWS;   // rows of a job: the products' N
constexpr int PW_ROW = 512 + 64;   // bytes of a row's chunk (neighbouring rows in different halves of the banks)
constexpr int PW_RING = PW_WARPS * 2 * NAT_TILE_BYTES;
constexpr int PW_SMEM = PW_RING + PW_BST * PW_N * PW_ROW;

__device__ __forceinline__ void pw_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MODE>
__global__ void __launch_bounds__(PW_THREADS, 1) k_prompt_few(const PnParams p) {
    pdl_begin();
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int KB = p.K / 256, units = MODE == 1 ? p.rows / 16 : p.rows / 32, parts = (units + PW_WARPS - 1) / PW_WARPS, total = *p.njobs * parts;
    if ((int) blockIdx.x >= total) return;
    uint8_t* ring = smem + warp * 2 * NAT_TILE_BYTES;
    uint8_t* Bs = smem + PW_RING;
    const uint32_t ring_s = smem_u32(ring) + lane * 16, b_s = smem_u32(Bs) + warp * PW_ROW + lane * 16;
    // the copies' cursor, two chunks ahead; the next item's job and entries are loaded ahead of it
    int cit = blockIdx.x, ckb = 0;
    const uint8_t* wsrc = nullptr;
    const __half* xsrc;   // the warp's row
    PnJob nx;
    int e;
    bool need_e = true;
    auto entries = [&]() {
        e = p.order[nx.start + min(warp, nx.n - 1)];
        need_e = false;
    };
    auto enter = [&]() {   // the cursor's item: `nx`
        if (need_e) entries();
        const int unit = cit % parts * PW_WARPS + warp;
        const uint8_t* W = nx.w >= p.E ? p.Wsh : p.W + (size_t) (nx.w - p.e_base) * p.stride;
        wsrc = unit < units ? W + (size_t) unit * KB * NAT_TILE_BYTES + lane * 16 : nullptr;
        const int row = MODE == 1 ? (e >= p.TKp ? e - p.TKp : e / p.Kp) : e;
        xsrc = warp < min(nx.n, PW_N) ? p.x + (size_t) row * p.K + lane * 8 : nullptr;
        if (cit + (int) gridDim.x < total) {
            nx = p.jobs[(cit + gridDim.x) / parts];
            need_e = true;
        }
    };
    auto advance = [&]() {
        if (cit >= total) return;
        if (++ckb == KB) {
            ckb = 0;
            cit += gridDim.x;
            if (cit < total) enter();
        } else if (need_e) {
            entries();
        }
    };
    auto fetch_rows = [&](int slot) {
        if (cit < total && xsrc) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(b_s + slot * PW_N * PW_ROW), "l"(xsrc + ckb * 256) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch_tile = [&](int slot) {
        if (cit < total && wsrc) {
            const uint32_t dst = ring_s + slot * NAT_TILE_BYTES;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + h * NAT_HALF_BYTES + j * 512), "l"(wsrc + h * NAT_HALF_BYTES + j * 512) : "memory");
                if (lane < 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + h * NAT_HALF_BYTES + NAT_META), "l"(wsrc + h * NAT_HALF_BYTES + NAT_META) : "memory");
            }
            wsrc += NAT_TILE_BYTES;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    nx = p.jobs[cit / parts];
    enter();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        fetch_rows(i);
        fetch_tile(i);
        advance();
    }
    int c = 0, bslot = 0;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const PnJob job = p.jobs[it / parts];
        const int unit = it % parts * PW_WARPS + warp;
        int mine = 0;   // lane: output row `lane` of the job
        float acc[2][4] = {};
        for (int kb = 0; kb < KB; ++kb, ++c) {
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            __syncthreads();   // the chunk's rows are in, and everyone is done with the chunk before: its place is free
            fetch_rows(bslot == 0 ? PW_BST - 1 : bslot - 1);
            const uint8_t* t = ring + (c & 1) * NAT_TILE_BYTES;
            const uint8_t* b = Bs + (bslot * PW_N + g) * PW_ROW + q * 16;
            if (unit < units) {
                const uint4 m0 = *reinterpret_cast<const uint4*>(t + NAT_META + g * 16), m1 = *reinterpret_cast<const uint4*>(t + NAT_HALF_BYTES + NAT_META + g * 16);
                const __half2 dd[2] = {pn_as_h2(m0.z), pn_as_h2(m1.z)};
                const uint32_t z = (m0.z & (m0.z << 1)) | (m1.z & (m1.z << 1));
#pragma unroll 1
                for (int jj = 0; jj < 2; ++jj) {
                    uint4 w[2][2];
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                        for (int h = 0; h < 2; ++h) w[hf][h] = *reinterpret_cast<const uint4*>(t + hf * NAT_HALF_BYTES + (2 * h + jj) * 512 + lane * 16);
                    auto products = [&](auto wide) {
#pragma unroll
                        for (int s2 = 0; s2 < 2; ++s2) {
                            __half2 f[2][2][2];   // [half tile][row half][sub-block]
#pragma unroll
                            for (int hf = 0; hf < 2; ++hf) {
                                pn_scales((hf ? m1.x : m0.x) >> (16 * jj), s2, __low2half2(dd[hf]), f[hf][0][0], f[hf][0][1]);
                                pn_scales((hf ? m1.y : m0.y) >> (16 * jj), s2, __high2half2(dd[hf]), f[hf][1][0], f[hf][1][1]);
                            }
#pragma unroll
                            for (int e2 = 0; e2 < 2; ++e2) {
                                const uint4 bv = *reinterpret_cast<const uint4*>(b + (4 * jj + 2 * s2 + e2) * 64);
#pragma unroll
                                for (int hf = 0; hf < 2; ++hf) {
                                    const uint32_t wa = s2 ? (e2 ? w[hf][0].w : w[hf][0].z) : (e2 ? w[hf][0].y : w[hf][0].x);
                                    const uint32_t wb = s2 ? (e2 ? w[hf][1].w : w[hf][1].z) : (e2 ? w[hf][1].y : w[hf][1].x);
                                    uint32_t a[4], d[4];
                                    pn_decode8<decltype(wide)::value>(wa, f[hf][0][e2], a[0], a[1], a[2], a[3]);
                                    pn_decode8<decltype(wide)::value>(wb, f[hf][1][e2], d[0], d[1], d[2], d[3]);
                                    pw_mma(acc[hf], a[0], d[0], a[1], d[1], bv.x, bv.y);
                                    pw_mma(acc[hf], a[2], d[2], a[3], d[3], bv.z, bv.w);
                                }
                            }
                        }
                    };
                    if (pn_wide(z)) products(std::true_type{});   // (asked behind the loads)
                    else products(std::false_type{});
                }
            }
            if (kb == 0) mine = p.order[job.start + min(lane, job.n - 1)];   // (used after the last chunk)
            __syncwarp();   // every lane is done with the tile
            fetch_tile(c & 1);
            advance();
            bslot = bslot + 1 == PW_BST ? 0 : bslot + 1;
        }
        // a lane holds the features g and g + 8 of its unit's two half tiles for the rows 2 q, + 1
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = 2 * q + r;
            const size_t o = (size_t) __shfl_sync(0xffffffffu, mine, row);
            if (row < job.n && unit < units) {
                if (MODE == 1) {
                    __half* dst = p.outh + o * p.rows + unit * 16;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int f = g + 8 * i;
                        const float a = acc[0][2 * i + r], b = acc[1][2 * i + r];
                        dst[(f & ~3) | ((f & 1) << 1) | ((f >> 1) & 1)] = __float2half_rn(__fdividef(a, 1.0f + __expf(-a)) * b);
                    }
                } else {
                    float* dst = p.out + o * p.ldo + unit * 32 + g;
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        dst[16 * hf] = acc[hf][r];
                        dst[16 * hf + 8] = acc[hf][2 + r];
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

int prompt_few(int mode, const PnParams& p, int max_jobs, cudaStream_t st) {
    FNX_REQUIRE(p.K % 256 == 0 && p.rows % 32 == 0, "prompt product: %d features x %d", p.rows, p.K);
    auto kernel = mode == 1 ? k_prompt_few<1> : k_prompt_few<0>;
    FNX_TRY(set_smem_limit((const void*) kernel, PW_SMEM));
    const int units = mode == 1 ? p.rows / 16 : p.rows / 32;
    const long long items = (long long) max_jobs * ((units + PW_WARPS - 1) / PW_WARPS);
    FNX_CUDA_OK(launch_after(kernel, dim3((unsigned) (items < sm_count() ? items : sm_count())), dim3(PW_THREADS), PW_SMEM, st, p));
    FNX_LAUNCH_OK("k_prompt_few");
    return FNX_OK;
}

__global__ void __launch_bounds__(256) k_prompt_nat_rows(const float* __restrict__ x, const float* __restrict__ norm_w, int H, float eps, __half* __restrict__ xh, int few) {
    pdl_begin();
    const float* xr = x + (size_t) blockIdx.x * H;
    __shared__ float ws[8];
    constexpr int HOLD = 4;   // the thread's pieces of up to 4,096 columns stay in registers
    float4 v[HOLD];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < HOLD; ++j) {
        const int i = (threadIdx.x + j * 256) * 4;
        v[j] = i < H ? *reinterpret_cast<const float4*>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
    }
    for (int i = (threadIdx.x + HOLD * 256) * 4; i < H; i += 1024) {
        const float4 q = *reinterpret_cast<const float4*>(xr + i);
        ss += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
    }
    float r = 1.0f;
    if (norm_w) {
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += ws[k];
        r = rsqrtf(ss / (float) H + eps);
    }
    auto put = [&](int i, float4 q) {
        if (norm_w) {
            const float4 w = *reinterpret_cast<const float4*>(norm_w + i);
            q.x *= w.x * r; q.y *= w.y * r; q.z *= w.z * r; q.w *= w.w * r;
        }
        const __half2 a = __floats2half2_rn(q.x, q.z), b = __floats2half2_rn(q.y, q.w);   // (pn_slot: columns 0 and 2 side by side, 1 and 3 eight slots on)
        __half* at = xh + (size_t) blockIdx.x * H;
        if (few) *reinterpret_cast<uint2*>(at + i) = make_uint2(pn_h2(a), pn_h2(b));
        else {
            at += pn_slot(i);
            *reinterpret_cast<__half2*>(at) = a;
            *reinterpret_cast<__half2*>(at + 8) = b;
        }
    };
#pragma unroll
    for (int j = 0; j < HOLD; ++j) {
        const int i = (threadIdx.x + j * 256) * 4;
        if (i < H) put(i, v[j]);
    }
    for (int i = (threadIdx.x + HOLD * 256) * 4; i < H; i += 1024) put(i, *reinterpret_cast<const float4*>(xr + i));
}

int prompt_nat_rows(const float* x, const float* norm_w, int T, int H, float eps, __half* xh, bool few, cudaStream_t st) {
    FNX_CUDA_OK(launch_after(k_prompt_nat_rows, dim3(T), dim3(256), 0, st, x, norm_w, H, eps, xh, few));
    FNX_LAUNCH_OK("k_prompt_nat_rows");
    return FNX_OK;
}

int prompt_nat(int mode, const PnParams& p, int max_jobs, cudaStream_t st) {
    FNX_REQUIRE(p.K % 256 == 0 && p.rows % (mode == 2 ? 16 : mode == 1 ? 128 : 256) == 0 && p.per >= 1 && p.per <= PN_N, "prompt product: %d features x %d, jobs of %d rows", p.rows, p.K, p.per);
    auto kernel = mode == 1 ? k_prompt_nat<1> : mode == 0 ? k_prompt_nat<0> : k_prompt_nat<2>;
    FNX_TRY(set_smem_limit((const void*) kernel, PN_SMEM));
    const long long items = (long long) max_jobs * (mode == 1 ? p.rows / 128 : (p.rows + 255) / 256);
    FNX_CUDA_OK(launch_after(kernel, dim3((unsigned) (items < sm_count() ? items : sm_count())), dim3(PN_THREADS), PN_SMEM, st, p));
    FNX_LAUNCH_OK("k_prompt_nat");
    return FNX_OK;
}

}  // namespace fnxb
