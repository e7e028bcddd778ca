// The windows' matrix x few-rows products on the engine's own weight layout (nat_tile.h): dense projections, the experts' gate|up with
// SwiGLU, and down.  The arithmetic is that of iq3s_mmv.cu (integer products of exact odd weights with two-level int8 activations,
// integer sub-block scales, float scales once per 256-column block); what differs is everything around it:
//   - no codebook: an operand register is a mask (and a shift) of the stored nibbles, so an item (one 16 x 256 tile against the rows)
//     takes about 200 warp instructions for four rows instead of about 600, and a block needs no 64 KB table;
//   - the rows come as their image (nat_image.cuh): a dense or gate|up block copies the rows it needs into shared memory and quantises
//     nothing (read through L1 from global memory instead, the operands cost more than the weights); down quantises its few rows itself;
//   - every lane copies its own 64 bytes of the next tiles into shared memory (cp.async): no mbarriers, no issuing lane;
//   - the eight-warp forms of up to two row groups take half an SM's registers, and most of them half its shared memory, so that the next kernel of the window can be
//     resident while this one drains (programmatic dependent launch): its first tiles are on their way before the rows it waits for are
//     written.  The sixteen-warp forms, for products that stream some 10 us and more, have an SM to themselves.
// Bound by HBM for the large expert products, by the launch and its dependent loads for the small dense ones.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "fnx_common.cuh"
#include "iq3s_grid.h"
#include "nat_image.cuh"
#include "nat_tile.h"

namespace cg = cooperative_groups;

namespace fnxb {

__device__ static const uint32_t g_grid_nat[512] = {FNX_IQ3S_GRID_VALUES};

struct NatParams {
    const uint8_t* W;
    size_t expert_stride;
    int e_base;
    const uint8_t* Wsh;
    int E;
    const fnx_job* jobs;
    const int* njobs;
    int njobs_max;
    int T;
    const uint8_t* img;
    int normed;
    float eps;
    const float* x;      // down: h rows
    float* out;
    int ldo;
    int rows, K;         // output rows per job (gate|up: F), columns
    int accumulate;
    int rmax;            // expert modes: rows a block holds at once
};

template <int NG, int MODE>
struct NatPiece {
    using AccT = typename MatAcc<MODE>::type;
    int unit;            // -1: none, -2: the warp had no items at all
    int b_hi;
    AccT v[2 * NG * 64];   // [half][group][16 lanes][4]
};

__device__ __forceinline__ void nm_mma(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// four nibbles of x -> bytes 8 m = 16 t + 8 (the high ones as they lie, the low ones shifted up)
__device__ __forceinline__ uint32_t nm_hi(uint32_t x) { return (x & 0xF0F0F0F0u) | 0x08080808u; }
// (the factor is hidden from the compiler: the shift it would make of it competes with the masks for the integer-logic pipe)
__device__ __forceinline__ uint32_t nm_lo(uint32_t x) {
    uint32_t k;
    asm("mov.u32 %0, 16;" : "=r"(k));
    return ((x * k) & 0xF0F0F0F0u) | 0x08080808u;
}

// Weights pass through L2 once a window and are the first to leave it: what they would push out (the kernels' own code, fetched from
// DRAM again at every launch, the router's weights, activations) is read again a layer later.
__device__ __forceinline__ uint64_t nm_stream_policy() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void nm_cp_stream(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}

// the two rows' eight sub-block scales 1 + 2 s as bytes: even sub-blocks in .x, odd ones in .y
struct NmScales {
    uint2 r0, r1;
};
__device__ __forceinline__ uint2 nm_scale_bytes(uint32_t n) {
    return make_uint2((n & 0x0F0F0F0Fu) * 2u + 0x01010101u, ((n >> 4) & 0x0F0F0F0Fu) * 2u + 0x01010101u);
}
template <int H>
__device__ __forceinline__ NmScales nm_scales(uint32_t am) {
    const uint2 sn = lds_v2<H * NAT_HALF_BYTES + NAT_META>(am);
    return NmScales{nm_scale_bytes(sn.x), nm_scale_bytes(sn.y)};
}
// One half of a tile (16 rows) over four sub-blocks (4 hf ..): decoded operands and the two rows' sub-block scales
struct NmHalf {
    uint32_t a[4][4];
    int f0[4], f1[4];
};
template <int H>
__device__ __forceinline__ void nm_decode(uint32_t a16, const NmScales& sc, int hf, NmHalf& w) {
    const uint4 w0 = lds_v4<H * NAT_HALF_BYTES>(a16 + hf * 512), w1 = lds_v4<H * NAT_HALF_BYTES + 1024>(a16 + hf * 512);
    const uint32_t wa[4] = {w0.x, w0.y, w0.z, w0.w}, wb[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        w.a[k][0] = nm_lo(wa[k]);
        w.a[k][1] = nm_lo(wb[k]);
        w.a[k][2] = nm_hi(wa[k]);
        w.a[k][3] = nm_hi(wb[k]);
        const uint32_t sel = 0x4440u + 2 * hf + (k >> 1);   // sub-block 4 hf + k: byte 2 hf + k / 2 of the even or the odd ones
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(w.f0[k]) : "r"(k & 1 ? sc.r0.y : sc.r0.x), "r"(0u), "r"(sel));
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(w.f1[k]) : "r"(k & 1 ? sc.r1.y : sc.r1.x), "r"(0u), "r"(sel));
    }
}
__device__ __forceinline__ void nm_products(const NmHalf& w, const uint4& x0, const uint4& x1, int (&accI)[4]) {
    const uint32_t b[4][2] = {{x0.x, x0.y}, {x0.z, x0.w}, {x1.x, x1.y}, {x1.z, x1.w}};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int c[4];
        nm_mma(c, w.a[k], b[k][0], b[k][1]);
        accI[0] += w.f0[k] * c[0];
        accI[1] += w.f0[k] * c[1];
        accI[2] += w.f1[k] * c[2];
        accI[3] += w.f1[k] * c[3];
    }
}
template <int H, typename AccT>
__device__ __forceinline__ void nm_flush(uint32_t am, float s0, float s1, const int (&accI)[4], AccT (&acc)[4]) {
    const uint32_t dw = lds_u32<H * NAT_HALF_BYTES + NAT_META + 8>(am);
    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&dw));
    const float d0 = d.x * 0.125f, d1 = d.y * 0.125f;   // (exact: the integers are 8 times the sums)
    if constexpr (sizeof(AccT) == 8) {
        acc[0] += (double) (d0 * s0) * (double) accI[0];
        acc[1] += (double) (d0 * s1) * (double) accI[1];
        acc[2] += (double) (d1 * s0) * (double) accI[2];
        acc[3] += (double) (d1 * s1) * (double) accI[3];
    } else {
        acc[0] += d0 * s0 * (float) accI[0];
        acc[1] += d0 * s1 * (float) accI[1];
        acc[2] += d1 * s0 * (float) accI[2];
        acc[3] += d1 * s1 * (float) accI[3];
    }
}
// One item: the tile at shared address tile_s against one block of the rows; adds into acc[half][ng][0..3] = (row g, column 2 q),
// (g, 2 q + 1), (g + 8, 2 q), (g + 8, 2 q + 1).  xb: shared address of the lane's cells in its column's row of group 0, x0 / x1: of its
// two C columns' scales; groups lie `group` bytes apart.  The integers are exact (8 times the sums of iq3s_mmv.cu's items).
// AccT double (expert modes): the rounded result does not depend on where a row's K-sum was cut, as there.
// The rows' operands are loaded once for both half tiles.  (Most jobs have one
// row, two of the eight columns; a form with half of the integer work for them was slower: 52 against 46 us for 205 jobs, the second
// copy of the code.)  The loop over four sub-blocks stays rolled for three row groups and more, where a thread has 255 registers and its block an SM (a half tile at a
// time in 128, with spills, 8 warps waited most of the time: a head of 151,936 rows over 20 rows 100 us, 62 now; 12,352 x 2,048 16 and 10.7.  The rows' image of the
// plain form leaves no room for a second block anyway; the split form's, a quarter of the columns, would, but its registers are worth more than a successor
// that waits there: windows of eight layers with that form in 128 and in 255, 9 rows 675 and 669 us, 12 rows 750 and 746, 16 rows 883 and 863, 32 rows 1,440 and
// 1,403); the short one is worth unrolling: 50 -> 47 us for 205 jobs.
template <int NG, typename AccT>
__device__ __forceinline__ void nm_item(uint32_t tile_s, uint32_t xb, uint32_t x0, uint32_t x1, uint32_t group, int lane, AccT (&acc)[2][NG][4]) {
    const uint32_t a16 = tile_s + lane * 16, am = tile_s + (lane >> 2) * 16;
    if constexpr (NG > 2) {
        int accI[2][NG][4];
#pragma unroll
        for (int i = 0; i < 2 * NG * 4; ++i) accI[i / (4 * NG)][(i / 4) % NG][i & 3] = 0;
        const NmScales sc0 = nm_scales<0>(am), sc1 = nm_scales<1>(am);
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
            NmHalf w0, w1;
            nm_decode<0>(a16, sc0, hf, w0);
            nm_decode<1>(a16, sc1, hf, w1);
#pragma unroll
            for (int ng = 0; ng < NG; ++ng) {
                const uint4 b0 = lds_v4(xb + ng * group + hf * 128), b1 = lds_v4<64>(xb + ng * group + hf * 128);
                nm_products(w0, b0, b1, accI[0][ng]);
                nm_products(w1, b0, b1, accI[1][ng]);
            }
        }
#pragma unroll
        for (int ng = 0; ng < NG; ++ng) {
            const float s0 = lds_f32(x0 + ng * group), s1 = lds_f32(x1 + ng * group);
            nm_flush<0>(am, s0, s1, accI[0][ng], acc[0][ng]);
            nm_flush<1>(am, s0, s1, accI[1][ng], acc[1][ng]);
        }
    } else {
        int accI[2][NG][4];
#pragma unroll
        for (int i = 0; i < 2 * NG * 4; ++i) accI[i / (4 * NG)][(i / 4) % NG][i & 3] = 0;
        const NmScales sc0 = nm_scales<0>(am), sc1 = nm_scales<1>(am);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            uint4 b0[NG], b1[NG];
#pragma unroll
            for (int ng = 0; ng < NG; ++ng) {
                b0[ng] = lds_v4(xb + ng * group + hf * 128);
                b1[ng] = lds_v4<64>(xb + ng * group + hf * 128);
            }
            {
                NmHalf w;
                nm_decode<0>(a16, sc0, hf, w);
#pragma unroll
                for (int ng = 0; ng < NG; ++ng) nm_products(w, b0[ng], b1[ng], accI[0][ng]);
            }
            {
                NmHalf w;
                nm_decode<1>(a16, sc1, hf, w);
#pragma unroll
                for (int ng = 0; ng < NG; ++ng) nm_products(w, b0[ng], b1[ng], accI[1][ng]);
            }
        }
#pragma unroll
        for (int ng = 0; ng < NG; ++ng) {
            const float s0 = lds_f32(x0 + ng * group), s1 = lds_f32(x1 + ng * group);
            nm_flush<0>(am, s0, s1, accI[0][ng], acc[0][ng]);
            nm_flush<1>(am, s0, s1, accI[1][ng], acc[1][ng]);
        }
    }
}

// the results of a unit, held by threads q < 2; rf: lane i holds 1 / rms of row i (normed rows; else 1); orow: the job's output rows
template <int NG, int MODE, typename AccT>
__device__ __forceinline__ void nm_write(const NatParams& p, int lu, const int* orow, int ntok, float rf, int lane, const AccT (&acc)[2][NG][4]) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int tok = 4 * ng + 2 * (q & 1) + (k & 1);
            const float r = MODE == MAT_DOWN ? 1.0f : __shfl_sync(0xffffffffu, rf, tok);
            if (q >= 2 || tok >= ntok) continue;
            float* out = p.out + (size_t) (MODE == MAT_DENSE ? tok : orow[tok]) * p.ldo;
            if (MODE == MAT_GATEUP) {
                out[lu * 16 + g + 8 * (k >> 1)] = siluf_((float) acc[0][ng][k] * r) * ((float) acc[1][ng][k] * r);
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = lu * 32 + h * 16 + g + 8 * (k >> 1);
                    const float v = MODE == MAT_DOWN ? (float) acc[h][ng][k] : (float) acc[h][ng][k] * r;
                    if (row < p.rows) out[row] = MODE == MAT_DENSE && p.accumulate ? out[row] + v : v;
                }
            }
        }
}

// 1 / rms of a row from its image (shared address of its first block)
__device__ __forceinline__ float nm_row_factor(uint32_t row_s, int KB, float eps) {
    float ss = 0.f;
    for (int c = 0; c < KB; ++c) ss += lds_f32<NI_RS>(row_s + c * NI_BYTES);
    return rsqrtf(ss / (float) (KB * 256) + eps);
}

// A block's items are the tiles of units [u0, u1) (a unit: one tile row across the columns), dealt to its warps in equal contiguous
// shares (mmv_core.cuh: units cut by share boundaries leave their pieces in shared memory, and after one barrier the warp with a
// unit's first piece adds the others in warp order).
// Dense products sum in f32, so a row's last bits show where its unit is cut, and a row gives the same bits whatever number of rows it comes with:
// sixteen warps, which small row counts of a large matrix take, share out the eight warps' shares two by two, at the boundary of a unit.
// C > 1 (dense, long rows): C blocks of a cluster share the units and split the columns, each holding its part of the rows' image;
// the partial sums are added in block order through distributed shared memory.  A 2048 x 4096 product at five rows would otherwise
// have every block copy 48 KB of image for one unit.
template <int NG, int MODE, int NW, int SLOTS, int C>
__device__ __forceinline__ void nm_body(const NatParams& p, uint8_t* smem) {
    using AccT = typename MatAcc<MODE>::type;
    using Piece = NatPiece<NG, MODE>;
    constexpr bool MOE = MODE != MAT_DENSE;
    constexpr int NT = NW * 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KB = p.K / 256, KBc = KB / C, nbu = KBc, upj = MODE == MAT_GATEUP ? p.rows / 16 : (p.rows + 31) / 32;
    const int crank = C > 1 ? (int) (blockIdx.x % C) : 0, bid = C > 1 ? (int) (blockIdx.x / C) : (int) blockIdx.x, nblk = (int) gridDim.x / C;
    const uint32_t RS = (uint32_t) ni_row_bytes(KBc);
    Piece* pieces = reinterpret_cast<Piece*>(smem + (size_t) NW * SLOTS * NAT_TILE_BYTES);   // [NW][2]
    uint8_t* pool = reinterpret_cast<uint8_t*>(pieces + NW * 2);                             // row images
    const int pool_rows = MOE ? p.rmax : 4 * NG;
    fnx_job* jobs_s = reinterpret_cast<fnx_job*>(pool + (size_t) pool_rows * RS);
    float* ub = reinterpret_cast<float*>(pool + (size_t) pool_rows * RS);                    // C > 1: the units' partial sums
    const uint64_t policy = nm_stream_policy();
    const uint32_t slots_s = smem_u32(smem) + (uint32_t) warp * (SLOTS * NAT_TILE_BYTES), pool_s = smem_u32(pool);
    // gate|up: the job list is the previous kernel's; down: it is older than the kernel whose rows this one waits for, and that
    // kernel lets dependents start only once it has itself waited for the list
    if (MODE == MAT_GATEUP) {
        pdl_wait();
        pdl_launch_dependents();
    }
    int njobs = 1;
    if (MOE) {
        njobs = min(__ldcg(p.njobs), p.njobs_max);
        const int n8 = p.njobs_max * (int) sizeof(fnx_job) / 8;   // 40 bytes a job
        for (int i = tid; i < n8; i += NT) reinterpret_cast<uint2*>(jobs_s)[i] = __ldcg(reinterpret_cast<const uint2*>(p.jobs) + i);
        __syncthreads();
    }
    const unsigned total = (unsigned) njobs * upj;
    const int u0 = (int) (total * bid / nblk), u1 = (int) (total * (bid + 1) / nblk);
    bool waited = MODE == MAT_GATEUP;
    for (int uc = u0; uc < u1 || !waited;) {
        // the pass's jobs: as many as fit the row pool
        const int j0 = uc / upj;
        int j1 = njobs, nrow = p.T;
        if (MOE) {
            const int jend = uc < u1 ? (u1 - 1) / upj + 1 : j0;
            nrow = 0;
            for (j1 = j0; j1 < jend; ++j1) {
                const int n = min(jobs_s[j1].n, 4);
                if (j1 > j0 && nrow + n > p.rmax) break;
                nrow += n;
            }
        }
        const int ue = min(u1, j1 * upj);
        const unsigned N = ue > uc ? (unsigned) (ue - uc) * nbu : 0u;
        int i0, i1;
        if (MODE == MAT_DENSE && NW == 16) {
            const int a = (int) (N * (warp >> 1) / 8), b = (int) (N * ((warp >> 1) + 1) / 8), m = max(a, min(b, ((a + b) / 2 + nbu / 2) / nbu * nbu));
            i0 = warp & 1 ? m : a;
            i1 = warp & 1 ? b : m;
        } else {
            i0 = (int) (N * warp / NW);
            i1 = (int) (N * (warp + 1) / NW);
        }
        if (MODE == MAT_GATEUP) {   // the jobs' rows
            const int per = KB * (NI_BYTES / 16);
            for (int i = tid; i < nrow * per; i += NT) {
                int r = i / per, j = j0;
                const int at = i - r * per, dr = r;
                for (int n; r >= (n = min(jobs_s[j].n, 4)); ++j) r -= n;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pool_s + dr * RS + at * 16), "l"(p.img + (size_t) jobs_s[j].y[r] * RS + at * 16) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        // ---- the copies run ahead of the items: each lane's 128 bytes of a tile, and one of eight lanes' 32 bytes of its scales
        auto job_base = [&](int j) {
            if (!MOE) return p.W;
            const int e = jobs_s[j].w;
            return e >= p.E ? p.Wsh : p.W + (size_t) (e - p.e_base) * p.expert_stride;
        };
        // the next item to fetch: block ab of unit au (of the job, in expert modes)
        int aj = MOE ? (uc + i0 / nbu) / upj : 0, au = MOE ? (uc + i0 / nbu) % upj : uc + i0 / nbu, ab = i0 % nbu;
        const uint8_t* asrc = i0 < i1 ? job_base(aj) + ((size_t) au * KB + crank * KBc + ab) * NAT_TILE_BYTES + lane * 16 : nullptr;
        auto fetch = [&](int item, int into) {   // (items in order, every one once)
            if (item < i1) {
                const uint32_t dst = slots_s + (uint32_t) (into * NAT_TILE_BYTES + lane * 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        nm_cp_stream(dst + h * NAT_HALF_BYTES + j * 512, asrc + h * NAT_HALF_BYTES + j * 512, policy);
                    if (lane < 8)
                        nm_cp_stream(dst + h * NAT_HALF_BYTES + NAT_META, asrc + h * NAT_HALF_BYTES + NAT_META, policy);
                }
                asrc += NAT_TILE_BYTES;
                if (MOE || C > 1) {
                    if (++ab == nbu) {
                        ab = 0;
                        if (C > 1) asrc += (size_t) (KB - KBc) * NAT_TILE_BYTES;
                        if (MOE && ++au == upj) {
                            au = 0;
                            ++aj;
                            if (item + 1 < i1) asrc = job_base(aj) + lane * 16;
                        }
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) fetch(i0 + k, k);
        if (!waited) {
            pdl_wait();   // from here on: what the previous kernel wrote (the rows)
            pdl_launch_dependents();
            waited = true;
            if (C == 1 && u0 >= u1) break;
        }
        if (MODE == MAT_DENSE) {
            const int per = KBc * (NI_BYTES / 16);
            const uint8_t* src = p.img + (size_t) crank * KBc * NI_BYTES;
            const size_t grs = ni_row_bytes(KB);
            for (int i = tid; i < nrow * per; i += NT) {
                const int r = i / per, at = i - r * per;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pool_s + r * RS + at * 16), "l"(src + r * grs + at * 16) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else if (MODE == MAT_DOWN) {   // the rows of the pass's jobs, quantised here (two 256-column blocks a row at 512 columns)
            for (int id = warp; id < nrow * KB; id += NW) {
                int r = id % nrow, j = j0;
                const int dr = r, blk = id / nrow;
                for (int n; r >= (n = min(jobs_s[j].n, 4)); ++j) r -= n;
                const float* src = p.x + (size_t) jobs_s[j].out[r] * p.K + blk * 256 + lane * 8;
                const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
                const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                ni_quant_at(pool + dr * RS + blk * NI_BYTES, v, 0.f, lane);
            }
        } else {
            asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS) : "memory");   // the rows were the first group
        }
        __syncthreads();
        Piece* mine = pieces + warp * 2;
        if (lane == 0) {
            mine[0].unit = i0 < i1 ? -1 : -2;
            mine[1].unit = -1;
        }
        // the lane's columns: row n & 3 of its group at level n / 4.  Expert modes: a job's missing rows read its last one (a dense group's
        // lie in the pool, whatever they hold); either way the columns are dropped.
        const int g = lane >> 2, q = lane & 3;
        uint32_t xb0 = 0, x00 = 0, x10 = 0;
        auto columns = [&](uint32_t base, int n) {
            const int last = MOE ? n - 1 : 4 * NG, r0 = (2 * q) & 3;
            xb0 = base + (uint32_t) min(g & 3, last) * RS + (uint32_t) (g >> 2) * 256u + q * 16;
            x00 = base + (uint32_t) min(r0, last) * RS + NI_SCALE + (uint32_t) (q >> 1) * 4u;
            x10 = base + (uint32_t) min(r0 + 1, last) * RS + NI_SCALE + (uint32_t) (q >> 1) * 4u;
        };
        int cur_job = -1, ntok = p.T, b_lo = 0;
        float rf = 1.0f;
        if (!MOE) {
            columns(pool_s, p.T);
            if (p.normed && lane < p.T) rf = nm_row_factor(pool_s + lane * RS, KB, p.eps);   // (normed rows are never split: C == 1)
        }
        AccT acc[2][NG][4];
        int b = i0 % nbu, u = uc + i0 / nbu, slot = 0;
        // a unit's sums: written, or (columns split) left for the cluster
        auto done = [&](int unit) {
            if (C > 1) {
                if ((lane & 3) < 2) {
                    const int l16 = (lane >> 2) * 2 + (lane & 3);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int ng = 0; ng < NG; ++ng)
                            *reinterpret_cast<float4*>(ub + (((size_t) (unit - u0) * 2 + h) * NG + ng) * 64 + l16 * 4) =
                                make_float4((float) acc[h][ng][0], (float) acc[h][ng][1], (float) acc[h][ng][2], (float) acc[h][ng][3]);
                }
            } else {
                nm_write<NG, MODE, AccT>(p, MOE ? unit % upj : unit, MOE ? jobs_s[unit / upj].out : nullptr, ntok, rf, lane, acc);
            }
        };
        for (int s = i0; s < i1; ++s) {
            if (b == 0 || s == i0) {
                b_lo = b;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[h][ng][k] = 0;
                if (MOE && u / upj != cur_job) {
                    cur_job = u / upj;
                    int r = 0;
                    for (int j = j0; j < cur_job; ++j) r += min(jobs_s[j].n, 4);
                    ntok = min(jobs_s[cur_job].n, 4);
                    columns(pool_s + (uint32_t) r * RS, ntok);
                    if (MODE == MAT_GATEUP && p.normed) rf = lane < ntok ? nm_row_factor(pool_s + (uint32_t) (r + lane) * RS, KB, p.eps) : 1.0f;
                }
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
            __syncwarp();   // (the scales came in by other lanes' copies)
            const uint32_t off = (uint32_t) b * NI_BYTES, tile_s = slots_s + (uint32_t) (slot * NAT_TILE_BYTES);
            nm_item<NG, AccT>(tile_s, xb0 + off, x00 + off, x10 + off, 4u * RS, lane, acc);
            __syncwarp();   // every lane is done with the slot
            fetch(s + SLOTS, slot);
            slot = slot + 1 == SLOTS ? 0 : slot + 1;
            if (b == nbu - 1 || s == i1 - 1) {
                // level 1 (threads q = 0, 1) + level 2 (q = 2, 3) of the same rows
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[h][ng][k] += __shfl_xor_sync(0xffffffffu, acc[h][ng][k], 2);
                if (b_lo == 0 && b == nbu - 1) {
                    done(u);
                } else {
                    Piece* ps = mine + (b_lo == 0 ? 1 : 0);
                    if (lane == 0) {
                        ps->unit = u;
                        ps->b_hi = b + 1;
                    }
                    if ((lane & 3) < 2) {
                        const int l16 = (lane >> 2) * 2 + (lane & 3);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                                for (int k = 0; k < 4; ++k) ps->v[((h * NG + ng) * 16 + l16) * 4 + k] = acc[h][ng][k];
                    }
                }
            }
            if (++b == nbu) {
                b = 0;
                ++u;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        {   // units cut by share boundaries (the warp's last unit: ntok and rf are those of its job)
            const Piece* first = pieces + warp * 2 + 1;
            const int fu = first->unit;
            if (fu >= 0) {
                const int l16 = (lane >> 2) * 2 + (lane & 3);
                const bool holder = (lane & 3) < 2;
#pragma unroll
                for (int i = 0; i < 2 * NG * 4; ++i) acc[i / (4 * NG)][(i / 4) % NG][i & 3] = holder ? first->v[((i / 4) * 16 + l16) * 4 + (i & 3)] : (AccT) 0;
                for (int ww = warp + 1; ww < NW; ++ww) {
                    const Piece* c = pieces + ww * 2;
                    if (c->unit == -2) continue;
                    if (c->unit != fu) break;
                    if (holder)
#pragma unroll
                        for (int i = 0; i < 2 * NG * 4; ++i) acc[i / (4 * NG)][(i / 4) % NG][i & 3] += c->v[((i / 4) * 16 + l16) * 4 + (i & 3)];
                    if (c->b_hi == nbu) break;
                }
                done(fu);
            }
        }
        uc = ue;
        if (uc < u1) __syncthreads();   // the row images and the pieces are rewritten by the next pass
        if (C > 1) break;
    }
    if constexpr (C > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        const int n = (u1 - u0) * 2 * NG * 64;
        cluster.sync();
        for (int i = crank * NT + tid; i < n; i += C * NT) {
            const int k = i & 3, l16 = (i >> 2) & 15, ng = (i >> 6) % NG, h = ((i >> 6) / NG) & 1, un = (i >> 6) / NG / 2;
            const int tok = 4 * ng + 2 * (l16 & 1) + (k & 1), row = (u0 + un) * 32 + h * 16 + (l16 >> 1) + 8 * (k >> 1);
            if (tok >= p.T || row >= p.rows) continue;
            float* dst = p.out + (size_t) tok * p.ldo + row;
            const float old = p.accumulate ? *dst : 0.f;
            float s = 0.f;
#pragma unroll
            for (int r = 0; r < C; ++r) s += cluster.map_shared_rank(ub, r)[i];
            *dst = p.accumulate ? old + s : s;
        }
        cluster.sync();   // no block may leave while a neighbour still reads its sums
    }
}

// two blocks an SM, up to two row groups (nm_item): the next kernel's may be resident while this one's drain
template <int NG, int MODE, int NW, int SLOTS>
__global__ void __launch_bounds__(NW * 32, NW > 12 || NG > 2 ? 1 : 2) k_nat_mmv(const NatParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    nm_body<NG, MODE, NW, SLOTS, 1>(p, smem);
}
constexpr int NM_SPLIT = 4;
template <int NG, int NW, int SLOTS>
__global__ void __cluster_dims__(NM_SPLIT, 1, 1) __launch_bounds__(NW * 32, NW > 12 || NG > 2 ? 1 : 2) k_nat_mmv_split(const NatParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    nm_body<NG, MAT_DENSE, NW, SLOTS, NM_SPLIT>(p, smem);
}

constexpr size_t NM_SMEM = 220 * 1024;   // a block's at most
// the tiles in flight and the cut units' pieces of a form, rows and jobs aside
template <int NG, int MODE, int NW, int SLOTS>
constexpr size_t nm_fixed_bytes() {
    return (size_t) NW * SLOTS * NAT_TILE_BYTES + (size_t) NW * 2 * sizeof(NatPiece<NG, MODE>);
}

template <int NG, int MODE, int NW, int SLOTS>
static int launch_nat(NatParams p, cudaStream_t st) {
    const size_t row = ni_row_bytes(p.K / 256);
    size_t smem = nm_fixed_bytes<NG, MODE, NW, SLOTS>();
    if (MODE == MAT_DENSE) {
        smem += 4 * NG * row;
    } else {
        // rows of the jobs a block meets in one pass: its units lie in one to three jobs of a row or so each, one of them perhaps the shared
        // expert's four (a second pass drains the copies: four rows instead of eight cost 1.3 us at five rows); with eight a gate|up
        // and a down block fit an SM together
        smem += (size_t) p.njobs_max * sizeof(fnx_job);
        p.rmax = 8;
        while (p.rmax > 4 && (p.rmax * row > 40 * 1024 || smem + p.rmax * row > NM_SMEM)) --p.rmax;
        smem += p.rmax * row;
    }
    if (smem > NM_SMEM) return fail(FNX_E_ARG, "nat_mmv: %d columns, %d rows, %d jobs need %zu bytes of shared memory", p.K, 4 * NG, p.njobs_max, smem);
    if (int rc = set_smem_limit((const void*) k_nat_mmv<NG, MODE, NW, SLOTS>, (int) NM_SMEM)) return rc;
    const cudaError_t le = launch_dep(true, k_nat_mmv<NG, MODE, NW, SLOTS>, dim3(sm_count()), dim3(NW * 32), smem, st, p);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "nat_mmv: launch failed: %s", cudaGetErrorString(le));
}

template <int NG, int NW, int SLOTS>
static int launch_nat_split(NatParams p, cudaStream_t st) {
    const int units = (p.rows + 31) / 32, most = sm_count() / NM_SPLIT, per = (units + most - 1) / most, clusters = (units + per - 1) / per;
    const size_t smem = nm_fixed_bytes<NG, MAT_DENSE, NW, SLOTS>() + 4 * NG * ni_row_bytes(p.K / 256 / NM_SPLIT) + (size_t) per * 2 * NG * 64 * sizeof(float);
    if (smem > NM_SMEM) return fail(FNX_E_ARG, "nat_mmv: %d columns, %d rows need %zu bytes of shared memory", p.K, 4 * NG, smem);
    if (int rc = set_smem_limit((const void*) k_nat_mmv_split<NG, NW, SLOTS>, (int) NM_SMEM)) return rc;
    const cudaError_t le = launch_dep(true, k_nat_mmv_split<NG, NW, SLOTS>, dim3(clusters * NM_SPLIT), dim3(NW * 32), smem, st, p);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "nat_mmv: launch failed: %s", cudaGetErrorString(le));
}

int nat_dense(const uint8_t* W, int rows, int K, const uint8_t* img, bool normed, float eps, int T, float* y, int ldy, int accumulate, cudaStream_t st) {
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS && rows % 16 == 0 && K % 256 == 0, "nat_dense: %d rows of %d x %d", T, rows, K);
    const size_t row = ni_row_bytes(K / 256);
    // columns split over a cluster: long rows that are not normed, and few enough units that their partial sums fit
    const bool split = K >= 4096 && K % (256 * NM_SPLIT) == 0 && !normed && (rows + 31) / 32 <= 8 * (sm_count() / NM_SPLIT);
    // a matrix that streams for some 10 us (a vocabulary's): sixteen warps, as for many expert jobs below, where their tiles leave room for the
    // rows (one group of four always, two up to 3,072 columns; three groups' sums would not leave the registers of sixteen warps).
    // Either number of warps gives the same bits.
    const bool large = !split && nat_bytes(rows, K) > ((size_t) 64 << 20), large2 = large && nm_fixed_bytes<2, MAT_DENSE, 16, 2>() + 8 * row <= NM_SMEM;
    // up to five groups of four rows a launch (more would leave no registers), fewer where their image would not fit beside the tiles
    int most = 5;
    while (most > 1 && 4 * most * (split ? ni_row_bytes(K / 256 / NM_SPLIT) : row) > 100 * 1024) --most;
    const int groups = (T + 3) / 4, calls = (groups + most - 1) / most, per = (groups + calls - 1) / calls;
    for (int g0 = 0; g0 < groups; g0 += per) {
        NatParams p{};
        const int ng = groups - g0 < per ? groups - g0 : per;
        p.W = W; p.T = T - 4 * g0 < 4 * ng ? T - 4 * g0 : 4 * ng; p.img = img + (size_t) 4 * g0 * row; p.normed = normed; p.eps = eps;
        p.out = y + (size_t) 4 * g0 * ldy; p.ldo = ldy; p.rows = rows; p.K = K; p.accumulate = accumulate;
        int rc;
        if (split) {
            switch (ng) {
                case 1: rc = launch_nat_split<1, 8, 2>(p, st); break;
                case 2: rc = launch_nat_split<2, 8, 2>(p, st); break;
                case 3: rc = launch_nat_split<3, 8, 2>(p, st); break;
                case 4: rc = launch_nat_split<4, 8, 2>(p, st); break;
                default: rc = launch_nat_split<5, 8, 2>(p, st); break;
            }
        } else {
            switch (ng) {
                case 1: rc = large ? launch_nat<1, MAT_DENSE, 16, 2>(p, st) : launch_nat<1, MAT_DENSE, 8, 3>(p, st); break;
                case 2: rc = large2 ? launch_nat<2, MAT_DENSE, 16, 2>(p, st) : launch_nat<2, MAT_DENSE, 8, 3>(p, st); break;
                case 3: rc = launch_nat<3, MAT_DENSE, 8, 2>(p, st); break;
                case 4: rc = launch_nat<4, MAT_DENSE, 8, 2>(p, st); break;
                default: rc = launch_nat<5, MAT_DENSE, 8, 2>(p, st); break;
            }
        }
        if (rc != FNX_OK) return rc;
    }
    return FNX_OK;
}

// From this many jobs on sixteen warps, which hide more of an item's latency, are worth more than a second resident block: 205 jobs 50 -> 45 us (gate|up)
// and 28 -> 24 us (down).  A window of twelve layers, ten picks a row, eight and sixteen warps, us: two rows (21 jobs) 601 and 611, three (31) 657 and 654, four 700
// and 694, five 787 and 772, six 837 and 813.
constexpr int NM_MANY_JOBS = 30;
// (the job list, 40 bytes a job, has to fit beside sixteen warps' tiles and four rows: 896 jobs at 2,048 columns; the bits are the same either way)
template <int MODE>
static int launch_nat_jobs(const NatParams& p, cudaStream_t st) {
    const size_t least = nm_fixed_bytes<1, MODE, 16, 2>() + 4 * ni_row_bytes(p.K / 256) + (size_t) p.njobs_max * sizeof(fnx_job);
    return p.njobs_max > NM_MANY_JOBS && least <= NM_SMEM ? launch_nat<1, MODE, 16, 2>(p, st) : launch_nat<1, MODE, 8, 2>(p, st);
}

int nat_gate_up(const uint8_t* Wgu, size_t stride, int e_base, const uint8_t* Wsh, int E, const fnx_job* jobs, const int* njobs, int njobs_max, const uint8_t* img,
                float eps, int H, int F, float* h, cudaStream_t st) {
    NatParams p{};
    p.W = Wgu; p.expert_stride = stride; p.e_base = e_base; p.Wsh = Wsh; p.E = E; p.jobs = jobs; p.njobs = njobs; p.njobs_max = njobs_max; p.img = img; p.normed = 1;
    p.eps = eps; p.out = h; p.ldo = F; p.rows = F; p.K = H;
    return launch_nat_jobs<MAT_GATEUP>(p, st);
}

int nat_down(const uint8_t* Wdn, size_t stride, int e_base, const uint8_t* Wsh, int E, const fnx_job* jobs, const int* njobs, int njobs_max, const float* h, int H,
             int F, float* part, cudaStream_t st) {
    NatParams p{};
    p.W = Wdn; p.expert_stride = stride; p.e_base = e_base; p.Wsh = Wsh; p.E = E; p.jobs = jobs; p.njobs = njobs; p.njobs_max = njobs_max; p.x = h;
    p.out = part; p.ldo = H; p.rows = H; p.K = F;
    return launch_nat_jobs<MAT_DOWN>(p, st);
}

// ------------------------------------------------------------------------------------------------ images of rows
// one warp per (256-column block, row)
__global__ void __launch_bounds__(32) k_nat_rows_image(const float* __restrict__ x, int ldx, const float* __restrict__ norm_w, uint8_t* __restrict__ img) {
    pdl_wait();
    pdl_launch_dependents();
    const int blk = blockIdx.x, t = blockIdx.y, lane = threadIdx.x, c = blk * 256 + lane * 8;
    const float4 a = *reinterpret_cast<const float4*>(x + (size_t) t * ldx + c), b = *reinterpret_cast<const float4*>(x + (size_t) t * ldx + c + 4);
    float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const float ss = ni_norm8(v, norm_w ? norm_w + c : nullptr);
    ni_quant(img, gridDim.x, v, ss, t, blk, lane);
}

__global__ void __launch_bounds__(32) k_nat_embed_image(const __half* __restrict__ table, const int* __restrict__ tok, float* __restrict__ R,
                                                        const float* __restrict__ norm_w, uint8_t* __restrict__ img) {
    pdl_wait();
    pdl_launch_dependents();
    const int blk = blockIdx.x, t = blockIdx.y, lane = threadIdx.x, c = blk * 256 + lane * 8, H = gridDim.x * 256;
    const uint4 h = *reinterpret_cast<const uint4*>(table + (size_t) tok[t] * H + c);
    const __half2* h2 = reinterpret_cast<const __half2*>(&h);
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h2[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
    float* o = R + (size_t) t * H + c;
    *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
    if (!img) return;
    const float ss = ni_norm8(v, norm_w ? norm_w + c : nullptr);
    ni_quant(img, gridDim.x, v, ss, t, blk, lane);
}

int nat_rows_image(const float* x, int ldx, int T, int K, const float* norm_w, uint8_t* img, cudaStream_t st) {
    FNX_REQUIRE(x && img && T >= 1 && K % 256 == 0 && ldx % 4 == 0, "nat_rows_image: %d rows of %d", T, K);
    const cudaError_t le = launch_dep(true, k_nat_rows_image, dim3(K / 256, T), dim3(32), 0, st, x, ldx, norm_w, img);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "nat_rows_image: launch failed: %s", cudaGetErrorString(le));
}

int nat_embed_image(const __half* table, const int* tok, int T, int H, float* R, const float* norm_w, uint8_t* img, cudaStream_t st) {
    FNX_REQUIRE(table && tok && R && T >= 1 && H % 256 == 0, "nat_embed_image: %d rows of %d", T, H);
    const cudaError_t le = launch_dep(true, k_nat_embed_image, dim3(H / 256, T), dim3(32), 0, st, table, tok, R, norm_w, img);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "nat_embed_image: launch failed: %s", cudaGetErrorString(le));
}

// ------------------------------------------------------------------------------------------------ layouts
__global__ void __launch_bounds__(128) k_nat_pack(const uint8_t* __restrict__ ggml, uint8_t* __restrict__ nat, size_t rows, size_t row0, size_t n, int KB, int gate_up) {
    __shared__ uint32_t grid[512];
    for (int i = threadIdx.x; i < 512; i += blockDim.x) grid[i] = g_grid_nat[i];
    __syncthreads();
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * KB) return;
    const size_t row = row0 + i / KB;
    const int b = (int) (i % KB);
    uint8_t blk[IQ3S_BLOCK_BYTES];
    const uint8_t* src = ggml + i * IQ3S_BLOCK_BYTES;
    for (int k = 0; k < IQ3S_BLOCK_BYTES; ++k) blk[k] = src[k];
    nat_put_block(nat + nat_half_at(row / 16, rows / 16, b, KB, gate_up), (int) (row % 16), blk, grid);
}

__global__ void __launch_bounds__(128) k_nat_unpack(const uint8_t* __restrict__ nat, uint8_t* __restrict__ tiles, size_t rows, int KB, int gate_up) {
    __shared__ uint16_t inv[4096];
    for (int e = threadIdx.x; e < 512; e += blockDim.x) {
        uint32_t key = 0;
        for (int j = 0; j < 4; ++j) key |= ((g_grid_nat[e] >> (8 * j + 1)) & 7u) << (3 * j);
        inv[key] = (uint16_t) e;
    }
    __syncthreads();
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * KB) return;
    const size_t row = i / KB;
    const int b = (int) (i % KB);
    uint8_t blk[IQ3S_BLOCK_BYTES];
    nat_get_block(nat + nat_half_at(row / 16, rows / 16, b, KB, gate_up), (int) (row % 16), blk, inv);
    tile_put_block(tiles + ((row / 16) * KB + b) * TILE_BYTES, (int) (row % 16), blk);
}

int nat_pack(const uint8_t* ggml, uint8_t* nat, size_t rows, size_t row0, size_t n, size_t cols, bool gate_up, cudaStream_t st) {
    FNX_REQUIRE(ggml && nat && rows % (gate_up ? 32 : 16) == 0 && row0 % 16 == 0 && n % 16 == 0 && n && row0 + n <= rows && cols % 256 == 0, "nat_pack: rows [%zu, + %zu) of %zu x %zu", row0, n, rows, cols);
    const size_t w = n * (cols / 256);
    k_nat_pack<<<(unsigned) ((w + 127) / 128), 128, 0, st>>>(ggml, nat, rows, row0, n, (int) (cols / 256), gate_up);
    FNX_LAUNCH_OK("nat_pack");
    return FNX_OK;
}

int nat_unpack(const uint8_t* nat, uint8_t* tiles, size_t rows, size_t cols, bool gate_up, cudaStream_t st) {
    FNX_REQUIRE(nat && tiles && rows % (gate_up ? 32 : 16) == 0 && cols % 256 == 0, "nat_unpack: %zu x %zu", rows, cols);
    const size_t w = rows * (cols / 256);
    k_nat_unpack<<<(unsigned) ((w + 127) / 128), 128, 0, st>>>(nat, tiles, rows, (int) (cols / 256), gate_up);
    FNX_LAUNCH_OK("nat_unpack");
    return FNX_OK;
}

}  // namespace fnxb
