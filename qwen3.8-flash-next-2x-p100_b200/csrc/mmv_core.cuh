// The inner pieces of the operators' IQ3_S matrix x few-rows product (mmv_stage.cuh): codebook table,
// one 16 x 256 tile against quantised activation cells, and the two-level int8 quantiser of activation rows.
//
// Activation image (in shared or global memory, same layout): rows in groups of four,
//   cells  uint2 [group][sub-block sbG = k / 32][column n = (row & 3) + 4 * level][q = (k % 32) / 8]   8 int8 each
//   scales float [group][block = k / 256][column n]                                                  d, d / 256
// so that the 8 columns of one mma.sync.m16n8k32.s8 hold both levels of up to four rows.
#pragma once

#include <cuda_fp16.h>

#include "fnx_common.cuh"
#include "iq3s_grid.h"
#include "iq3s_tile.h"

namespace fnxb {

__device__ static const uint32_t g_grid_core[512] = {FNX_IQ3S_GRID_VALUES};

constexpr int CORE_TABLE_BYTES = 512 * 128;
// the codebook, one copy per bank: entry e at byte e * 128 + 4 * lane
__device__ __forceinline__ void core_fill_table(uint8_t* table, int tid, int nthreads) {
    // a warp writes 32 entries: each store instruction covers 4 whole entries (512 contiguous bytes: no bank conflicts)
    const int warp = tid >> 5, lane = tid & 31, nwarp = nthreads >> 5;
    for (int e0 = warp * 32; e0 < 512; e0 += nwarp * 32) {
        const uint32_t mine = g_grid_core[e0 + lane];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t v = __shfl_sync(0xffffffffu, mine, 4 * i + (lane >> 3));
            *reinterpret_cast<uint4*>(table + (e0 + 4 * i) * 128 + lane * 16) = make_uint4(v, v, v, v);
        }
    }
}

__device__ __forceinline__ void core_mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0), "r"(0), "r"(0), "r"(0));
}

// four s32 -> four saturated s8 in one word (byte 0 = a)
__device__ __forceinline__ uint32_t core_pack_s8x4(int a, int b, int c, int d) {
    uint32_t hi, r;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(d), "r"(c));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
    return r;
}

// shared-memory loads by 32-bit shared address plus a compile-time offset that rides in the instruction: no 64-bit
// generic pointer arithmetic and no address adds in the decode loop
template <int OFF = 0>
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF = 0>
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint16_t v;
    asm("ld.shared.u16 %0, [%1+%2];" : "=h"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF = 0>
__device__ __forceinline__ uint2 lds_v2(uint32_t a) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF = 0>
__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
    uint4 v;
    asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF = 0>
__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}

template <int I>
__device__ __forceinline__ uint32_t core_decode(const uint32_t (&S)[5], const uint32_t (&G)[2], uint32_t table_s, uint32_t lane4) {
    // (field & 0xFF80) | 4 lane: one logic op; the table's (uniform) shared address rides in the load's address
    const uint32_t off = tile_field<I>(S) | lane4;
    const uint32_t mag = lds_u32(table_s + off);
    return tile_apply_sign(mag, tile_sign_mask<I>(G));
}

// What one lane reads of the activations: for each row group, its B cells (column = lane / 4) and the scales of its
// two C columns (2 q, 2 q + 1).  Every column is read: what an empty row's cells hold stays in that row's own sums.
template <int NG>
struct LaneX {
    uint32_t b[NG];     // shared addresses
    uint32_t s0[NG];
    uint32_t s1[NG];
    float r0[NG], r1[NG];   // factors of the two C columns' rows (1 / rms of a normed row, else 1)
};

// lane pointers: group ng holds image rows 4 ng .. 4 ng + 3
template <int NG>
__device__ __forceinline__ void lane_x_set(LaneX<NG>& lx, const uint2* xq, const float* xs, int K, int lane) {
    const int q = lane & 3, KB = K / 256;
#pragma unroll
    for (int ng = 0; ng < NG; ++ng) {
        lx.b[ng] = smem_u32(xq + (size_t) ng * (K / 32) * 32 + lane);
        lx.s0[ng] = smem_u32(xs + (size_t) ng * KB * 8 + 2 * q);
        lx.s1[ng] = lx.s0[ng] + 4u;
    }
}

template <int NG, int SB>
__device__ __forceinline__ void core_sub_block(const uint32_t (&S0)[5], const uint32_t (&G0)[2], const uint32_t (&S1)[5], const uint32_t (&G1)[2],
                                               uint2 sc0, uint2 sc1, uint32_t table_s, uint32_t lane4, const uint32_t (&bx)[NG],
                                               int (&accI)[NG][4]) {
    const uint32_t a0 = core_decode<2 * SB>(S0, G0, table_s, lane4);
    const uint32_t a2 = core_decode<2 * SB + 1>(S0, G0, table_s, lane4);
    const uint32_t a1 = core_decode<2 * SB>(S1, G1, table_s, lane4);
    const uint32_t a3 = core_decode<2 * SB + 1>(S1, G1, table_s, lane4);
    // sc0 / sc1: the rows' eight scales 1 + 2 s as bytes (even sub-blocks in .x, odd in .y): one byte extract each
    int w0, w1;
    {
        const uint32_t a = SB & 1 ? sc0.y : sc0.x, b = SB & 1 ? sc1.y : sc1.x;
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(w0) : "r"(a), "r"(0u), "r"(0x4440u + (SB >> 1)));
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(w1) : "r"(b), "r"(0u), "r"(0x4440u + (SB >> 1)));
    }
#pragma unroll
    for (int ng = 0; ng < NG; ++ng) {
        const uint2 b = lds_v2<SB * 256>(bx[ng]);   // bx: this lane's cells of the block's first sub-block
        int c[4];
        core_mma_s8(c, a0, a1, a2, a3, b.x, b.y);
        accI[ng][0] += w0 * c[0];
        accI[ng][1] += w0 * c[1];
        accI[ng][2] += w1 * c[2];
        accI[ng][3] += w1 * c[3];
    }
}

// One item: tile (16 rows x 256 columns, block `blk` of its rows) against the lane's activation cells; adds into
// acc[ng][0..3] = (row g, col 2q), (row g, col 2q+1), (row g+8, col 2q), (row g+8, col 2q+1).
// AccT double: the block's four products are exact in double and their sums carry ~2^-53 relative error, so that the
// rounded result does not depend on where a row's K-sum was cut into pieces (expert modes, where the cuts move with the
// number of jobs: a row must give the same bits whatever else is in the window).
template <int NG, typename AccT>
__device__ __forceinline__ void core_item(uint32_t tile_s, uint32_t table_s, const LaneX<NG>& lx, int blk, int lane, AccT (&acc)[NG][4]) {
    const int g = lane >> 2;
    const uint32_t lane4 = (uint32_t) lane * 4u;
    const uint32_t a16 = tile_s + lane * 16, a8 = tile_s + lane * 8, a2 = tile_s + lane * 2, ag4 = tile_s + g * 4, ag2 = tile_s + g * 2;
    const uint4 i0 = lds_v4<TILE_IDX>(a16);
    const uint4 i1 = lds_v4<TILE_IDX + 512>(a16);
    const uint2 s0 = lds_v2<TILE_SGN>(a8);
    const uint2 s1 = lds_v2<TILE_SGN + 256>(a8);
    const uint32_t t0 = lds_u16<TILE_TAIL>(a2);
    const uint32_t t1 = lds_u16<TILE_TAIL + 64>(a2);
    const uint32_t sn0 = lds_u32<TILE_SCL>(ag4);
    const uint32_t sn1 = lds_u32<TILE_SCL + 32>(ag4);
    // nibbles -> bytes 1 + 2 s: even sub-blocks (low nibbles) and odd ones (high nibbles)
    const uint2 sc0 = make_uint2((sn0 & 0x0F0F0F0Fu) * 2u + 0x01010101u, ((sn0 >> 4) & 0x0F0F0F0Fu) * 2u + 0x01010101u);
    const uint2 sc1 = make_uint2((sn1 & 0x0F0F0F0Fu) * 2u + 0x01010101u, ((sn1 >> 4) & 0x0F0F0F0Fu) * 2u + 0x01010101u);
    const float d0 = __half2float(__ushort_as_half((unsigned short) lds_u16<TILE_D>(ag2)));
    const float d1 = __half2float(__ushort_as_half((unsigned short) lds_u16<TILE_D + 16>(ag2)));
    const uint32_t S0[5] = {i0.x, i0.y, i0.z, i0.w, t0}, S1[5] = {i1.x, i1.y, i1.z, i1.w, t1};
    const uint32_t G0[2] = {s0.x, s0.y}, G1[2] = {s1.x, s1.y};
    uint32_t bx[NG];
#pragma unroll
    for (int ng = 0; ng < NG; ++ng) bx[ng] = lx.b[ng] + (uint32_t) blk * 2048u;
    int accI[NG][4];
#pragma unroll
    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
        for (int i = 0; i < 4; ++i) accI[ng][i] = 0;
    core_sub_block<NG, 0>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 1>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 2>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 3>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 4>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 5>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 6>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
    core_sub_block<NG, 7>(S0, G0, S1, G1, sc0, sc1, table_s, lane4, bx, accI);
#pragma unroll
    for (int ng = 0; ng < NG; ++ng) {
        const float x0 = lds_f32(lx.s0[ng] + (uint32_t) blk * 32u) * lx.r0[ng], x1 = lds_f32(lx.s1[ng] + (uint32_t) blk * 32u) * lx.r1[ng];
        if constexpr (sizeof(AccT) == 8) {
            acc[ng][0] += (double) (d0 * x0) * (double) accI[ng][0];
            acc[ng][1] += (double) (d0 * x1) * (double) accI[ng][1];
            acc[ng][2] += (double) (d1 * x0) * (double) accI[ng][2];
            acc[ng][3] += (double) (d1 * x1) * (double) accI[ng][3];
        } else {
            acc[ng][0] += d0 * x0 * (float) accI[ng][0];
            acc[ng][1] += d0 * x1 * (float) accI[ng][1];
            acc[ng][2] += d1 * x0 * (float) accI[ng][2];
            acc[ng][3] += d1 * x1 * (float) accI[ng][3];
        }
    }
}

// Quantises 8 consecutive values of one lane (a cell) given the block's maximum over the warp; returns the cells.
// Rounding rides on the FMA pipe: adding 1.5 * 2^23 leaves round-to-nearest-even(x) in the low mantissa bits (its low
// byte is the s8 code), so no value passes through the conversion unit.
__device__ __forceinline__ void core_quant_cell(const float (&x8)[8], float am, uint2& c1, uint2& c2, float& d) {
    constexpr float MAGIC = 12582912.0f;
    d = am * (1.0f / 127.0f);
    const float inv = am > 0.f ? __fdividef(127.0f, am) : 0.f, inv2 = inv * 256.0f;
    uint32_t a8[8], b8[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float ta = fmaf(x8[i], inv, MAGIC);              // |x inv| <= 127
        const float af = ta - MAGIC;
        const float tb = fminf(fmaf(fmaf(-af, d, x8[i]), inv2, MAGIC), MAGIC + 127.0f);   // the residue, in steps of d / 256
        a8[i] = __float_as_uint(ta);
        b8[i] = __float_as_uint(tb);
    }
    auto pack = [](uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
        uint32_t lo, hi, r;
        asm("prmt.b32 %0, %1, %2, 0x0040;" : "=r"(lo) : "r"(v0), "r"(v1));
        asm("prmt.b32 %0, %1, %2, 0x0040;" : "=r"(hi) : "r"(v2), "r"(v3));
        asm("prmt.b32 %0, %1, %2, 0x5410;" : "=r"(r) : "r"(lo), "r"(hi));
        return r;
    };
    c1 = make_uint2(pack(a8[0], a8[1], a8[2], a8[3]), pack(a8[4], a8[5], a8[6], a8[7]));
    c2 = make_uint2(pack(b8[0], b8[1], b8[2], b8[3]), pack(b8[4], b8[5], b8[6], b8[7]));
}

}  // namespace fnxb

// ------------------------------------------------------------------------------------------------ rows -> image
// A quantisation TASK is one 256-column block of one live row, done by one warp (8 values per lane); a warp works on
// a batch of up to QUANT_BATCH tasks at once so that their loads and their warp reductions overlap.  quant_fetch() starts a
// task's loads, quant_finish() turns a batch into image cells and scales at (cells, scales) for image rows t (group
// t / 4, column t % 4).  With norm_w the codes are those of x * w and the block's sum of squares goes to
// rs[t * 16 + blk]: the row's 1 / rms (quant_row_factor) multiplies the products later, it is uniform along the row.
namespace fnxb {
constexpr int QUANT_BATCH = 3;

struct QuantTask {
    const float* src;   // the block's 256 values
    int t, blk;
};

// (the block's norm weights ride with the values: one latency, not two)
__device__ __forceinline__ void quant_fetch(const QuantTask& q, const float* norm_w, int lane, float (&v)[8], float (&w)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(q.src + lane * 8), b = *reinterpret_cast<const float4*>(q.src + lane * 8 + 4);
    if (norm_w) {
        const float4 c = *reinterpret_cast<const float4*>(norm_w + q.blk * 256 + lane * 8), d = *reinterpret_cast<const float4*>(norm_w + q.blk * 256 + lane * 8 + 4);
        w[0] = c.x; w[1] = c.y; w[2] = c.z; w[3] = c.w;
        w[4] = d.x; w[5] = d.y; w[6] = d.z; w[7] = d.w;
    }
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <int NB, int NV>
__device__ __forceinline__ void quant_finish(const QuantTask (&q)[NB], float (&v)[NV][8], const float (&w)[NV][8], int K, const float* norm_w, uint2* cells, float* scales,
                                             float* rs, int lane) {
    static_assert(NB <= NV, "a batch's values");
    const int KB = K / 256;
    float am[NB], ss[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        ss[j] = 0.f;
        if (norm_w) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                ss[j] = fmaf(v[j][i], v[j][i], ss[j]);
                v[j][i] *= w[j][i];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        am[j] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) am[j] = fmaxf(am[j], fabsf(v[j][i]));
    }
    // the batch's maxima (and sums of squares) cross the warp together: five rounds for all of them
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            am[j] = fmaxf(am[j], __shfl_xor_sync(0xffffffffu, am[j], o));
            if (norm_w) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
        }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const int t = q[j].t, blk = q[j].blk, ng = t >> 2, n = t & 3;
        uint2 c1, c2;
        float d;
        core_quant_cell(v[j], am[j], c1, c2, d);
        const int sbG = blk * 8 + (lane >> 2), qq = lane & 3;
        uint2* cell = cells + ((size_t) (ng * (K / 32) + sbG) * 8 + n) * 4 + qq;
        cell[0] = c1;
        cell[16] = c2;
        if (lane == 0) {
            float* sc = scales + (size_t) (ng * KB + blk) * 8;
            sc[n] = d;
            sc[n + 4] = d * (1.0f / 256.0f);
            if (norm_w) rs[t * 16 + blk] = ss[j];
        }
    }
}

// 1 / rms of image row t from the block sums (after the barrier that follows the tasks)
__device__ __forceinline__ float quant_row_factor(const float* rs, int t, int K, float eps) {
    float ss = 0.f;
    for (int c = 0; c < K / 256; ++c) ss += rs[t * 16 + c];
    return rsqrtf(ss / (float) K + eps);
}
}  // namespace fnxb

namespace fnxb {

enum { MAT_DENSE = 0, MAT_GATEUP = 1, MAT_DOWN = 2 };

// accumulator of a row's K-sum: the dense product is cut the same way for any number of rows (float, summed in a fixed
// order); the expert products are cut where the job count puts the warps' shares (double, see core_item)
template <int MODE>
struct MatAcc {
    using type = double;
};
template <>
struct MatAcc<MAT_DENSE> {
    using type = float;
};

// fixed-point image of a float addend: integer sums do not depend on the order of their terms, so rows summed in any
// order (a loop, several kernels, expert-parallel ranks) give the same bits
constexpr float FIX_SCALE = 4294967296.0f;            // 2^32
constexpr double FIX_INV = 1.0 / 4294967296.0;
__device__ __forceinline__ unsigned long long fix_from_float(float v) { return (unsigned long long) __float2ll_rn(v * FIX_SCALE); }
__device__ __forceinline__ float fix_to_float(unsigned long long a) { return (float) ((double) (long long) a * FIX_INV); }

}  // namespace fnxb
