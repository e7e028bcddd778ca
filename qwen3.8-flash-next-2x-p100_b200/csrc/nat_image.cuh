// The activation image that the windows' products read (nat_mmv.cu): rows quantised once, by the kernel that completes them, to two
// int8 levels per 256-column block (x ~ d (q1 + q2 / 256), error <= amax / 65024; the codes are core_quant_cell's), laid out so
// that a lane's operands of one 256-column block are a few 16-byte loads.  Row t lies at t * ni_row_bytes(KB) (the spare bytes put
// neighbouring rows into different halves of the shared-memory banks); its block blk at blk * NI_BYTES:
//   lev * 256     cells of level lev: [pair 0..3][q 0..3] of 16 bytes, the 8 codes of columns 8 q .. 8 q + 7 of sub-blocks 2 pair
//                 and 2 pair + 1
//   512           the levels' scales f32 (d, d / 256), the block's sum of squares f32 (normed rows: the consumers multiply by 1 / rms)
#pragma once

#include "mmv_core.cuh"

namespace fnxb {

constexpr int NI_SCALE = 512, NI_RS = 520, NI_BYTES = 528;

__host__ __device__ __forceinline__ size_t ni_row_bytes(int KB) { return ((size_t) KB * NI_BYTES + 127) / 128 * 128 + 64; }
__host__ __device__ inline size_t ni_bytes(int T, int K) { return (size_t) T * ni_row_bytes(K / 256); }

// one value's two codes (in the words' low bytes: core_quant_cell's) and its block's scale, given the block's maximum
__device__ __forceinline__ void ni_code(float x, float am, uint32_t& a, uint32_t& b, float& d) {
    constexpr float MAGIC = 12582912.0f;
    d = am * (1.0f / 127.0f);
    const float inv = am > 0.f ? __fdividef(127.0f, am) : 0.f, ta = fmaf(x, inv, MAGIC);
    a = __float_as_uint(ta) & 255u;
    b = __float_as_uint(fminf(fmaf(fmaf(-(ta - MAGIC), d, x), inv * 256.0f, MAGIC), MAGIC + 127.0f)) & 255u;
}

// One warp, one 256-column block of a row: v = the lane's 8 values (columns 8 lane ..), times the norm weight where there is one;
// ss = the lane's share of the raw values' sum of squares (not normed: 0).
__device__ __forceinline__ void ni_quant_at(uint8_t* rec, const float (&v)[8], float ss, int lane) {
    float am = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) am = fmaxf(am, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
    }
    uint2 c1, c2;
    float d;
    core_quant_cell(v, am, c1, c2, d);
    const int sb = lane >> 2, q = lane & 3;
    uint8_t* cell = rec + (sb >> 1) * 64 + q * 16 + (sb & 1) * 8;
    *reinterpret_cast<uint2*>(cell) = c1;
    *reinterpret_cast<uint2*>(cell + 256) = c2;
    if (lane == 0) *reinterpret_cast<float4*>(rec + NI_SCALE) = make_float4(d, d * (1.0f / 256.0f), ss, 0.f);
}
__device__ __forceinline__ void ni_quant(uint8_t* img, int KB, const float (&v)[8], float ss, int t, int blk, int lane) {
    ni_quant_at(img + (size_t) t * ni_row_bytes(KB) + (size_t) blk * NI_BYTES, v, ss, lane);
}

// the block's eight values of one lane, squared up and times the norm weights (w null: as they are)
__device__ __forceinline__ float ni_norm8(float (&v)[8], const float* w8) {
    float ss = 0.f;
    if (w8) {
        const float4 a = *reinterpret_cast<const float4*>(w8), b = *reinterpret_cast<const float4*>(w8 + 4);
        const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            ss = fmaf(v[i], v[i], ss);
            v[i] *= w[i];
        }
    }
    return ss;
}

// ---- launchers of nat_mmv.cu (weights in the layout of nat_tile.h)
// y[t][r] (+)= W[r] . x[t], t < T <= FNX_MAX_ROWS, x given as its image (normed: times 1 / rms)
int nat_dense(const uint8_t* W, int rows, int K, const uint8_t* img, bool normed, float eps, int T, float* y, int ldy, int accumulate, cudaStream_t st);
// the expert products of a job list: gate|up + SwiGLU from the rows' image into h [out][F]; down from h into part [out][H]
int nat_gate_up(const uint8_t* Wgu, size_t stride, int e_base, const uint8_t* Wsh, int E, const fnx_job* jobs, const int* njobs, int njobs_max, const uint8_t* img,
                float eps, int H, int F, float* h, cudaStream_t st);
int nat_down(const uint8_t* Wdn, size_t stride, int e_base, const uint8_t* Wsh, int E, const fnx_job* jobs, const int* njobs, int njobs_max, const float* h, int H,
             int F, float* part, cudaStream_t st);
// the image of T rows of x (row stride ldx), normed by norm_w when it is not null
int nat_rows_image(const float* x, int ldx, int T, int K, const float* norm_w, uint8_t* img, cudaStream_t st);
// the embedding rows of tok and, with img, the image of rmsnorm(row) * norm_w
int nat_embed_image(const __half* table, const int* tok, int T, int H, float* R, const float* norm_w, uint8_t* img, cudaStream_t st);
// GGML blocks -> native tiles and native tiles -> interchange tiles (iq3s_tile.h); gate_up: the matrix is [gate; up], whose 16-row tiles
// alternate in the native layout (gate tile i, up tile i), so that a unit of the gate|up product is one contiguous run
// (pack: rows [row0, row0 + n) of a matrix of `rows` rows, from blocks that start at row0)
int nat_pack(const uint8_t* ggml, uint8_t* nat, size_t rows, size_t row0, size_t n, size_t cols, bool gate_up, cudaStream_t st);
int nat_unpack(const uint8_t* nat, uint8_t* tiles, size_t rows, size_t cols, bool gate_up, cudaStream_t st);

}  // namespace fnxb
