// Gated attention's operators: per-head norm + rotary + KV append, window attention (attn_win.cu) and prompt attention.
//
// fnx_attn_prep_append replaces attn_prep_append / k_attn_prep_append (engine/src/kernels.hpp:259,
// engine/src/kernels.cu:1880-1910; norm_rope :513-530).  fnx_attn replaces attn / k_attn_part + k_attn_local +
// k_attn_combine (engine/src/kernels.hpp:238, engine/src/kernels.cu:558-667, 786-803): the same online-softmax
// split over positions, except that one block serves every row of the window for its share of the positions (the
// K and V rows are read once per window, not once per row), the cache is not split across cards by position, and
// a row may see only the window rows on its path to the root (the reference's windows are chains).
#include "attn_core.cuh"
#include "attn_win.h"

namespace fnxb {

// grid (nq + 2 nkv heads, rows, lanes).  Bound by latency (a few hundred KB in all).  EARLY: the rotations, whose frequencies go through a double
// pow, and the norm weights are ready before the rows are (3.3 us a launch with them behind the wait, in a window).  Otherwise nothing is
// read ahead, and the rotations come last, behind the row's barriers (before them: 17.3 against 16.2 us for 200 rows of 18 heads, 256 rotary dims).
// Batched lanes: lane j holds the consecutive rows [lane_row0[j], lane_row0[j + 1]) of sequence lane_seq[j]: a chain that starts at that
// sequence's position pos[seq] and appends to that sequence's caches (GdnLanes / enqueue_rows, engine/src/kernels.hpp:103-110,
// engine/src/engine.cu:1936).
template <bool EARLY>
__global__ void k_attn_prep_append(const AttnPrep a) {
    extern __shared__ float xrow[];   // hd floats
    __shared__ float red[32];
    const int i = threadIdx.x, h = blockIdx.x, t = blockIdx.y, lane = blockIdx.z;
    if (!EARLY) pdl_begin();
    const int row0 = a.lane_seq ? a.lane_row0[lane] : 0, seq = a.lane_seq ? a.lane_seq[lane] : 0;
    const bool live = !a.lane_seq || (seq >= 0 && t < a.lane_row0[lane + 1] - row0);   // (a negative sequence: another rank's lane)
    const int pos0 = live ? a.pos[seq] : 0;
    const bool normed = live && h < a.nq + a.nkv;
    auto rotation = [&]() { return normed ? attn_rotation(pos0 + (a.depth ? a.depth[t] : t), a.nrot, a.rope_base, i) : make_float2(1.f, 0.f); };
    auto weight = [&]() { return normed ? (h < a.nq ? a.qn : a.kn)[i] : 0.f; };
    float2 rot;
    float w;
    if (EARLY) {
        rot = rotation();
        w = weight();
        pdl_begin();
    }
    if (!live) return;
    const size_t crow = (a.lane_seq ? (size_t) seq * a.seq_rows : 0) + pos0 + t;
    attn_prep_body(a.qg, a.ldq, a.k, a.ldk, a.v, a.ldv, [&]() { return EARLY ? w : weight(); }, a.kc, a.vc, a.nq, a.nkv, a.hd, a.nrot, crow,
                   [&]() { return EARLY ? rot : rotation(); }, a.eps, row0 + t, h, i, xrow, red);
}

// The same for a prompt's rows where a head has 256 dims and 64 rotary ones: a warp takes one head of PREP_ROWS rows, lane = dims lane + 32 j, so
// that a rotated pair lies in one lane, nothing is block-wide and the frequency (a double pow) is worked out once a warp.  Bound by the rows' bytes;
// a block a row and head, with its pow and barriers, took 2.2 ms for 38,912 rows against 0.24 ms of them.
// (Its own chain of eight rows takes 5.2 us however few there are: 20 heads, blocks a row and head against this, 48 rows: 4.2 and 5.6 us, 80 rows: 5.8 and
// 5.8, 128 rows: 8.2 and 5.8.)
constexpr int PREP_ROWS = 8, PREP_WARPS = 8, PREP_MANY = 1500;   // from that many (row, head) pairs on
__global__ void __launch_bounds__(PREP_WARPS * 32) k_attn_prep_rows(const AttnPrep a, int T) {
    pdl_begin();
    constexpr int HD = 256, NROT = 64;
    const int h = blockIdx.x, lane = threadIdx.x & 31, ta = ((int) blockIdx.y * PREP_WARPS + (threadIdx.x >> 5)) * PREP_ROWS, tb = min(T, ta + PREP_ROWS), pos0 = *a.pos;
    if (h >= a.nq + a.nkv) {   // a V head: store only
        const int kvh = h - a.nq - a.nkv;
        for (int t = ta; t < tb; ++t) {
            const float* x = a.v + (size_t) t * a.ldv + (size_t) kvh * HD;
            __half* o = a.vc + ((size_t) (pos0 + t) * a.nkv + kvh) * HD;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = x[lane + 32 * j];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[lane + 32 * j] = __float2half_rn(v[j]);
        }
        return;
    }
    const bool isq = h < a.nq;
    const float fe = (float) pow((double) a.rope_base, -2.0 * (double) lane / (double) NROT);   // (attn_rotation's)
    float w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = (isq ? a.qn : a.kn)[lane + 32 * j];
    for (int t0 = ta; t0 < tb; t0 += 2) {   // two rows in flight
        float v[2][8];
        float* x[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = min(t0 + r, tb - 1);
            x[r] = isq ? a.qg + (size_t) t * a.ldq + (size_t) h * 2 * HD : a.k + (size_t) t * a.ldk + (size_t) (h - a.nq) * HD;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[r][j] = x[r][lane + 32 * j];
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = t0 + r;
            // the sums that attn_prep_body takes (a warp_sum of every 32 dims, added in order), so that a row's bits do not depend on the form: the
            // first three of warp_sum's five exchanges halve the values a lane carries
            float q[8], s4[4], s2[2], s1;
#pragma unroll
            for (int j = 0; j < 8; ++j) q[j] = v[r][j] * v[r][j];
#pragma unroll
            for (int j = 0; j < 4; ++j) s4[j] = (lane & 16 ? q[4 + j] : q[j]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? q[j] : q[4 + j], 16);
#pragma unroll
            for (int j = 0; j < 2; ++j) s2[j] = (lane & 8 ? s4[2 + j] : s4[j]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? s4[j] : s4[2 + j], 8);
            s1 = (lane & 4 ? s2[1] : s2[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? s2[0] : s2[1], 4);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) ss += __shfl_sync(0xffffffffu, s1, 4 * j);   // (lanes 4 j: the sum of dims 32 j ..)
            const float n = rsqrtf(ss / (float) HD + a.eps);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[r][j] = v[r][j] * n * w[j];
            float sn, cs;
            sincosf((float) (pos0 + t) * fe, &sn, &cs);
            const float x0 = v[r][0], x1 = v[r][1];
            v[r][0] = x0 * cs - x1 * sn;
            v[r][1] = x0 * sn + x1 * cs;
            if (t >= tb) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) x[r][lane + 32 * j] = v[r][j];
            if (!isq) {
                __half* o = a.kc + ((size_t) (pos0 + t) * a.nkv + (h - a.nq)) * HD;
#pragma unroll
                for (int j = 0; j < 8; ++j) o[lane + 32 * j] = __float2half_rn(v[r][j]);
            }
        }
    }
}

int attn_prep(const AttnPrep& a, int rows, int n_lanes, bool early, cudaStream_t st) {
    if ((long long) rows * (a.nq + 2 * a.nkv) > PREP_MANY && rows > FNX_MAX_ROWS && !a.lane_seq && !a.depth && a.hd == 256 && a.nrot == 64) {
        FNX_CUDA_OK(launch_after(k_attn_prep_rows, dim3(a.nq + 2 * a.nkv, (rows + PREP_ROWS * PREP_WARPS - 1) / (PREP_ROWS * PREP_WARPS)), dim3(PREP_WARPS * 32), 0, st, a, rows));
        FNX_LAUNCH_OK("k_attn_prep_rows");
        return FNX_OK;
    }
    const cudaError_t le = launch_dep(true, early ? k_attn_prep_append<true> : k_attn_prep_append<false>, dim3(a.nq + 2 * a.nkv, rows, n_lanes), dim3(a.hd), a.hd * sizeof(float), st, a);
    return le == cudaSuccess ? FNX_OK : fail(FNX_E_CUDA, "k_attn_prep_append: launch failed: %s", cudaGetErrorString(le));
}

// grid (KV heads, groups of ATT_ROWS rows); a block runs over all the positions its rows see, so there is one partial per (row, head), which
// k_attn_gate normalises and gates
__global__ void __launch_bounds__(ATT_THREADS) k_attn_part_prompt(const float* __restrict__ qg, int ldq, const __half* __restrict__ kc,
                                                                  const __half* __restrict__ vc, float* __restrict__ acc_out,
                                                                  AttPartial* __restrict__ mz_out, int T, int nq, int nkv, const int* __restrict__ pos0p) {
    extern __shared__ __align__(16) uint8_t smem[];
    attn_prompt_body(qg, ldq, kc, vc, acc_out, mz_out, T, nq, nkv, *pos0p, (int) blockIdx.x, (int) blockIdx.y * ATT_ROWS, (int) threadIdx.x, smem);
}

// grid (heads, rows).  Bound by its bytes.  500 rows of 16 heads, with the kernel before it: 66 us; 172 with the windows' merge of many partials in its
// place, whose block of 1,024 threads has one to read here.
__global__ void __launch_bounds__(ATT_HD) k_attn_gate(const float* __restrict__ acc, const AttPartial* __restrict__ mz, const float* __restrict__ qg, int ldq,
                                                      float* __restrict__ out, int nq) {
    pdl_begin();
    const int h = blockIdx.x, t = blockIdx.y, i = threadIdx.x;
    const size_t slot = (size_t) t * nq + h;
    out[slot * ATT_HD + i] = acc[slot * ATT_HD + i] / mz[slot].z * sigmoidf_(qg[(size_t) t * ldq + (size_t) h * 2 * ATT_HD + ATT_HD + i]);
}

}  // namespace fnxb

using namespace fnxb;

extern "C" int fnx_attn_prep_append(float* qg, int ldq, float* k, int ldk, const float* v, int ldv, const float* q_norm, const float* k_norm,
                                    void* kc, void* vc, int T, int nq, int nkv, int hd, int nrot, const int* pos0, const int* depth, float eps,
                                    float rope_base, fnx_stream st) {
    FNX_REQUIRE(qg && k && v && q_norm && k_norm && kc && vc && pos0, "fnx_attn_prep_append: null pointer");
    FNX_REQUIRE(T >= 1 && (depth ? T <= FNX_MAX_ROWS : T <= 65535), "fnx_attn_prep_append: %d rows", T);
    FNX_REQUIRE(hd % 32 == 0 && hd <= 1024 && nrot <= hd && nrot % 2 == 0, "fnx_attn_prep_append: head dim %d, rotary %d", hd, nrot);
    return attn_prep(AttnPrep{qg, ldq, k, ldk, v, ldv, q_norm, k_norm, (__half*) kc, (__half*) vc, 0, nq, nkv, hd, nrot, pos0, depth, nullptr, nullptr, eps, rope_base}, T, 1,
                     false, as_stream(st));
}

extern "C" size_t fnx_attn_scratch_bytes(int T, int nq, int hd) {
    const size_t S = (size_t) sm_count();   // an upper bound of the splits for any KV-head count
    return (size_t) T * nq * S * ((size_t) hd * sizeof(float) + sizeof(AttPartial)) + 16;   // (room to align)
}

extern "C" int fnx_attn(const float* qg, int ldq, const void* kc, const void* vc, float* out, int T, int nq, int nkv, int hd, const int* pos0,
                        const int* parent, void* scratch, fnx_stream st) {
    FNX_REQUIRE(qg && kc && vc && out && pos0 && scratch, "fnx_attn: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS, "fnx_attn: %d rows", T);
    FNX_REQUIRE(hd == ATT_THREADS, "fnx_attn: head dim %d (this build: %d)", hd, ATT_THREADS);
    FNX_REQUIRE(nkv >= 1 && nq % nkv == 0 && nq / nkv <= ATT_MAXQ, "fnx_attn: %d q heads over %d KV heads", nq, nkv);
    return attn_window(AttnWin{qg, ldq, (const __half*) kc, (const __half*) vc, 0, T, nq, nkv, hd, pos0, parent, nullptr, nullptr, 0, nullptr}, scratch, out, nullptr, false,
                       as_stream(st));
}

extern "C" size_t fnx_attn_prompt_scratch_bytes(int T, int nq, int hd) { return (size_t) T * nq * ((size_t) hd * sizeof(float) + sizeof(AttPartial)); }

namespace fnxb {
bool attn_prompt_tc_fits(int nq, int nkv, int hd);
int attn_prompt_tc_launch(const float* qg, int ldq, const __half* kc, const __half* vc, float* out, int T, int nq, int nkv, const int* pos0, unsigned* err,
                          cudaStream_t st);
}  // namespace fnxb

extern "C" int fnx_attn_prompt(const float* qg, int ldq, const void* kc, const void* vc, float* out, int T, int nq, int nkv, int hd, const int* pos0,
                               void* scratch, unsigned* err, int use_mma_sync, fnx_stream st) {
    FNX_REQUIRE(qg && kc && vc && out && pos0 && scratch, "fnx_attn_prompt: null pointer");
    FNX_REQUIRE(T >= 1 && T <= 65535, "fnx_attn_prompt: %d rows", T);
    FNX_REQUIRE(hd == ATT_THREADS, "fnx_attn_prompt: head dim %d (this build: %d)", hd, ATT_THREADS);
    FNX_REQUIRE(nkv >= 1 && nq % nkv == 0 && nq / nkv <= ATT_MAXQ, "fnx_attn_prompt: %d q heads over %d KV heads", nq, nkv);
    if (!use_mma_sync && attn_prompt_tc_fits(nq, nkv, hd)) {
        FNX_REQUIRE(ldq % 4 == 0 && ((uintptr_t) qg & 15) == 0 && ((uintptr_t) kc & 15) == 0 && ((uintptr_t) vc & 15) == 0 && ((uintptr_t) out & 15) == 0,
                    "fnx_attn_prompt: rows and caches must be 16-byte aligned");
        return attn_prompt_tc_launch(qg, ldq, (const __half*) kc, (const __half*) vc, out, T, nq, nkv, pos0, err, as_stream(st));
    }
    float* acc = (float*) scratch;
    AttPartial* mz = (AttPartial*) (acc + (size_t) T * nq * hd);
    if (int rc = set_smem_limit((const void*) k_attn_part_prompt, (int) attn_prompt_smem())) return rc;
    k_attn_part_prompt<<<dim3(nkv, (T + ATT_ROWS - 1) / ATT_ROWS), ATT_THREADS, attn_prompt_smem(), as_stream(st)>>>(qg, ldq, (const __half*) kc, (const __half*) vc, acc, mz,
                                                                                                                     T, nq, nkv, pos0);
    FNX_LAUNCH_OK("fnx_attn_prompt (partials)");
    FNX_CUDA_OK(launch_after(k_attn_gate, dim3(nq, T), dim3(ATT_HD), 0, as_stream(st), acc, mz, qg, ldq, out, nq));
    FNX_LAUNCH_OK("fnx_attn_prompt (gate)");
    return FNX_OK;
}

// ---- allocation-free variant: the split partials live in a file-scope device array -------------------------------------------------

namespace fnxb {

constexpr int ATT_STATIC_SLOTS = FNX_ATTN_STATIC_MAX_SLOTS;   // (row, head, split) partials
constexpr int ATT_STATIC_HD = ATT_THREADS;
constexpr size_t ATT_STATIC_BYTES = (size_t) ATT_STATIC_SLOTS * (ATT_STATIC_HD * sizeof(float) + sizeof(AttPartial));
static __device__ __align__(256) unsigned char g_attn_static_scratch[ATT_STATIC_BYTES];

constexpr int ATT_STATIC_MAX_DEV = 64;
static void* g_attn_static_ptr[ATT_STATIC_MAX_DEV];   // per device: the array's address, resolved once

static int attn_static_resolve(void** out) {
    int dev = -1;
    FNX_CUDA_OK(cudaGetDevice(&dev));
    FNX_REQUIRE(dev >= 0 && dev < ATT_STATIC_MAX_DEV, "fnx_attn_static: device %d", dev);
    if (!g_attn_static_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t rc = cudaGetSymbolAddress((void**) &p, g_attn_static_scratch);
        if (rc != cudaSuccess || !p) return fail(FNX_E_CUDA, "fnx_attn_static: cudaGetSymbolAddress: %s", cudaGetErrorString(rc));
        FNX_TRY(attn_window_setup());
        g_attn_static_ptr[dev] = p;
    }
    *out = g_attn_static_ptr[dev];
    return FNX_OK;
}

}  // namespace fnxb

extern "C" int fnx_attn_static_setup(void) {
    void* p = nullptr;
    return attn_static_resolve(&p);
}

extern "C" int fnx_attn_static(const float* qg, int ldq, const void* kc, const void* vc, float* out, int T, int nq, int nkv, int hd, const int* pos0,
                               const int* parent, fnx_stream st) {
    FNX_REQUIRE(qg && kc && vc && out && pos0, "fnx_attn_static: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS, "fnx_attn_static: %d rows", T);
    FNX_REQUIRE(hd == ATT_THREADS, "fnx_attn_static: head dim %d (this build: %d)", hd, ATT_THREADS);
    FNX_REQUIRE(nkv >= 1 && nq % nkv == 0 && nq / nkv <= ATT_MAXQ, "fnx_attn_static: %d q heads over %d KV heads", nq, nkv);
    const int S = sm_count() / nkv < 1 ? 1 : sm_count() / nkv;
    const long long slots = (long long) T * nq * S;
    FNX_REQUIRE(slots <= ATT_STATIC_SLOTS,
                "fnx_attn_static: %d rows x %d heads x %d splits = %lld partials exceed the built-in scratch of %d; use fnx_attn with caller scratch",
                T, nq, S, slots, ATT_STATIC_SLOTS);
    void* scratch = nullptr;
    if (const int rc = attn_static_resolve(&scratch)) return rc;
    return attn_window(AttnWin{qg, ldq, (const __half*) kc, (const __half*) vc, 0, T, nq, nkv, hd, pos0, parent, nullptr, nullptr, 0, nullptr}, scratch, out, nullptr, false,
                       as_stream(st));
}

// ---- batched lanes (see k_attn_prep_append)
extern "C" int fnx_attn_prep_append_lanes(float* qg, int ldq, float* k, int ldk, const float* v, int ldv, const float* q_norm, const float* k_norm,
                                          void* kc_base, void* vc_base, size_t seq_stride_rows, int n_lanes, int max_lane_rows, int nq, int nkv, int hd,
                                          int nrot, const int* pos, const int* lane_seq, const int* lane_row0, float eps, float rope_base, fnx_stream st) {
    FNX_REQUIRE(qg && k && v && q_norm && k_norm && kc_base && vc_base && pos && lane_seq && lane_row0, "fnx_attn_prep_append_lanes: null pointer");
    FNX_REQUIRE(n_lanes >= 1 && n_lanes <= FNX_MAX_ROWS && max_lane_rows >= 1 && max_lane_rows <= FNX_MAX_ROWS, "fnx_attn_prep_append_lanes: %d lanes of up to %d rows",
                n_lanes, max_lane_rows);
    FNX_REQUIRE(hd % 32 == 0 && hd <= 1024 && nrot <= hd && nrot % 2 == 0, "fnx_attn_prep_append_lanes: head dim %d, rotary %d", hd, nrot);
    return attn_prep(AttnPrep{qg, ldq, k, ldk, v, ldv, q_norm, k_norm, (__half*) kc_base, (__half*) vc_base, seq_stride_rows, nq, nkv, hd, nrot, pos, nullptr, lane_seq,
                              lane_row0, eps, rope_base},
                     max_lane_rows, n_lanes, false, as_stream(st));
}

extern "C" int fnx_attn_lanes(const float* qg, int ldq, const void* kc_base, const void* vc_base, size_t seq_stride_rows, float* out, int T, int n_lanes,
                              int nq, int nkv, int hd, const int* pos, const int* lane_seq, const int* lane_row0, void* scratch, fnx_stream st) {
    FNX_REQUIRE(qg && kc_base && vc_base && out && pos && lane_seq && lane_row0 && scratch, "fnx_attn_lanes: null pointer");
    FNX_REQUIRE(T >= 1 && T <= FNX_MAX_ROWS && n_lanes >= 1 && n_lanes <= T, "fnx_attn_lanes: %d rows in %d lanes", T, n_lanes);
    FNX_REQUIRE(hd == ATT_THREADS, "fnx_attn_lanes: head dim %d (this build: %d)", hd, ATT_THREADS);
    FNX_REQUIRE(nkv >= 1 && nq % nkv == 0 && nq / nkv <= ATT_MAXQ, "fnx_attn_lanes: %d q heads over %d KV heads", nq, nkv);
    return attn_window(AttnWin{qg, ldq, (const __half*) kc_base, (const __half*) vc_base, seq_stride_rows, T, nq, nkv, hd, pos, nullptr, lane_seq, lane_row0, n_lanes, nullptr},
                       scratch, out, nullptr, false, as_stream(st));
}
