// Prompt products from the engine's own weight layout (prompt_nat.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace fnxb {

// Activations of these products are f16 rows whose columns lie, within every 32, in the order that the weight words decode in: lane q of a
// fragment row holds the columns 8 q .. 8 q + 7, column 8 q + j at slot 16 (j / 4) + 2 q + {0, 8, 1, 9}[j % 4].
__host__ __device__ __forceinline__ int pn_slot(int c) {
    const int j = c & 7, q = (c >> 3) & 3, k = j & 3;
    return (c & ~31) + 16 * (j >> 2) + 2 * q + ((k & 1) << 3 | k >> 1);
}

constexpr int PN_N = 64;       // rows per job at most

struct PnJob {
    int w, n, start;           // expert (E: the shared one), rows, first entry of `order`
};

struct PnParams {
    const uint8_t* W;          // expert matrices [e_base ..) (dense: one matrix)
    size_t stride;
    int e_base, E;
    const uint8_t* Wsh;        // job.w >= E
    const PnJob* jobs;         // (dense: the T rows in order)
    const int* njobs;
    const int* order;          // per entry the pair t Kp + k; shared expert: TKp + t
    int T, TKp, Kp, per;       // per: the jobs' rows at most (dense: exactly, but for the last)
    const __half* x;           // gate|up, dense: [token][K]; down: [pair][K]
    int rows, K;               // features (gate|up: F), inner dimension
    float* out;                // down: [pair][rows]; dense: [token][ldo]
    __half* outh;              // gate|up: [pair][F], in slot order
    int ldo, accumulate;
    unsigned* err;
};

// mode 1: outh = silu(x Wg^T) (x Wu^T); mode 0: out = x W^T over the jobs' pairs; mode 2: out (+)= x W^T over T rows.  max_jobs: as many
// as there can be
int prompt_nat(int mode, const PnParams& p, int max_jobs, cudaStream_t st);
// xh[t] = f16(x[t] norm_w / rms(x[t])) in slot order, or in prompt_few's (norm_w null: f16(x[t]))
int prompt_nat_rows(const float* x, const float* norm_w, int T, int H, float eps, __half* xh, bool few, cudaStream_t st);
// modes 1 and 0 for jobs of up to PROMPT_FEW_ROWS rows
constexpr int PROMPT_FEW_ROWS = 8;
int prompt_few(int mode, const PnParams& p, int max_jobs, cudaStream_t st);
// where those are taken: up to four rows an expert.  A layer's experts by these and by prompt_nat's jobs of 64, us, 512 experts: ten picks a row, 100 rows 194 and
// 201, 150 rows 222 and 224, 180 rows 233 and 233, 204 rows (the line) 257 and 243, 333 rows 319 and 261; four picks, 204 rows 180 and 185, 256 rows 199 and
// 200, 333 rows 220 and 212, 512 rows (the line) 265 and 241.  So they win up to some two and a half to three rows an expert; the line lies where it did for
// the form of prompt_nat with four stages of rows, which came level at four
inline bool prompt_few_fits(long long pairs, int E) { return pairs <= 4ll * E; }
// the rows of a dense product's jobs: fewer, in sixteens, as long as the items of `slabs` x the jobs all run at once (2,048 x 4,096, 332 rows: 30 us with
// jobs of 64 on 48 SMs, 28 with jobs of 32 on 88; where they would not, 34 us become 52)
inline int prompt_dense_rows(int T, long long slabs, int sms) {
    int per = PN_N;
    while (per > 16 && slabs * ((T + per - 17) / (per - 16)) <= sms) per -= 16;
    return per;
}

}  // namespace fnxb
