// Attention of a decode window (attn_win.cu): one sequence's rows, a chain or a tree, or the rows of several sequences' lanes.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace fnxb {

struct AttPartial;   // attn_core.cuh

struct AttnWin {
    const float* qg;        // [T][ldq]: nq heads of (q 256 | gate 256)
    int ldq;
    const __half* kc;       // caches [rows][nkv][256]; lanes: sequence s at row s * seq_rows
    const __half* vc;
    size_t seq_rows;
    int T, nq, nkv, hd;     // hd: 256
    const int* pos;         // one sequence: its position; lanes: every sequence's
    const int* parent;      // one sequence: the rows' parents (null: a chain)
    const int* lane_seq;    // lanes: their sequences (negative: skipped) and first rows [n_lanes + 1]; null: one sequence
    const int* lane_row0;
    int n_lanes;
    unsigned* err;          // FNX_ERR_TIMEOUT (may be null: the output rows are NaN then)
};

// The prep of the rows: per-head norm, rotary, the caches' new rows.
struct AttnPrep {
    float* qg;
    int ldq;
    float* k;
    int ldk;
    const float* v;
    int ldv;
    const float* qn;
    const float* kn;
    __half* kc;
    __half* vc;
    size_t seq_rows;        // lanes
    int nq, nkv, hd, nrot;
    const int* pos;         // as above
    const int* depth;       // one sequence: the rows' depths (null: a chain)
    const int* lane_seq;
    const int* lane_row0;
    float eps, rope_base;
};
// rows: the window's, or the longest lane's.  early: launch_dep's (positions and lane tables are read ahead)
int attn_prep(const AttnPrep& a, int rows, int n_lanes, bool early, cudaStream_t st);

// out [T][nq][256], or with img their image (nat_image.cuh: the row's block h is head h).  scratch: fnx_attn_scratch_bytes().
// early: launch_dep's; everything but the window's own rows is read ahead
int attn_window(const AttnWin& a, void* scratch, float* out, uint8_t* img, bool early, cudaStream_t st);
// the kernels' limits and the driver's entry point, resolved outside any capture
int attn_window_setup();

}  // namespace fnxb
