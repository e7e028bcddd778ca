// The DeltaNet core of a window as the engine calls it (gdn.cu).
#pragma once

#include "fnx_common.cuh"

namespace fnxb {

// what a window's DeltaNet kernel reads and writes (one sequence's rows)
struct GdnArgs {
    const float* qkvz;
    int stride;
    const float* ab;
    int ldab;
    float* hist_pool;
    const float *convw, *dt, *a, *nw;
    float* S_pool;
    int NS;
    const int* parent;
    float* y;
    uint8_t* img;      // the output rows' image (nat_image.cuh), or null
    int nk, nv, T;
    float eps;
};

int gdn_window(const GdnArgs& p, const int* cur, bool early, cudaStream_t st);
// rows: of all the lanes
int gdn_window_lanes(const GdnArgs& p, size_t hist_seq_stride, size_t s_seq_stride, const int* cur, const int* lane_seq, const int* lane_row0, int n_lanes, int max_rows,
                     int rows, bool early, cudaStream_t st);

}  // namespace fnxb
