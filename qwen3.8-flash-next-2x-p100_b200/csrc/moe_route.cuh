// Routing pieces of the router kernels (moe_route.cu), the window form and the prompt form:
// order-preserving logit keys, the top-K of one row by one warp, and the block-wide job list builder.
// Semantics: k_topk + k_jobs (engine/src/kernels.cu:338-398) and k_router_route (engine/src/moe.cuh:382-411).
#pragma once

#include "fnx_common.cuh"

namespace fnxb {

constexpr int RT_MAXE = 1024;

// float -> unsigned key with the same order (so that warp-wide integer maxima rank logits)
__device__ __forceinline__ unsigned rt_key(float v) {
    const unsigned u = __float_as_uint(v);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}

// Top K <= 32 of one row's E logits by one warp: (largest value, lowest index) first.  SL = slots per lane (index lane + 32 j).
// The K-th largest of the lanes' own maxima bounds the K-th largest logit from below, so the logits at or above it (a dozen at
// K = 10) hold the top K: they are collected in shared memory (scr: 64 words of the warp's) and each finds its place by counting the
// larger ones.  (K rounds of a warp maximum took 3.6 us, this 0.7.)  More than 32 of them (many equal logits): K rounds.
// topi_g / topw_g (global) may be null; topi_s / topw_s (shared) may be null.
template <int SL>
__device__ __forceinline__ void rt_topk_row(const float* l, int E, int K, int lane, unsigned* scr, int* topi_g, int* topi_s, float* topw_g, float* topw_s) {
    unsigned key[SL];
#pragma unroll
    for (int j = 0; j < SL; ++j) key[j] = lane + 32 * j < E ? rt_key(__ldcg(l + lane + 32 * j)) : 0u;
    unsigned mx = key[0];
#pragma unroll
    for (int j = 1; j < SL; ++j) mx = max(mx, key[j]);
    // (through shared memory, a few instructions in a loop: the block runs this code once, and fetching it is part of its time)
    scr[lane] = mx;
    __syncwarp();
    int rank = 0;
#pragma unroll 1
    for (int o = 0; o < 32; o += 4) {
        const uint4 m = *reinterpret_cast<const uint4*>(scr + o);
        rank += (m.x > mx || (m.x == mx && o < lane)) + (m.y > mx || (m.y == mx && o + 1 < lane)) + (m.z > mx || (m.z == mx && o + 2 < lane)) +
                (m.w > mx || (m.w == mx && o + 3 < lane));
    }
    __syncwarp();
    const unsigned low = __shfl_sync(0xffffffffu, mx, __ffs(__ballot_sync(0xffffffffu, rank == K - 1)) - 1);
    int n = 0;
#pragma unroll
    for (int j = 0; j < SL; ++j) {
        const bool in = key[j] >= low && key[j] != 0u;
        const unsigned who = __ballot_sync(0xffffffffu, in);
        const int at = n + __popc(who & ((1u << lane) - 1u));
        if (in && at < 32) {
            scr[at] = key[j];
            scr[32 + at] = (unsigned) (lane + 32 * j);
        }
        n += __popc(who);
    }
    __syncwarp();
    unsigned mine = 0u;   // the pick of place `lane`
    int my_i = 0;
    if (n <= 32) {
        const unsigned k = lane < n ? scr[lane] : 0u, ix = lane < n ? scr[32 + lane] : 0xffffffffu;
        int place = 0;
        if (lane >= n) scr[lane] = 0u;
        __syncwarp();
#pragma unroll 1
        for (int i = 0; i < n; i += 4) {
            const uint4 a = *reinterpret_cast<const uint4*>(scr + i), b = *reinterpret_cast<const uint4*>(scr + 32 + i);
            place += (a.x > k || (a.x == k && b.x < ix)) + (a.y > k || (a.y == k && b.y < ix)) + (a.z > k || (a.z == k && b.z < ix)) + (a.w > k || (a.w == k && b.w < ix));
        }
        __syncwarp();
        if (lane < n && place < K) {
            scr[place] = k;
            scr[32 + place] = ix;
        }
        __syncwarp();
        if (lane < K) {
            mine = scr[lane];
            my_i = (int) scr[32 + lane];
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            unsigned bk = 0u;
            int bj = 0;
#pragma unroll
            for (int j = 0; j < SL; ++j)   // among equals the lower slot
                if (key[j] > bk) {
                    bk = key[j];
                    bj = j;
                }
            const unsigned wk = __reduce_max_sync(0xffffffffu, bk);
            const int bi = __reduce_min_sync(0xffffffffu, bk == wk ? lane + 32 * bj : 0x7fffffff);
            if (lane == k) {
                mine = wk;
                my_i = bi;
            }
#pragma unroll
            for (int j = 0; j < SL; ++j)
                if (lane + 32 * j == bi) key[j] = 0u;
        }
    }
    __syncwarp();
    const float v = __uint_as_float(mine & 0x80000000u ? mine & 0x7fffffffu : ~mine), top = __shfl_sync(0xffffffffu, v, 0);
    const float w = lane < K ? expf(v - top) : 0.f;
    float z = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; ++k) z += __shfl_sync(0xffffffffu, w, k);   // in pick order
    if (lane < K) {
        if (topi_g) topi_g[lane] = my_i;
        if (topi_s) topi_s[lane] = my_i;
        if (topw_g) topw_g[lane] = w / z;
        if (topw_s) topw_s[lane] = w / z;
    }
}

// Shared memory of the job list builder: s_topi [T][K] (filled by the caller), s_rows and s_base [RT_MAXE], wsum [32],
// total [2], js = the job list (room for T K + ceil(T / 4) jobs).
struct RtJobSmem {
    int* s_topi;
    unsigned* s_rows;
    int* s_base;
    int* wsum;
    int* total;
    fnx_job* js;
};

// The job list of T <= 32 rows' picks, by all NTH threads of the block (every thread calls; the function synchronises the
// block): jobs in ascending expert order, expert e's rows in row order, 4 per job; then (add_shared) the shared expert's.
// A row picks an expert at most once, so the rows of an expert are a bit mask: its population is their number, and the bits below a
// row's are that row's place among them.
// rt_clear_jobs comes first (nothing of it depends on the picks); then, behind a barrier, each row's warp leaves its picks (rt_note_picks); rt_build_jobs does the rest.
// Thread `tid` owns experts [tid * EPT, (tid + 1) * EPT) below RT_MAXE: a block-wide exclusive scan of their job counts gives each
// expert's first job; then one thread per (row, pick) entry places itself.  The number of jobs in total[0], the routed ones in
// total[1] (valid after the call in every thread).
template <int NTH>
__device__ __forceinline__ void rt_clear_jobs(const RtJobSmem& s, int tid, int T, int K) {
    for (int e = tid; e < RT_MAXE; e += NTH) s.s_rows[e] = 0u;
    // unused row slots of the jobs stay zero
    const int cap = (T * K + (T + FNX_JOB_TOK - 1) / FNX_JOB_TOK) * (int) (sizeof(fnx_job) / 4);
    for (int w = tid; w < cap; w += NTH) reinterpret_cast<int*>(s.js)[w] = 0;
}
// row t's warp, its picks in s_topi
__device__ __forceinline__ void rt_note_picks(const RtJobSmem& s, int t, int K, int e_lo, int e_hi, int lane) {
    __syncwarp();
    if (lane < K) {
        const int e = s.s_topi[t * K + lane];
        if (e >= e_lo && e < e_hi) atomicOr(&s.s_rows[e], 1u << t);
    }
}
template <int NTH>
__device__ __forceinline__ void rt_build_jobs(const RtJobSmem& s, int tid, int T, int E, int K, int e_lo, int e_hi, int add_shared) {
    constexpr int EPT = (RT_MAXE + NTH - 1) / NTH;
    const int warp = tid >> 5, lane = tid & 31;
    __syncthreads();
    int cnt_[EPT], mine = 0;
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
        const int e = tid * EPT + j;
        cnt_[j] = e < RT_MAXE ? (__popc(s.s_rows[e]) + FNX_JOB_TOK - 1) / FNX_JOB_TOK : 0;
        mine += cnt_[j];
    }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s.wsum[warp] = incl;
    __syncthreads();
    int base_ = incl - mine;
    for (int w = 0; w < warp; ++w) base_ += s.wsum[w];
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
        if (cnt_[j]) s.s_base[tid * EPT + j] = base_;
        base_ += cnt_[j];
    }
    if (tid == NTH - 1) {
        s.total[1] = base_;
        s.total[0] = base_ + (add_shared ? (T + FNX_JOB_TOK - 1) / FNX_JOB_TOK : 0);
    }
    __syncthreads();
    const int routed_total = s.total[1];
    for (int t = warp; t < T; t += NTH / 32) {
        const int i = t * K + lane, e = lane < K ? s.s_topi[i] : -1;
        if (e < e_lo || e >= e_hi) continue;
        const unsigned rows = s.s_rows[e];
        const int rank = __popc(rows & ((1u << t) - 1u));
        fnx_job& jj = s.js[s.s_base[e] + rank / FNX_JOB_TOK];
        jj.y[rank % FNX_JOB_TOK] = t;
        jj.out[rank % FNX_JOB_TOK] = i;
        if (rank % FNX_JOB_TOK == 0) {
            jj.w = e;
            jj.n = min(FNX_JOB_TOK, __popc(rows) - rank);
        }
    }
    if (add_shared)
        for (int t = tid; t < T; t += NTH) {
            fnx_job& j = s.js[routed_total + t / FNX_JOB_TOK];
            j.y[t % FNX_JOB_TOK] = t;
            j.out[t % FNX_JOB_TOK] = T * K + t;
            if (t % FNX_JOB_TOK == 0) {
                j.w = E;
                j.n = min(FNX_JOB_TOK, T - t);
            }
        }
    __syncthreads();
}

}  // namespace fnxb
