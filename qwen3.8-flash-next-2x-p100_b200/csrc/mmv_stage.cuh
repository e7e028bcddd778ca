// One matrix stage of a block: the body of the IQ3_S matrix x rows kernel (iq3s_mmv.cu).  The block quantises the
// activation rows it needs into its own shared-memory images (or copies the image their producer left), streams its share of the tile blocks
// through the warps' rings, combines the pieces of tiles cut by warp shares, and writes the results.
//
// The product is a sequence of ITEMS: one 16-row x 256-column tile block against the activation cells.  A unit is a 16-row tile across all of K
// (gate|up: the gate tile, then its up tile): nbu consecutive items.  A block's items are dealt to its warps in equal contiguous shares, so every
// warp has the same decode work whatever the number of units.  Each warp streams its items through its PRIVATE ring of bulk async copies and
// accumulates in registers.  A unit that lies wholly inside one warp's share is finished and written by that warp; a unit cut by share boundaries
// leaves its pieces in shared memory, and after ONE block barrier the warp that holds its first piece adds the others in warp order and writes it.
//
// A warp has two or three items of a 12,352 x 2,048 product (some 350 instructions each), so what surrounds them counts as much: divisions are shifts
// or multiplications by inverses that the host made (mmv_inverse), the ring's first copies leave from as many lanes, a row's 1 / rms is worked out
// once a warp, and image rows that hold nothing stay whatever they are (their sums are dropped).  Up to three blocks of rows a warp are quantised
// together, their loads on the way before the block's first barrier.  Twelve such products of five rows: 157 us with divisions, a lane that issued
// alone and rows quantised two by two (3,100 instructions a warp, 900 of them items'), 110 now; one MoE block of five rows, its combine's shorter way included, in a
// graph 52.4 and 48.4.
#pragma once

#include <type_traits>

#include "mmv_core.cuh"

namespace fnxb {

constexpr int MMV_THREADS = 512, MMV_WARPS = 16;

struct MmvParams {
    const uint8_t* W;
    size_t expert_stride;
    int e_base;
    const uint8_t* Wsh;
    int E;
    const fnx_job* jobs;
    const int* njobs;
    int njobs_max;
    int T;
    const float* x;
    int ldx;
    const float* norm_w;
    float eps;
    float* out;
    int ldo;
    int rows;   // output rows per job (gate|up: F)
    int K;
    int accumulate;
    int R;      // ring slots per warp
    unsigned upj_inv, nblk_inv;   // mmv_inverse() of the units a job has, of the blocks
    unsigned share, rest;         // dense: units a block, units left over
    unsigned* err;
    // dense: the rows' image, already built (stage_image_bytes() bytes in the layout of the block's own image): the
    // block copies it instead of quantising x
    const uint8_t* ximg;
};

// bytes of a dense image of NG row groups over K columns: cells, scales, block sums of squares (the order the block
// holds them in)
__host__ __device__ inline size_t stage_image_bytes(int NG, int K) {
    return (size_t) NG * ((size_t) (K / 32) * 32 * 8 + (size_t) (K / 256) * 8 * 4 + 4 * 16 * 4);
}

// jobs whose activation images a block holds at once: its range of units spans at most two jobs of gate|up and a
// few of down; anything wider is walked in passes
template <int MODE>
__host__ __device__ constexpr int mmv_jmax() { return MODE == MAT_DENSE ? 1 : MODE == MAT_GATEUP ? 2 : 4; }

// a piece of a unit: slot [warp][0] = one that continues a unit begun by an earlier warp, slot [warp][1] = the first piece of a unit that later
// warps continue
template <int NG, int MODE>
struct MmvPiece {
    static constexpr int KINDS = MODE == MAT_GATEUP ? 2 : 1;   // (gate, up)
    int unit;                // -1: none
    int pad[3];
    typename MatAcc<MODE>::type v[KINDS * NG * 64];   // [kind][group][16 lanes][4]
};

template <int NG, int MODE>
__host__ __device__ inline size_t mmv_image_bytes(int K) {
    return (size_t) mmv_jmax<MODE>() * NG * ((size_t) (K / 32) * 32 * 8 + (size_t) (K / 256) * 8 * 4);
}
template <int NG, int MODE>
__host__ __device__ inline size_t mmv_smem_bytes(int K, int R, int njobs_max) {
    constexpr int rows = mmv_jmax<MODE>() * 4 * NG;
    return (size_t) CORE_TABLE_BYTES + (size_t) MMV_WARPS * R * (TILE_BYTES + 8) + mmv_image_bytes<NG, MODE>(K) + rows * 16 * sizeof(float) +
           (size_t) MMV_WARPS * 2 * sizeof(MmvPiece<NG, MODE>) + (MODE == MAT_DENSE ? 0 : (size_t) njobs_max * sizeof(fnx_job)) + 64;
}

constexpr int MMV_JOB_WORDS = sizeof(fnx_job) / 4, MMV_JOB_REGS = 3;   // job-list words a thread holds across the set-up

// the block's shared memory for a stage (carved by the caller; the table is filled and the barriers initialised)
struct StageSmem {
    uint32_t table_s;       // the replicated codebook
    uint8_t* slots;         // MMV_WARPS x R tile-block slots
    uint64_t* bars;         // MMV_WARPS x R mbarriers
    uint2* cells;           // images: jmax x NG x (K / 32) x 32 cells, then their scales and chunk sums
    float* scales;
    float* rs;
    void* pieces;           // MMV_WARPS x 2 MmvPiece of the stage's row groups and mode
    fnx_job* jobs_s;        // njobs_max jobs (expert modes)
};

// what a thread holds from stage_begin() to stage_run(): loads in flight
struct StageRegs {
    int njobs;
    int jw[MMV_JOB_REGS];
    float v[QUANT_BATCH][8];
    float w[QUANT_BATCH][8];   // their norm weights
};

// dense stage: task id -> (row id % T, block id / T), id < T K / 256 <= 192
__device__ __forceinline__ QuantTask stage_dense_task(const MmvParams& p, int id) {
    QuantTask q;
    q.blk = (id * (65536 / p.T + 1)) >> 16;
    q.t = id - q.blk * p.T;
    q.src = p.x + (size_t) q.t * p.ldx + q.blk * 256;
    return q;
}

// Starts the loads whose latency the caller may hide behind other work: the job list (expert modes) or the warp's
// first rows to quantise (dense).
template <int NG, int MODE>
__device__ __forceinline__ void stage_begin(const MmvParams& p, StageRegs& h, int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    h.njobs = 1;
    if constexpr (MODE != MAT_DENSE) {
        const int nword = p.njobs_max * MMV_JOB_WORDS;
        h.njobs = *p.njobs;
#pragma unroll
        for (int i = 0; i < MMV_JOB_REGS; ++i) {
            const int w = tid + i * MMV_THREADS;
            h.jw[i] = w < nword ? reinterpret_cast<const int*>(p.jobs)[w] : 0;
        }
    } else if (p.ximg) {
        // the image's first 16-byte words ride in the registers the rows would have used
        static_assert(QUANT_BATCH >= 2, "eight 16-byte words per thread");
        const int n16 = (int) (stage_image_bytes(NG, p.K) / 16);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = tid + j * MMV_THREADS;
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < n16) t = __ldcg(reinterpret_cast<const float4*>(p.ximg) + i);
            float* d = j < 4 ? &h.v[j >> 1][(j & 1) * 4] : &h.w[(j - 4) >> 1][(j & 1) * 4];
            d[0] = t.x; d[1] = t.y; d[2] = t.z; d[3] = t.w;
        }
    } else {
        const int ntask = p.T * (p.K / 256);
#pragma unroll
        for (int j = 0; j < QUANT_BATCH; ++j)
            if (warp + j * MMV_WARPS < ntask) quant_fetch(stage_dense_task(p, warp + j * MMV_WARPS), p.norm_w, lane, h.v[j], h.w[j]);
    }
}

// the 16 x rows results of a unit (local tile lu) from this lane's sums (threads q < 2 hold them); orow: the job's output rows (dense: the row itself)
template <int NG, int MODE, typename AccT>
__device__ __forceinline__ void stage_write(const MmvParams& p, int lu, const int* orow, int ntok, int lane, const AccT (&gacc)[NG][4], const AccT (&acc)[NG][4]) {
    const int g = lane >> 2, q = lane & 3;
    if (q >= 2) return;
    float* dst[NG][2];
    float old[NG][4];
#pragma unroll
    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int tok = 4 * ng + 2 * q + (k & 1);
            old[ng][k] = 0.f;
            if (k < 2) dst[ng][k] = p.out + (size_t) (MODE == MAT_DENSE ? tok : tok < ntok ? orow[tok] : 0) * p.ldo + lu * 16 + g;
            if (MODE == MAT_DENSE && p.accumulate && tok < ntok) old[ng][k] = dst[ng][k & 1][8 * (k >> 1)];
        }
#pragma unroll
    for (int ng = 0; ng < NG; ++ng)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float v = MODE == MAT_GATEUP ? siluf_((float) gacc[ng][k]) * (float) acc[ng][k] : (float) acc[ng][k];
            if (4 * ng + 2 * q + (k & 1) < ntok) dst[ng][k & 1][8 * (k >> 1)] = MODE == MAT_DENSE && p.accumulate ? old[ng][k] + v : v;
        }
}

// The stage proper: `bid` of `nblk` blocks share the matrix.  Ends with every result of the block written (no trailing barrier).
// stamp(): a tracing hook called at the phase boundaries.
template <int NG, int MODE, typename Stamp>
__device__ __forceinline__ void stage_run(const MmvParams& p, const StageSmem& S, StageRegs& h, int tid, int bid, int nblk, Stamp&& stamp) {
    using AccT = typename MatAcc<MODE>::type;
    using Piece = MmvPiece<NG, MODE>;
    constexpr int JMAX = mmv_jmax<MODE>();
    constexpr bool MOE = MODE != MAT_DENSE;
    const int warp = tid >> 5, lane = tid & 31;
    const int KB = p.K / 256, lkb = 31 - __clz(KB), lnb = lkb + (MODE == MAT_GATEUP ? 1 : 0), nbu = 1 << lnb;   // (the columns are a power of two)
    int njobs = 1;
    if (MOE) {
        const int nword = p.njobs_max * MMV_JOB_WORDS;
#pragma unroll
        for (int i = 0; i < MMV_JOB_REGS; ++i) {
            const int w = tid + i * MMV_THREADS;
            if (w < nword) reinterpret_cast<int*>(S.jobs_s)[w] = h.jw[i];
        }
        for (int w = tid + MMV_JOB_REGS * MMV_THREADS; w < nword; w += MMV_THREADS) reinterpret_cast<int*>(S.jobs_s)[w] = reinterpret_cast<const int*>(p.jobs)[w];
        njobs = min(h.njobs, p.njobs_max);
        __syncthreads();
    }
    stamp();
    const unsigned upj = p.rows / 16;
    unsigned share = p.share, rest = p.rest;
    if (MOE) {
        const unsigned total = (unsigned) njobs * upj;
        share = mmv_div(total, nblk, p.nblk_inv);
        rest = total - share * nblk;
    }
    const int u0 = (int) mmv_first_unit(share, rest, bid, nblk, p.nblk_inv), u1 = (int) mmv_first_unit(share, rest, bid + 1, nblk, p.nblk_inv);
    auto job_of = [&](int u) { return MOE ? (int) mmv_div(u, upj, p.upj_inv) : 0; };
    const float* norm_w = MODE == MAT_DOWN ? nullptr : p.norm_w;
    uint8_t* slots = S.slots + (size_t) warp * p.R * TILE_BYTES;
    const uint32_t slots_s = smem_u32(slots);
    uint64_t* bars = S.bars + warp * p.R;
    unsigned parity = 0;         // bit i: the phase parity slot i's next read waits for
    Piece* pieces = static_cast<Piece*>(S.pieces);
    Piece* mine = pieces + warp * 2;
    bool first = true, ok = true;
    for (int uc = u0; uc < u1;) {
        const int j0 = job_of(uc), j1 = min(j0 + JMAX, job_of(u1 - 1) + 1), ue = MOE ? min(u1, j1 * (int) upj) : u1;
        const unsigned N = (unsigned) (ue - uc) << lnb;   // (16 N < 2^32: N tiles of 1,760 bytes a block)
        const int i0 = (int) ((N * warp) / MMV_WARPS), i1 = (int) ((N * (warp + 1)) / MMV_WARPS);
        auto item_src = [&](int item) -> const uint8_t* {
            if (!MOE) return p.W + ((size_t) uc * KB + item) * TILE_BYTES;
            const int u = uc + (item >> lnb), j = job_of(u), e = S.jobs_s[j].w;
            int b = item & (nbu - 1);
            size_t tile = (size_t) (u - j * (int) upj);
            if (MODE == MAT_GATEUP && b >= KB) {
                tile += upj;
                b -= KB;
            }
            return (e >= p.E ? p.Wsh : p.W + (size_t) (e - p.e_base) * p.expert_stride) + (tile * KB + b) * TILE_BYTES;
        };
        auto issue = [&](int item, int st) {
            mbar_expect_tx(&bars[st], TILE_BYTES);
            bulk_g2s(slots + (size_t) st * TILE_BYTES, item_src(item), TILE_BYTES, &bars[st]);
        };
        // the pass's first tile blocks are on their way while the rows are quantised, a lane each (the ring is empty: slot i takes item i0 + i)
        if (ok && lane < p.R && i0 + lane < i1) issue(i0 + lane, lane);
        int nlive = p.T, cum[JMAX + 1];
        cum[0] = 0;
        if (MOE) {
#pragma unroll
            for (int sl = 0; sl < JMAX; ++sl) cum[sl + 1] = cum[sl] + (j0 + sl < j1 ? min(S.jobs_s[j0 + sl].n, 4) : 0);
            nlive = cum[JMAX];
        }
        if (!MOE && p.ximg) {   // the image comes ready-made
            const int n16 = (int) (stage_image_bytes(NG, p.K) / 16);
            float4* dst = reinterpret_cast<float4*>(S.cells);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = tid + j * MMV_THREADS;
                const float* d = j < 4 ? &h.v[j >> 1][(j & 1) * 4] : &h.w[(j - 4) >> 1][(j & 1) * 4];
                if (i < n16) dst[i] = make_float4(d[0], d[1], d[2], d[3]);
            }
            for (int i = tid + 8 * MMV_THREADS; i < n16; i += MMV_THREADS) dst[i] = __ldcg(reinterpret_cast<const float4*>(p.ximg) + i);
        } else {
            const int ntask = nlive * KB;
            auto task = [&](int id) {
                if (!MOE) return stage_dense_task(p, id);
                QuantTask q;
                const int i = id >> lkb;   // (the jobs' live rows one after another)
                int sl = 0;
#pragma unroll
                for (int k = 1; k < JMAX; ++k) sl += i >= cum[k];
                const int r = i - cum[sl];
                const fnx_job& jb = S.jobs_s[j0 + sl];
                q.t = sl * 4 + r;
                q.blk = id & (KB - 1);
                q.src = p.x + (size_t) (MODE == MAT_DOWN ? jb.out[r] : jb.y[r]) * p.ldx + q.blk * 256;
                return q;
            };
            auto batch = [&](auto nb, int id0, bool have) {
                constexpr int NB = decltype(nb)::value;
                QuantTask q[NB];
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    q[j] = task(id0 + j * MMV_WARPS);
                    if (!have) quant_fetch(q[j], norm_w, lane, h.v[j], h.w[j]);
                }
                quant_finish(q, h.v, h.w, p.K, norm_w, S.cells, S.scales, S.rs, lane);
            };
            for (int id0 = warp; id0 < ntask; id0 += QUANT_BATCH * MMV_WARPS) {
                const int n = (ntask - id0 + MMV_WARPS - 1) / MMV_WARPS;
                const bool have = !MOE && first && id0 == warp;
                if (n >= 3) batch(std::integral_constant<int, 3>{}, id0, have);
                else if (n == 2) batch(std::integral_constant<int, 2>{}, id0, have);
                else batch(std::integral_constant<int, 1>{}, id0, have);
            }
            static_assert(QUANT_BATCH == 3, "the batches above");
        }
        first = false;
        if (lane < 2) mine[lane].unit = -1;
        __syncthreads();
        stamp();
        // ---- the warp's items
        int cur_job = -1, ntok = p.T, b_lo = 0;
        const int* orow = nullptr;
        LaneX<NG> lx;
        AccT acc[NG][4], gacc[NG][4];
        int b = i0 & (nbu - 1), u = uc + (i0 >> lnb), st = 0;
        for (int s = i0; s < i1 && ok; ++s) {
            if (b == 0 || s == i0) {
                b_lo = b;
#pragma unroll
                for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[ng][k] = gacc[ng][k] = 0;
                const int j = job_of(u);
                if (j != cur_job) {
                    cur_job = j;
                    const int slot = MOE ? j - j0 : 0;
                    if (MOE) {
                        ntok = min(S.jobs_s[j].n, 4);
                        orow = S.jobs_s[j].out;
                    }
                    lane_x_set<NG>(lx, S.cells + (size_t) slot * NG * (p.K / 32) * 32, S.scales + (size_t) slot * NG * KB * 8, p.K, lane);
                    float f = 1.0f;   // lane i: of the image's row i
                    if (norm_w && lane < 4 * NG) f = quant_row_factor(S.rs, slot * 4 * NG + lane, p.K, p.eps);
#pragma unroll
                    for (int ng = 0; ng < NG; ++ng) {
                        lx.r0[ng] = __shfl_sync(0xffffffffu, f, 4 * ng + ((2 * lane) & 2));
                        lx.r1[ng] = __shfl_sync(0xffffffffu, f, 4 * ng + ((2 * lane) & 2) + 1);
                    }
                }
            }
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars[st], (parity >> st) & 1u, 8000000u));
            if (!ok) {
                atomicOr(p.err, (unsigned) FNX_ERR_TIMEOUT);
                break;
            }
            parity ^= 1u << st;
            const uint32_t tile_s = slots_s + st * (uint32_t) TILE_BYTES;
            if (MODE == MAT_GATEUP && b < KB) core_item<NG, AccT>(tile_s, S.table_s, lx, b, lane, gacc);
            else core_item<NG, AccT>(tile_s, S.table_s, lx, MODE == MAT_GATEUP ? b - KB : b, lane, acc);
            __syncwarp();   // every lane is done with the slot
            if (lane == 0 && s + p.R < i1) issue(s + p.R, st);
            st = st + 1 == p.R ? 0 : st + 1;
            if (b == nbu - 1 || s == i1 - 1) {
                // level 1 (threads q = 0, 1) + level 2 (q = 2, 3) of the same rows
#pragma unroll
                for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        acc[ng][k] += __shfl_xor_sync(0xffffffffu, acc[ng][k], 2);
                        if (MODE == MAT_GATEUP) gacc[ng][k] += __shfl_xor_sync(0xffffffffu, gacc[ng][k], 2);
                    }
                if (b_lo == 0 && b == nbu - 1) {
                    stage_write<NG, MODE, AccT>(p, u - cur_job * (int) upj, orow, ntok, lane, gacc, acc);
                } else {
                    Piece* ps = mine + (b_lo == 0 ? 1 : 0);
                    if (lane == 0) ps->unit = u;
                    if ((lane & 3) < 2) {
                        const int l16 = (lane >> 2) * 2 + (lane & 3);
#pragma unroll
                        for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if (MODE == MAT_GATEUP) ps->v[(ng * 16 + l16) * 4 + k] = gacc[ng][k];
                                ps->v[(((Piece::KINDS - 1) * NG + ng) * 16 + l16) * 4 + k] = acc[ng][k];
                            }
                    }
                }
            }
            if (++b == nbu) {
                b = 0;
                ++u;
            }
        }
        __syncthreads();
        stamp();
        // ---- the unit whose first piece the warp holds: the later warps' pieces in warp order
        const int fu = mine[1].unit;
        if (fu >= 0) {
            unsigned rest = __ballot_sync(0xffffffffu, lane > warp && lane < MMV_WARPS && pieces[(lane & (MMV_WARPS - 1)) * 2].unit == fu);
            const int l16 = (lane >> 2) * 2 + (lane & 1);   // (threads q >= 2 read along)
#pragma unroll
            for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    gacc[ng][k] = MODE == MAT_GATEUP ? mine[1].v[(ng * 16 + l16) * 4 + k] : (AccT) 0;
                    acc[ng][k] = mine[1].v[(((Piece::KINDS - 1) * NG + ng) * 16 + l16) * 4 + k];
                }
            for (; rest; rest &= rest - 1) {
                const Piece* c = pieces + (__ffs(rest) - 1) * 2;
#pragma unroll
                for (int ng = 0; ng < NG; ++ng)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (MODE == MAT_GATEUP) gacc[ng][k] += c->v[(ng * 16 + l16) * 4 + k];
                        acc[ng][k] += c->v[(((Piece::KINDS - 1) * NG + ng) * 16 + l16) * 4 + k];
                    }
            }
            const int j = job_of(fu);
            stage_write<NG, MODE, AccT>(p, fu - j * (int) upj, MOE ? S.jobs_s[j].out : nullptr, MOE ? min(S.jobs_s[j].n, 4) : p.T, lane, gacc, acc);
        }
        uc = ue;
        if (uc < u1) __syncthreads();   // the images and the pieces are rewritten by the next pass
        stamp();
    }
}

}  // namespace fnxb
