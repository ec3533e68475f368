// batch.cu -- one persistent launch for many independent propagation requests.
//
// Requests differ in object count, duration, step size and gravity degree. A request's objects
// advance one step at a time, so its duration sets a critical path that a larger batch cannot
// shorten; the planner (batch_api.cu) therefore gives long requests several lanes per object:
// the lanes of an object split the gravity columns (lane l of P takes m = l, l + P, ...) and add
// their sums with warp shuffles. Warps pull work items (a request's group of 32 / P objects, all of
// its steps) from a global queue ordered longest first, so the grid stays busy until the end.
#include "batch.cuh"
#include "common.cuh"
#include "corrector.cuh"
#include "frames_block.cuh"
#include "gravity.cuh"
#include "gj8_tables.cuh"
#include "lanes.cuh"
#include "startup.cuh"
#include "team.cuh"

#include <type_traits>

namespace gpop {

template <bool MIXED>
__device__ __forceinline__ bool stage_batch_table(uint8_t* smem, const TableSrc& ts, unsigned* err, GravSmem& g)
{
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);
    uint8_t* tab = smem + 128;
    const bool ok = stage_to_smem(tab, ts.src, ts.bytes, mbar, err, ts.wait_spins);
    g.L = ts.L;
    g.Lt = ts.L;
    g.radius = ts.radius;
    g.gm = ts.gm;
    g.t64 = reinterpret_cast<const GravEntry64*>(tab);
    g.t32 = reinterpret_cast<const GravEntry32*>(tab + ts.off32);
    return ok;
}

// Two objects per lane may walk the gravity columns two at a time (as gj8_kernel does), in
// batches whose items all have one lane per object (BatchArgs::pair_walk).
#ifndef GPOP_BATCH_PAIRS
#define GPOP_BATCH_PAIRS 1
#endif
constexpr bool kBatchPairs = GPOP_BATCH_PAIRS != 0;
// Two-object items park the corrector's constants (as in gj8_kernel: 12 doubles per object) in
// shared memory while the gravity walk runs, as gj8_kernel does, when that fits beside the table.
#ifndef GPOP_BATCH_STAGE
#define GPOP_BATCH_STAGE 1
#endif
constexpr bool kBatchStage = GPOP_BATCH_STAGE != 0;
constexpr int kBatchStageDoubles = 24; // two objects x 12
// Batches of single-lane items stage the plain table and run gj8_kernel's gravity walk (no lane
// code in that kernel).
#ifndef GPOP_BATCH_PLAIN
#define GPOP_BATCH_PLAIN 1
#endif
constexpr bool kBatchPlain = GPOP_BATCH_PLAIN != 0;

// One work item on one warp: K = 2 objects per lane for single-lane items (up to 64 objects),
// else one object per group of P lanes (up to 32 / P objects).
template <bool MIXED, int K, bool STAGE, bool PAIRS>
__device__ __forceinline__ void run_item(const GravSmem& g0, const CorrModel& cm, const BatchArgs& a, const BatchItem& it,
    const BatchReq& rq, int lane, double* stage)
{
    constexpr bool kStage = K == 2 && STAGE;
    // staged value q (0..3: s2, last, prev, s1) of object k, axis j
    auto slot = [&](int q, int k, int j) { return stage + (size_t)((q * K + k) * 3 + j) * blockDim.x; };
    const int64_t n = a.n_obj;
    double* st = a.state;
    const int P = K == 1 ? rq.lpo : 1;
    const int sl = lane % P;
    int64_t o[K];
    bool valid[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int slot = K == 1 ? lane / P : lane + 32 * k;
        valid[k] = slot < it.count;
        o[k] = rq.obj0 + it.first + (valid[k] ? slot : 0); // idle slots shadow slot 0
    }
    const bool lead = sl == 0;
    GravSmem g = g0;
    g.L = rq.L;
    const double h = rq.h;
    double r[K][3], v[K][3], s[K][3], S[K][3];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            r[k][j] = st[(kR + j) * n + o[k]];
            v[k][j] = st[(kV + j) * n + o[k]];
            s[k][j] = st[(kSs + j) * n + o[k]];
            S[k][j] = st[(kSb + j) * n + o[k]];
        }
    for (int step = 1; step <= rq.steps; ++step) {
        if (step <= 4) {
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    r[k][j] = st[(kRep + (step - 1) * 6 + j) * n + o[k]];
                    v[k][j] = st[(kRep + (step - 1) * 6 + 3 + j) * n + o[k]];
                }
            continue;
        }
        const int ring0 = (step - 5) % 9;
        double s1[K][3], s2[K][3], prev[K][3], a7[K][3], last[K][3], a8[K][3]; // as gj8_kernel
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double hist[9][3];
#pragma unroll
            for (int c = 0; c < 9; ++c) {
                int sl9 = ring0 + c;
                sl9 -= sl9 >= 9 ? 9 : 0;
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    hist[c][j] = st[(kHist + sl9 * 3 + j) * n + o[k]];
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) { // predictor, as in gj8_kernel
                double vt = 0.0, rt = 0.0;
#pragma unroll
                for (int c = 0; c < 9; ++c) {
                    vt = fma(hist[c][j], c_SA[9][c], vt);
                    rt = fma(hist[c][j], c_GJ[9][c], rt);
                }
                S[k][j] += s[k][j] + hist[8][j] / 2;
                v[k][j] = (vt + s[k][j] + hist[8][j] / 2) * h;
                r[k][j] = (rt + S[k][j]) * h * h;
                double c1 = 0.0, c2 = 0.0;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    c1 = fma(hist[c + 1][j], c_SA[8][c], c1);
                    c2 = fma(hist[c + 1][j], c_GJ[8][c], c2);
                }
                s1[k][j] = c1;
                s2[k][j] = c2;
                prev[k][j] = s[k][j];
                a7[k][j] = hist[8][j];
                last[k][j] = r[k][j];
                if constexpr (kStage) {
                    st_stage(slot(0, k, j), s2[k][j]);
                    st_stage(slot(1, k, j), last[k][j]);
                    st_stage(slot(2, k, j), prev[k][j]);
                    st_stage(slot(3, k, j), s1[k][j]);
                }
            }
        }
        const double* M = rq.prop_m + (size_t)(step + 4) * 9;
        bool done[K] = {}, fast[K] = {};
        for (int itc = 0; itc < a.ncorr; ++itc) { // as gj8_kernel
            if constexpr (K == 2 && PAIRS && kBatchPlain) {
                gravity_gcrs<MIXED, 2>(g, M, r, a8); // the plain table: gj8_kernel's walk
            } else if constexpr (K == 2 && PAIRS) {
                // two objects per lane: the two-column walk on the lane-layout tables (mixed
                // needs degree > 8 for it)
                if (!MIXED || g.L > kMixedSplit)
                    gravity_gcrs<MIXED, 2, true>(g, M, r, a8);
                else
                    gravity_gcrs_lk<MIXED, K>(g, sl, P, M, r, a8, 0xffffffffu);
            } else {
                gravity_gcrs_lk<MIXED, K>(g, sl, P, M, r, a8, 0xffffffffu);
            }
            bool all = true;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (!done[k]) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        if constexpr (kStage) {
                            s2[k][j] = ld_stage(slot(0, k, j));
                            last[k][j] = ld_stage(slot(1, k, j));
                        }
                    }
                    done[k] = correct_position(cm, h, itc, a.ncorr, s2[k], S[k], a8[k], last[k], fast[k]);
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        if constexpr (kStage) {
                            st_stage(slot(1, k, j), last[k][j]);
                            if (done[k])
                                st_stage(slot(0, k, j), a8[k][j]);
                        } else if (done[k]) {
                            s2[k][j] = a8[k][j];
                        }
                    }
                }
                all = all && done[k];
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    r[k][j] = kStage ? ld_stage(slot(1, k, j)) : last[k][j];
            }
            if (__all_sync(0xffffffffu, all)) // the lane walk's shuffles name the whole warp
                break;
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                a8[k][j] = kStage ? ld_stage(slot(0, k, j)) : s2[k][j];
                if constexpr (kStage) {
                    prev[k][j] = ld_stage(slot(2, k, j));
                    s1[k][j] = ld_stage(slot(3, k, j));
                    a7[k][j] = __ldcg(st + (kHist + (ring0 + 8 - (ring0 > 0 ? 9 : 0)) * 3 + j) * n + o[k]);
                }
                s[k][j] = prev[k][j] + (a8[k][j] + a7[k][j]) / 2;
                v[k][j] = h * (s1[k][j] + a8[k][j] * c_SA[8][8] + s[k][j]);
            }
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (lead && valid[k])
                for (int j = 0; j < 3; ++j)
                    st[(kHist + ring0 * 3 + j) * n + o[k]] = a8[k][j];
        __syncwarp(); // the ring write precedes the other lanes' loads of the next step
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (lead && valid[k])
            for (int j = 0; j < 3; ++j) {
                st[(kR + j) * n + o[k]] = r[k][j];
                st[(kV + j) * n + o[k]] = v[k][j];
                st[(kSs + j) * n + o[k]] = s[k][j];
                st[(kSb + j) * n + o[k]] = S[k][j];
                a.r_out[o[k] * 3 + j] = rq.steps > 0 ? r[k][j] : a.r0[o[k] * 3 + j];
                a.v_out[o[k] * 3 + j] = rq.steps > 0 ? v[k][j] : a.v0[o[k] * 3 + j];
            }
}

// Persistent GJ8 kernel: warps pull work items until the queue is empty. One 256-thread block per
// SM: the two-object path needs the registers of 8 warps.
template <bool MIXED, bool STAGE, bool PAIRS>
__global__ void __launch_bounds__(256, 1) batch_gj8_kernel(TableSrc ts, BatchArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr bool kPlain = PAIRS && kBatchPlain;
    GravSmem g0;
    if constexpr (kPlain) {
        if (!stage_batch_table<MIXED>(smem, ts, a.err, g0))
            return;
    } else {
        if (!bind_lane_table(smem, ts, a.err, g0))
            return;
    }
    const int lane = threadIdx.x & 31;
    double* stage = reinterpret_cast<double*>(smem + stage_offset(ts)) + threadIdx.x;
    for (;;) {
        int item = 0;
        if (lane == 0)
            item = atomicAdd(a.next_item, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.n_items)
            break;
        const BatchItem it = a.items[item];
        const BatchReq rq = a.reqs[it.req];
        if constexpr (kPlain) { // every item has one lane per object
            run_item<MIXED, 2, STAGE, PAIRS>(g0, ts.corr, a, it, rq, lane, stage);
        } else {
            if (rq.lpo == 1)
                run_item<MIXED, 2, STAGE, PAIRS>(g0, ts.corr, a, it, rq, lane, stage);
            else
                run_item<MIXED, 1, false, false>(g0, ts.corr, a, it, rq, lane, stage);
        }
    }
}

// Objects of the longest requests, each by a team of warps with a lane per column (team.cuh) on SMs of their own:
// a request's steps follow one another, so the longest one bounds the batch. 24 objects x 7,780 steps at 70x70,
// 256 requests of one to 512 objects: 72 of 81 ms on warps of the persistent kernel (9.3 us per step), 38 here, the
// call 57 with the other requests on more lanes. FP64 in mixed precision too: it is the faster one there.
__global__ void __launch_bounds__(kTeamBlock, 1) batch_team_kernel(TableSrc ts, BatchArgs a, int P)
{
    extern __shared__ __align__(128) uint8_t smem[];
    GravSmem g;
    if (!bind_lane_table(smem, ts, a.err, g))
        return;
    double* hist = reinterpret_cast<double*>(smem + stage_offset(ts))
        + (size_t)(threadIdx.x / P) * team_doubles(P, true);
    int* item = reinterpret_cast<int*>(hist + team_doubles(P, true) - 1);
    const auto team = make_team<true>(P, hist + 27);
    for (;;) {
        if (team.l == 0)
            *item = atomicAdd(a.next_item + 1, 1);
        team.sync();
        const int i = *item;
        team.sync(); // read by all before the next one is fetched
        if (i >= a.n_team)
            break;
        const BatchItem it = a.team_items[i];
        const BatchReq rq = a.reqs[it.req];
        g.L = rq.L;
        PropArgs p;
        p.n = a.n_obj;
        p.state = a.state;
        p.h = rq.h;
        p.ncorr = a.ncorr;
        p.prop_m = rq.prop_m;
        p.step_end = rq.steps + 1;
        p.out_r = a.r_out;
        p.out_v = a.v_out;
        team_steps<false, true>(ts, g, p, team, rq.obj0 + it.first, P, hist, 0xffffffffu);
    }
}

template <class K> static cudaError_t set_smem(K kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t launch_batch_startup(const TableSrc& lane_ts, const TableSrc& plain_ts, const BatchArgs& a,
    int num_sms, cudaStream_t s)
{
    StartupArgs b;
    b.n = a.n_obj;
    b.reqs = a.reqs;
    b.obj_req = a.obj_req;
    b.ncorr = a.ncorr;
    b.flags = a.flags;
    b.r0 = a.r0;
    b.v0 = a.v0;
    b.state = a.state;
    b.counters = reinterpret_cast<int*>(a.state + (size_t)kStateArrays * a.n_obj);
    b.err = a.err;
    return launch_startup_gravity(plain_ts, lane_ts, b, num_sms, s);
}

template <bool MIXED, bool STAGE, bool PAIRS>
static cudaError_t launch_batch_gj8_k(const TableSrc& ts, const BatchArgs& a, int blocks, int block,
    size_t smem, cudaStream_t s)
{
    cudaError_t e = set_smem(batch_gj8_kernel<MIXED, STAGE, PAIRS>, smem);
    if (e != cudaSuccess)
        return e;
    batch_gj8_kernel<MIXED, STAGE, PAIRS><<<blocks, block, smem, s>>>(ts, a);
    return cudaGetLastError();
}

template <bool MIXED>
static cudaError_t launch_batch_gj8_m(const TableSrc& lane_ts, const TableSrc& plain_ts, const BatchArgs& a,
    int blocks, int block, cudaStream_t s)
{
    const bool pairs = kBatchPairs && a.pair_walk;
    const TableSrc& ts = pairs && kBatchPlain ? plain_ts : lane_ts;
    const size_t staged = stage_offset(ts) + (size_t)kBatchStageDoubles * 8 * block;
    const bool stage = kBatchStage && staged <= max_smem_optin();
    const size_t smem = stage ? staged : table_smem_bytes(ts);
    if (stage)
        return pairs ? launch_batch_gj8_k<MIXED, true, true>(ts, a, blocks, block, smem, s)
                     : launch_batch_gj8_k<MIXED, true, false>(ts, a, blocks, block, smem, s);
    return pairs ? launch_batch_gj8_k<MIXED, false, true>(ts, a, blocks, block, smem, s)
                 : launch_batch_gj8_k<MIXED, false, false>(ts, a, blocks, block, smem, s);
}

cudaError_t launch_batch_gj8(const TableSrc& lane_ts, const TableSrc& plain_ts, const BatchArgs& a,
    int blocks, int block, cudaStream_t s)
{
    if (a.n_items <= 0)
        return cudaSuccess;
    return lane_ts.mixed ? launch_batch_gj8_m<true>(lane_ts, plain_ts, a, blocks, block, s)
                         : launch_batch_gj8_m<false>(lane_ts, plain_ts, a, blocks, block, s);
}

cudaError_t launch_batch_teams(const TableSrc& lane64, const BatchArgs& a, int blocks, int teams, int lanes,
    cudaStream_t s)
{
    const size_t bytes = stage_offset(lane64) + (size_t)teams * team_doubles(lanes, true) * sizeof(double);
    cudaError_t e = set_smem(batch_team_kernel, bytes);
    if (e != cudaSuccess)
        return e;
    batch_team_kernel<<<blocks, teams * lanes, bytes, s>>>(lane64, a, lanes);
    return cudaGetLastError();
}

// ---- epoch tables of many requests: epoch e uses calendar cal[5 * epoch_req[e]] ----
__global__ void __launch_bounds__(kFrameThreads) frames_batch_kernel(FrameData fd, const int* __restrict__ cal,
    const int* __restrict__ epoch_req, const double* __restrict__ sec_args, double* __restrict__ m_out)
{
    const int e = (int)blockIdx.x;
    const int* c = cal + 5 * epoch_req[e];
    frames_epoch(fd, c[0], c[1], c[2], c[3], c[4], sec_args[e], m_out + (size_t)e * 9, nullptr);
}

cudaError_t launch_frames_batch(const FrameData& fd, const int* cal, const int* epoch_req,
    const double* sec_args, int count, double* m_out, cudaStream_t s)
{
    if (count <= 0)
        return cudaSuccess;
    frames_batch_kernel<<<count, kFrameThreads, 0, s>>>(fd, cal, epoch_req, sec_args, m_out);
    return cudaGetLastError();
}

} // namespace gpop
