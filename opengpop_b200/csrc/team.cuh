// team.cuh -- GJ8 steps of one object by a group of lanes (few objects, long requests of a batch).
#pragma once
#include "common.cuh"
#include "corrector.cuh"
#include "gj8_tables.cuh"
#include "lanes.cuh"

namespace gpop {

constexpr int kTeamBlock = 256; // largest block of the kernels that use it

// Steps [a.step_begin, a.step_end) of object obj. The lanes of the team split its gravity columns (lanes.cuh,
// lane-layout table) and hold identical state, and lane 0 stores. A team is P lanes of a warp, or (WARPS) whole
// warps with a lane per column. The acceleration history lies in shared memory (hist, 27 doubles) meanwhile.
// warp: the lanes of this warp that run (teams of lanes).
// Bounds: the latency of an evaluation (one chain of FMAs per column, then a sum over the lanes; captured for one
// object at 70x70: an instruction issued in 23 % of the cycles, waits per issue 1.36 on fixed latency, 1.0 at the
// team's barrier, 0.56 on shared memory), so what a
// step needs besides is kept short: history and sums in shared memory, the next step's rotation in registers
// (prefetched into L1 only: 2.2 instead of 2.05 us per step at 8x8).
// In blocks of at most 256 threads: with 255 registers a step of one object on 32 lanes takes 9.2 us at 70x70
// (FP64), with the 168 of 384 threads 16.9. At 70x70 on 96 lanes, of 13,400 cycles per step two walks of the
// columns take 3,750 each (54 a term; nine FP64 instructions of one warp issue in 30), their sums, rotations
// and start 1,900 each, the corrector 630 per evaluation, prediction and end 700.
// Taken back: two warps per 32 columns, each with half of the sums (6.5 us per step, as without: the loads of
// more warps meet at the one shared-memory port), and four terms loaded ahead (6.4, as without).
template <bool MIXED, bool WARPS, class Team>
__device__ __forceinline__ void team_steps(const TableSrc& ts, const GravSmem& g, const PropArgs& a, const Team& team,
    int64_t obj, int P, double* hist, unsigned warp)
{
    const int64_t n = a.n; // the state's stride
    const int l = team.l;
    const bool lead = l == 0;
    double* st = a.state + obj;
    for (int i = l; i < 27; i += P)
        hist[i] = st[(kHist + i) * n];
    team.sync();
    const double h = a.h;
    double r[1][3], v[3], s[3], S[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        r[0][j] = st[(kR + j) * n];
        v[j] = st[(kV + j) * n];
        s[j] = st[(kSs + j) * n];
        S[j] = st[(kSb + j) * n];
    }
    int ring0 = a.step_begin >= 5 ? (a.step_begin - 5) % 9 : 0;
    double next_m[9]; // the next step's rotation
    auto rotation = [&](int step) {
#pragma unroll
        for (int i = 0; i < 9; ++i)
            next_m[i] = __ldg(a.prop_m + (size_t)(step + 4) * 9 + i);
    };
    rotation(max(a.step_begin, 5) < a.step_end ? max(a.step_begin, 5) : a.step_begin);
    for (int step = a.step_begin; step < a.step_end; ++step) {
        double a8[1][3];
        if (step <= 4) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                r[0][j] = st[(kRep + (step - 1) * 6 + j) * n];
                v[j] = st[(kRep + (step - 1) * 6 + 3 + j) * n];
                a8[0][j] = st[(kRepA + (step - 1) * 3 + j) * n];
            }
        } else {
            double M[9];
#pragma unroll
            for (int i = 0; i < 9; ++i)
                M[i] = next_m[i];
            if (step + 1 < a.step_end)
                rotation(step + 1);
            double s1[3], s2[3], prev[3], a7[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) { // as gj8_kernel
                double q[9];
#pragma unroll
                for (int c = 0; c < 9; ++c) {
                    int slot = ring0 + c;
                    slot -= slot >= 9 ? 9 : 0;
                    q[c] = hist[slot * 3 + j];
                }
                double rt = 0.0, c1 = 0.0, c2 = 0.0;
#pragma unroll
                for (int c = 0; c < 9; ++c)
                    rt = fma(q[c], c_GJ[9][c], rt);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    c1 = fma(q[c + 1], c_SA[8][c], c1);
                    c2 = fma(q[c + 1], c_GJ[8][c], c2);
                }
                S[j] += s[j] + q[8] / 2;
                r[0][j] = (rt + S[j]) * h * h;
                s1[j] = c1;
                s2[j] = c2;
                prev[j] = s[j];
                a7[j] = q[8];
            }
            bool fast = false;
            for (int it = 0; it < a.ncorr; ++it) {
                gravity_gcrs_team<MIXED, 1, !WARPS>(g, team, M, r, a8);
                if (correct_position(ts.corr, h, it, a.ncorr, s2, S, a8[0], r[0], fast))
                    break; // the same for the lanes of a group
            }
            if constexpr (!WARPS)
                __syncwarp(warp); // groups that were done earlier wait: the warp's walks stay converged
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                s[j] = prev[j] + (a8[0][j] + a7[j]) / 2;
                v[j] = h * (s1[j] + a8[0][j] * c_SA[8][8] + s[j]);
            }
            if (lead)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    hist[ring0 * 3 + j] = a8[0][j];
            team.sync(); // the ring write precedes the group's loads of the next step
            ring0 = ring0 == 8 ? 0 : ring0 + 1;
        }
        if (lead) {
            const int64_t t = step - a.traj_step0;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                if (a.traj_r)
                    a.traj_r[(t * 3 + j) * n + obj] = r[0][j];
                if (a.traj_v)
                    a.traj_v[(t * 3 + j) * n + obj] = v[j];
                if (a.traj_a)
                    a.traj_a[(t * 3 + j) * n + obj] = a8[0][j];
            }
        }
    }
    for (int i = l; i < 27; i += P)
        st[(kHist + i) * n] = hist[i];
    if (!lead)
        return;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        st[(kR + j) * n] = r[0][j];
        st[(kV + j) * n] = v[j];
        st[(kSs + j) * n] = s[j];
        st[(kSb + j) * n] = S[j];
        if (a.out_r)
            a.out_r[obj * 3 + j] = r[0][j];
        if (a.out_v)
            a.out_v[obj * 3 + j] = v[j];
    }
}

} // namespace gpop
