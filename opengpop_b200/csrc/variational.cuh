// variational.cuh -- state transition matrices (forward variational equations) and the adjoint of
// the GJ8 propagation with respect to the initial state, plus the closest approach of explicit
// object pairs with the gradient of its miss distance (FP64 throughout).
#pragma once
#include "kernels.h"

#include <cstdint>

namespace gpop {

constexpr int kCheckpointSteps = 64; // GJ8 state saved every 64 steps for the reverse sweep
constexpr int kCheckpointArrays = 33; // s, S and the 9-slot history (state arrays kSs .. kHist + 26)

// Jacobians at many positions: item i (a step, an RK8 stage, a column) of object o lies at
// pos[(i 3 + j) n + o] in the frame M[i 9 ..]. Entry t of the result, 9 arrays of `total`, is item i's
// u-th object (obj[u], or u): t = i width + u, or offset[i] + u where the items hold fewer and fewer.
// With acc (laid out as pos) the Jacobian is taken where gravity is acc, next to pos: the positions of a step are
// those after its last corrector pass, its acceleration that of the evaluation before.
struct JacPoints {
    int64_t n = 0; // stride of the positions
    const double* pos = nullptr;
    const double* acc = nullptr;
    const double* M = nullptr;
    int frames = 0; // M of item i is that of i % frames (0: of i)
    const double* mark = nullptr; // [n]: objects with NaN here are left out (may be NULL)
    int64_t width = 0;
    int items = 0;
    const int64_t* offset = nullptr; // [items], ascending
    const int* obj = nullptr;
    int64_t total = 0;
    double* jac = nullptr;
    unsigned* err = nullptr;
};

// Startup tangents of n objects along the six initial-state directions: kStartupTangents arrays of 6 n
// (direction-major): accelerations of the nine columns, s and S of column 8, positions, then velocities of
// columns 5..8.
constexpr int kStartupTangents = 57;
struct StartupTangentArgs {
    int64_t n = 0;
    double h = 0;
    int ncorr = 7;
    const double* stage_jac = nullptr; // 9 arrays of 80 n, stages in the order of gen_m
    const double* col_jac = nullptr; // 9 arrays of 9 n, at the columns' last positions
    const double* mark = nullptr; // [n] StartupArgs::pass_pos: NaN where the passes have converged
    // passes [pass_lo, pass_hi) of the other objects: Jacobians at the columns in front of each, 9 arrays of
    // (pass_hi - pass_lo) 9 n
    const double* pass_jac = nullptr;
    int pass_lo = 0, pass_hi = 0;
    double* out = nullptr;
};

// Tangents through steps step_lo..step_hi (>= 5).
constexpr int kStmSweep = 39;
struct StmArgs {
    int64_t n = 0;
    int steps = 0, step_lo = 5, step_hi = 4;
    double h = 0;
    int ncorr = 7;
    bool first = false, last = false; // first: starts from `startup`; last: writes phi
    const double* startup = nullptr;
    const double* jac = nullptr; // 9 arrays of (step_hi - step_lo + 1) n
    double* sweep = nullptr; // kStmSweep arrays of 6 n, carried between windows
    double* phi = nullptr; // [n][6][6], phi[i][j] = d x_N,i / d x_0,j with x = (r, v)
};

// One adjoint unit: an object with cotangents ("seeds") on its trajectory (r, v, a) at up to three
// consecutive steps step0, step0 + 1, step0 + 2 (1-based; steps beyond the run are ignored). Ranks order
// the units by their last seeded step, latest first (unit: NULL for the identity).
constexpr int kAdjSweep = 33;
struct AdjSweepArgs {
    int64_t n_units = 0;
    const int* unit = nullptr;
    const int* seed_step0 = nullptr;
    const double* seeds = nullptr; // [n_units][3 nodes][r 3 | v 3 | a 3]
    int steps = 0, step_lo = 5, step_hi = 4;
    double h = 0;
    int ncorr = 7;
    bool first = false;
    const double* jac = nullptr; // 9 arrays of total
    const int64_t* offset = nullptr; // as JacPoints::offset
    int64_t total = 0;
    double* sweep = nullptr; // kAdjSweep arrays of n_units, carried between windows
};
struct AdjFinishArgs {
    int64_t n_units = 0;
    const int* unit = nullptr;
    const int* unit_obj = nullptr;
    const int* seed_step0 = nullptr;
    const double* seeds = nullptr;
    int steps = 0;
    uint32_t flags = 0;
    const double* sweep = nullptr;
    const double* startup = nullptr; // tangents of objects [obj_lo, obj_lo + n)
    int64_t obj_lo = 0, n = 0;
    double* grad = nullptr; // [n_units][6] d(seeded sum) / d(r0, v0)
};

// Closest approach of listed pairs over a stored trajectory ([steps][3][n] r, v, a) and the seeds
// of the miss-distance adjoint (units 2p and 2p + 1 = the pair's two objects).
struct PairArgs {
    int64_t n_obj = 0;
    int64_t n_pairs = 0;
    const int* pairs = nullptr; // [n_pairs][2]
    int steps = 0;
    double h = 0;
    const double* traj_r = nullptr;
    const double* traj_v = nullptr;
    const double* traj_a = nullptr;
    double* tca = nullptr; // [n_pairs]
    double* miss = nullptr;
    int* closest = nullptr; // trajectory index of the sampled minimum
    int* unit_obj = nullptr; // [2 n_pairs]
    int* seed_step0 = nullptr;
    double* seeds = nullptr; // [2 n_pairs][27]
};

cudaError_t launch_jac_points(const TableSrc& plain64, const JacPoints& a, int num_sms, cudaStream_t s);
// Of the startup, in this order: the RK8 chains, the plain corrector passes (in as many windows as their Jacobians
// come in), the end.
cudaError_t launch_rk8_tangents(const StartupTangentArgs& a, cudaStream_t s);
cudaError_t launch_pass_tangents(const StartupTangentArgs& a, cudaStream_t s);
cudaError_t launch_corrector_tangents(const StartupTangentArgs& a, cudaStream_t s);
cudaError_t launch_stm_sweep(const StmArgs& a, cudaStream_t s);
cudaError_t launch_adjoint_sweep(const AdjSweepArgs& a, cudaStream_t s);
cudaError_t launch_adjoint_finish(const AdjFinishArgs& a, cudaStream_t s);
cudaError_t launch_pair_approach(const PairArgs& a, cudaStream_t s);
// Acceleration (may be NULL) and 3x3 Jacobian [n][3][3] at GCRS positions r [n][3] with the frame
// matrix M of gravity_gcrs (NULL = Earth-fixed positions, no rotation).
cudaError_t launch_jacobian(const TableSrc& plain64, const TableSrc& lane64, int64_t n, const double* r,
    const double* M, double* acc, double* jac, unsigned* err, int num_sms, cudaStream_t s);

} // namespace gpop
