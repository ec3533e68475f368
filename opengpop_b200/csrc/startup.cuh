// startup.cuh -- the GJ8 startup under gravity as a pipeline over all objects (startup.cu).
#pragma once
#include "batch.cuh"
#include "kernels.h"

namespace gpop {

// The objects of one startup: all of one propagation (h, L, tables here), or the flattened objects of
// a batch (reqs and obj_req set: each request has its own).
struct StartupArgs {
    int64_t n = 0;
    double h = 0;
    const double* gen_m = nullptr;
    const double* prop_m = nullptr;
    const BatchReq* reqs = nullptr;
    const int* obj_req = nullptr;
    int ncorr = 7;
    uint32_t flags = 0;
    const double* r0 = nullptr; // AoS [n][3]
    const double* v0 = nullptr;
    double* state = nullptr; // kStateArrays x n; holds the startup's matrices until it ends
    int* counters = nullptr; // kStartupCounters: evaluations listed by each corrector pass
    bool check = false; // raise kErrBadInput for states gravity cannot take
    unsigned* err = nullptr;
    // for the variational equations (may be NULL): positions of the 80 RK8 stages, in the order of gen_m,
    // and of the nine columns at the end, [.][3][n]; of the columns in front of every corrector pass,
    // [ncorr][9][3][n], for objects that take the plain passes (NaN in the first value of the others)
    double* stage_pos = nullptr;
    double* col_pos = nullptr;
    double* pass_pos = nullptr;
};

// plain: the plain table, lanes: the lane-layout table of the same precision.
cudaError_t launch_startup_gravity(const TableSrc& plain, const TableSrc& lanes, const StartupArgs& a,
    int num_sms, cudaStream_t s);

} // namespace gpop
