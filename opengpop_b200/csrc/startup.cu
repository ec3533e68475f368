// startup.cu -- RK8 startup and mid-corrector under gravity (lib/gpu_startup/src/gpu_startup.cu) as a
// pipeline of kernels, for one propagation's objects or a batch's.
//
// The startup is 8 RK8 steps of 10 stages and 7 mid-corrector passes over 8 columns, 145 evaluations per
// object when one thread makes them in a row, with 3.6 KB of matrices per thread. Here
// - the forward and the backward RK8 chain of an object run side by side (40 evaluations in a row), a
//   stage keeps only the accelerations (the velocity stages are folded into the position's
//   coefficients), and the accelerations at columns 4..7 are those of the forward steps' first stage;
// - the evaluations of the corrector's columns are independent: a kernel of its own makes them, one
//   (object, column) per thread or lane group, from a list of the columns that moved;
// - the corrector's linear algebra is one thread per object between them. Like correct_position it moves
//   to the fixed point of the passes with the Jacobian of the central term and J2, when the passes would
//   reach it, so two rounds of evaluations serve for seven: 93 evaluations per object instead of 145.
// Bounds: the gravity walk for many objects, its latency times 45 for few. Measured on B200 at 70x70, the
// whole startup, one thread per object (65,536: the split block) -> here: 1 object FP64 5.88 -> 0.19 ms;
// 18,501 FP64 7.8 -> 4.0 ms; 65,536 mixed 14.1 -> 6.3 ms. Captured, RK8 chains of 18,501 objects, FP64 at one per
// thread (3.2 ms): shared-memory loads at 91 % of their port, FP64 pipe 62 % busy.
#include "common.cuh"
#include "corrector.cuh"
#include "gj8_tables.cuh"
#include "gravity.cuh"
#include "integrator.cuh"
#include "lanes.cuh"
#include "startup.cuh"

#include <algorithm>

namespace gpop {

namespace {

// ---- coefficients ----
struct Rkn {
    double c[10], a[10][9]; // position stage k: r + hh (c[k] v + hh sum_j a[k][j] K_j)
    double b[9]; // new position: r + hh (v + hh sum_j b[j] K_j)
};
// c = the row sums of A, a = A^2 and b = B A of the RK8 table. (Row 7 of the reference's table sums to
// 17/20 while its node is 1; the sums are what its velocity stages take.)
constexpr Rkn make_rkn()
{
    constexpr double A[10][9] = { {}, { 4.0 / 27 }, { 1.0 / 18, 3.0 / 18 }, { 1.0 / 12, 0.0, 3.0 / 12 },
        { 1.0 / 8, 0, 0, 3.0 / 8 }, { 13.0 / 54, 0.0, -27.0 / 54, 42.0 / 54, 8.0 / 54 },
        { 389.0 / 4320, 0.0, -54.0 / 4320, 966.0 / 4320, -824.0 / 4320.0, 243.0 / 4320 },
        { -234.0 / 20, 0, 81.0 / 20, -1164.0 / 20, 656.0 / 20, -122.0 / 20, 800.0 / 20 },
        { -127.0 / 288, 0.0, 18.0 / 288, -678.0 / 288, 456.0 / 288, -9.0 / 288, 576.0 / 288, 4.0 / 288 },
        { 1481.0 / 820, 0.0, -81.0 / 820, 7104.0 / 820, -3376.0 / 820, 72.0 / 820, -5040.0 / 820,
            -60.0 / 820, 720.0 / 820 } };
    constexpr double B[10] = { 41.0 / 840.0, 0.0, 0.0, 27.0 / 840.0, 272.0 / 840.0, 27.0 / 840.0,
        216.0 / 840.0, 0.0, 216.0 / 840.0, 41.0 / 840.0 };
    Rkn t {};
    for (int k = 0; k < 10; ++k)
        for (int j = 0; j < 9; ++j) {
            t.c[k] += A[k][j];
            for (int i = j + 1; i < k; ++i)
                t.a[k][j] += A[k][i] * A[i][j];
        }
    for (int j = 0; j < 9; ++j)
        for (int i = j + 1; i < 10; ++i)
            t.b[j] += B[i] * A[i][j];
    return t;
}
__constant__ Rkn c_rkn = make_rkn();

// How the positions of a corrector pass answer to its accelerations: dr_c = h^2 sum_k m[c][k] da_k, the
// GJ sums and the s, S chain from column 4 (corrector_s0, corrector_all_s), column 4 held.
struct PassMatrix {
    float m[9][9];
};
constexpr PassMatrix make_pass()
{
    constexpr double GJ4[9] = { 317.0 / 22809600.0, -2539.0 / 13305600.0, 55067.0 / 39916800.0,
        -326911.0 / 39916800.0, 14797.0 / 152064.0, -326911.0 / 39916800.0, 55067.0 / 39916800.0,
        -2539.0 / 13305600.0, 317.0 / 22809600.0 };
    constexpr double SA4[9] = { -2497.0 / 7257600.0, 1469.0 / 403200.0, -68119.0 / 3628800.0,
        252769.0 / 3628800.0, 0.0, -252769.0 / 3628800.0, 68119.0 / 3628800.0, -1469.0 / 403200.0,
        2497.0 / 7257600.0 };
    PassMatrix t {};
    for (int k = 0; k < 9; ++k) {
        double s[9] = {}, S[9] = {}, a[9] = {};
        a[k] = 1.0;
        s[4] = -SA4[k];
        S[4] = -GJ4[k];
        for (int i = 1; i <= 4; ++i) {
            s[4 + i] = s[3 + i] + (a[3 + i] + a[4 + i]) / 2;
            s[4 - i] = s[5 - i] - (a[5 - i] + a[4 - i]) / 2;
            S[4 + i] = s[3 + i] + S[3 + i] + a[3 + i] / 2;
            S[4 - i] = -s[5 - i] + S[5 - i] + a[5 - i] / 2;
        }
        for (int c = 0; c < 9; ++c)
            t.m[c][k] = (float)S[c]; // the GJ row of column c is added on the device
    }
    return t;
}
__constant__ PassMatrix c_pass = make_pass();

// ---- layout of the state while the startup runs (final layout: StateSlot) ----
// 0..3 list of (object, column) evaluations as 8 n ints; 6..11 s and S of column 8 (final place);
// 12..38 accelerations (final place); 39..65 positions; 66..77 velocities of columns 5..8; 78..80 the
// initial velocity; 81 per-object flags (int).
constexpr int kSr = 39, kSv = 66, kSv4 = 78, kSflag = 81;
static_assert(kSflag < kStateArrays && kHist == 12 && kSs == 6, "startup layout");
enum : int { kFlagDone = 1, kFlagFast = 2 };

struct ObjSrc {
    double h;
    int L;
    const double* gen_m;
    const double* prop_m;
};
template <bool BATCH> __device__ __forceinline__ ObjSrc source(const StartupArgs& a, int64_t o, int L)
{
    if constexpr (BATCH) {
        const BatchReq& q = a.reqs[a.obj_req[o]];
        return { q.h, q.L, q.gen_m, q.prop_m };
    } else {
        return { a.h, L, a.gen_m, a.prop_m };
    }
}

template <bool MIXED>
__device__ __forceinline__ bool bind_plain(uint8_t* smem, const TableSrc& ts, unsigned* err, GravSmem& g)
{
    const bool ok = stage_to_smem(smem + 128, ts.src, ts.bytes, reinterpret_cast<uint64_t*>(smem), err, ts.wait_spins);
    g.L = ts.L;
    g.Lt = ts.L;
    g.radius = ts.radius;
    g.gm = ts.gm;
    g.t64 = reinterpret_cast<const GravEntry64*>(smem + 128);
    g.t32 = reinterpret_cast<const GravEntry32*>(smem + 128 + ts.off32);
    return ok;
}

// Rotations of gravity_gcrs for objects of different epochs.
__device__ __forceinline__ void to_itrs(const double* __restrict__ M, const double (&r)[3], double& x,
    double& y, double& z)
{
    x = __ldg(M + 0) * r[0] + __ldg(M + 1) * r[1] + __ldg(M + 2) * r[2];
    y = __ldg(M + 3) * r[0] + __ldg(M + 4) * r[1] + __ldg(M + 5) * r[2];
    z = __ldg(M + 6) * r[0] + __ldg(M + 7) * r[1] + __ldg(M + 8) * r[2];
}
__device__ __forceinline__ void to_gcrs(const double* __restrict__ M, double x, double y, double z, double (&a)[3])
{
    a[0] = __ldg(M + 0) * x + __ldg(M + 3) * y + __ldg(M + 6) * z;
    a[1] = __ldg(M + 1) * x + __ldg(M + 4) * y + __ldg(M + 7) * z;
    a[2] = __ldg(M + 2) * x + __ldg(M + 5) * y + __ldg(M + 8) * z;
}

// ---- RK8 ----
// Chain 0 of an object runs columns 4 -> 8, chain 1 columns 4 -> 0; K objects in lockstep. eval(M, r, acc)
// evaluates the K objects, keep.put/get hold the stage accelerations, put(...) writes a value of an
// object to the state and stage(...) a stage's position (one lane of its group each).
template <int K, class Eval, class Keep, class Put, class Stage>
__device__ __forceinline__ void rk8_chain(int chain, double h, const double* gen_m, double (&r)[K][3],
    double (&v)[K][3], const Eval& eval, const Keep& keep, const Put& put, const Stage& stage)
{
    const double hh = chain == 0 ? h : -h;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (chain == 0) {
                put(k, kSr + 4 * 3 + j, r[k][j]);
                put(k, kSv4 + j, v[k][j]);
            }
    for (int i = 1; i <= 4; ++i) {
        const int s = chain == 0 ? i - 1 : -i; // ForceModel::ComputeGenerationAcceleration
        for (int st = 0; st <= 9; ++st) {
            double t[K][3], acc[K][3];
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    double q = 0.0;
                    for (int p = 0; p < st - 1; ++p)
                        q = fma(c_rkn.a[st][p], keep.get(p, k, j), q);
                    t[k][j] = fma(hh, fma(c_rkn.c[st], v[k][j], hh * q), r[k][j]);
                    stage(k, (s + 4) * 10 + st, j, t[k][j]);
                }
            eval(gen_m + (size_t)((s + 4) * 10 + st) * 9, t, acc);
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    keep.put(st, k, j, acc[k][j]);
                    if (chain == 0 && st == 0) // column 3 + i: its own epoch and position
                        put(k, kHist + (3 + i) * 3 + j, acc[k][j]);
                }
            keep.sync();
        }
        const int col = chain == 0 ? 4 + i : 4 - i;
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                double sx = 0.0, sv = 0.0;
                for (int p = 0; p < 9; ++p) {
                    const double a = keep.get(p, k, j);
                    sx = fma(c_rkn.b[p], a, sx);
                    sv = fma(c_RKB[p], a, sv);
                }
                sv = fma(c_RKB[9], keep.get(9, k, j), sv);
                r[k][j] = fma(hh, fma(hh, sx, v[k][j]), r[k][j]);
                v[k][j] = fma(hh, sv, v[k][j]);
                put(k, kSr + col * 3 + j, r[k][j]);
                if (chain == 0)
                    put(k, kSv + (col - 5) * 3 + j, v[k][j]);
            }
        keep.sync(); // the sums are read before the next step's first stage
    }
}

// Initial state of an object; states gravity cannot take are flagged (the object runs all the same).
__device__ __forceinline__ void initial_state(const StartupArgs& a, int64_t o, double (&r)[3], double (&v)[3],
    bool flag)
{
    bool usable = true;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        r[j] = a.r0[o * 3 + j];
        v[j] = a.v0[o * 3 + j];
        usable = usable && isfinite(r[j]) && isfinite(v[j]);
    }
    if (r[0] == 0.0 && r[1] == 0.0 && r[2] == 0.0)
        usable = false;
    if (a.check && flag && !usable && a.err)
        atomicOr(a.err, kErrBadInput);
}

// The lists of the corrector passes start empty, also where a block gives up on its table.
__device__ __forceinline__ void clear_counters(const StartupArgs& a)
{
    if (blockIdx.x == 0)
        for (int i = (int)threadIdx.x; i < kStartupCounters; i += (int)blockDim.x)
            a.counters[i] = 0;
}

// Stage accelerations in the thread's local memory.
template <int K> struct KeepLocal {
    double (*q)[K][3];
    __device__ __forceinline__ double get(int p, int k, int j) const { return q[p][k][j]; }
    __device__ __forceinline__ void put(int p, int k, int j, double x) const { q[p][k][j] = x; }
    __device__ __forceinline__ void sync() const {}
};

template <bool MIXED, int K, bool BATCH>
__global__ void __launch_bounds__(256, 1) startup_rk8_kernel(TableSrc ts, StartupArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    clear_counters(a);
    GravSmem g;
    if (!bind_plain<MIXED>(smem, ts, a.err, g))
        return;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t half = (a.n + K - 1) / K; // threads of a chain; object k of thread t is t + k half
    if (t >= 2 * half)
        return;
    const int chain = t >= half;
    int64_t obj[K];
    bool live[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int64_t o = (chain ? t - half : t) + k * half;
        live[k] = o < a.n;
        obj[k] = live[k] ? o : a.n - 1;
    }
    const ObjSrc src = source<BATCH>(a, obj[0], ts.L);
    g.L = src.L;
    double r[K][3], v[K][3], kept[10][K][3];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        initial_state(a, obj[k], r[k], v[k], live[k] && chain == 0);
        if (live[k] && chain == 0)
            reinterpret_cast<int*>(a.state + (size_t)kSflag * a.n)[obj[k]] = 0;
    }
    auto eval = [&](const double* M, const double (&p)[K][3], double (&acc)[K][3]) {
        gravity_gcrs<MIXED, K>(g, M, p, acc);
    };
    auto put = [&](int k, int slot, double x) {
        if (live[k])
            a.state[(size_t)slot * a.n + obj[k]] = x;
    };
    auto stage = [&](int k, int i, int j, double x) {
        if (a.stage_pos && live[k])
            a.stage_pos[((size_t)i * 3 + j) * a.n + obj[k]] = x;
    };
    rk8_chain<K>(chain, src.h, src.gen_m, r, v, eval, KeepLocal<K> { kept }, put, stage);
}

// Stage accelerations of a lane group in shared memory, written by its first lane.
template <class Team> struct KeepShared {
    double* q; // this group's 30
    const Team& team;
    __device__ __forceinline__ double get(int p, int, int j) const { return q[p * 3 + j]; }
    __device__ __forceinline__ void put(int p, int, int j, double x) const
    {
        if (team.l == 0)
            q[p * 3 + j] = x;
    }
    __device__ __forceinline__ void sync() const { team.sync(); }
};

template <bool MIXED, bool WARPS, bool BATCH>
__global__ void __launch_bounds__(256, 1) startup_rk8_team_kernel(TableSrc ts, StartupArgs a, int P)
{
    extern __shared__ __align__(128) uint8_t smem[];
    clear_counters(a);
    GravSmem g;
    if (!bind_lane_table(smem, ts, a.err, g))
        return;
    const int in_block = (int)threadIdx.x / P;
    const int64_t grp = (int64_t)blockIdx.x * (blockDim.x / P) + in_block;
    if (grp >= 2 * a.n)
        return; // whole groups leave
    // 30 doubles of stages per group, then 8 per warp of a group of warps for its sums
    double* own = reinterpret_cast<double*>(smem + stage_offset(ts)) + (size_t)in_block * (30 + (WARPS ? P / 4 : 0));
    const auto team = make_team<WARPS>(P, own + 30);
    const int chain = grp >= a.n;
    const int64_t o = chain ? grp - a.n : grp;
    const ObjSrc src = source<BATCH>(a, o, ts.L);
    g.L = src.L;
    double r[1][3], v[1][3];
    initial_state(a, o, r[0], v[0], chain == 0 && team.l == 0);
    if (team.l == 0 && chain == 0)
        reinterpret_cast<int*>(a.state + (size_t)kSflag * a.n)[o] = 0;
    auto eval = [&](const double* M, const double (&p)[1][3], double (&acc)[1][3]) {
        gravity_gcrs_team<MIXED, 1, !MIXED && !WARPS>(g, team, M, p, acc);
    };
    auto put = [&](int, int slot, double x) {
        if (team.l == 0)
            a.state[(size_t)slot * a.n + o] = x;
    };
    using Team = typename TeamOf<WARPS>::type;
    auto stage = [&](int, int i, int j, double x) {
        if (a.stage_pos && team.l == 0)
            a.stage_pos[((size_t)i * 3 + j) * a.n + o] = x;
    };
    rk8_chain<1>(chain, src.h, src.gen_m, r, v, eval, KeepShared<Team> { own, team }, put, stage);
}

// ---- accelerations of columns ----
// pass < 0: columns 0..3 and 8 of every object (the RK8 chain left 4..7); else the list of that pass.
struct EvalItems {
    const StartupArgs& a;
    int pass;
    int64_t count;
    __device__ __forceinline__ EvalItems(const StartupArgs& args, int p)
        : a(args)
        , pass(p)
        , count(p < 0 ? 5 * args.n : (int64_t)args.counters[p])
    {
    }
    __device__ __forceinline__ void at(int64_t i, int64_t& o, int& col) const
    {
        if (pass < 0) {
            const int c = (int)(i / a.n);
            o = i - (int64_t)c * a.n;
            col = c == 4 ? 8 : c;
        } else {
            const unsigned e = reinterpret_cast<const unsigned*>(a.state)[i];
            o = e >> 3;
            const int c = (int)(e & 7u);
            col = c < 4 ? c : c + 1; // column 4 is never listed
        }
    }
};

template <bool MIXED, int K, bool BATCH>
__global__ void __launch_bounds__(256, 1) startup_eval_kernel(TableSrc ts, StartupArgs a, int pass)
{
    extern __shared__ __align__(128) uint8_t smem[];
    const EvalItems items(a, pass);
    const int64_t half = (items.count + K - 1) / K, T = (int64_t)gridDim.x * blockDim.x;
    if ((int64_t)blockIdx.x * blockDim.x >= half)
        return; // nothing for this block: it stages nothing
    GravSmem g;
    if (!bind_plain<MIXED>(smem, ts, a.err, g))
        return;
    const size_t n = (size_t)a.n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < half; t += T) {
        int64_t o[K];
        int col[K];
        bool live[K];
        const double* M[K];
        double x[K], y[K], z[K], ax[K], ay[K], az[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            live[k] = t + k * half < items.count;
            items.at(live[k] ? t + k * half : t, o[k], col[k]);
            const ObjSrc src = source<BATCH>(a, o[k], ts.L);
            if (k == 0)
                g.L = src.L;
            M[k] = src.prop_m + (size_t)col[k] * 9;
            double r[3];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                r[j] = a.state[(kSr + col[k] * 3 + j) * n + o[k]];
            to_itrs(M[k], r, x[k], y[k], z[k]);
        }
        gravity_itrs<MIXED, K>(g, x, y, z, ax, ay, az);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double acc[3];
            to_gcrs(M[k], ax[k], ay[k], az[k], acc);
            if (live[k])
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    a.state[(kHist + col[k] * 3 + j) * n + o[k]] = acc[j];
        }
    }
}

template <bool MIXED, bool WARPS, bool BATCH>
__global__ void __launch_bounds__(256, 1) startup_eval_team_kernel(TableSrc ts, StartupArgs a, int pass, int P)
{
    extern __shared__ __align__(128) uint8_t smem[];
    const EvalItems items(a, pass);
    const int per = (int)blockDim.x / P, in_block = (int)threadIdx.x / P;
    if ((int64_t)blockIdx.x * per >= items.count)
        return;
    GravSmem g;
    if (!bind_lane_table(smem, ts, a.err, g))
        return;
    const auto team = make_team<WARPS>(P,
        reinterpret_cast<double*>(smem + stage_offset(ts)) + (size_t)in_block * (WARPS ? P / 4 : 0));
    const size_t n = (size_t)a.n;
    for (int64_t i = (int64_t)blockIdx.x * per + in_block; i < items.count; i += (int64_t)gridDim.x * per) {
        int64_t o;
        int col;
        items.at(i, o, col);
        const ObjSrc src = source<BATCH>(a, o, ts.L);
        g.L = src.L;
        double r[1][3], acc[1][3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
            r[0][j] = a.state[(kSr + col * 3 + j) * n + o];
        gravity_gcrs_team<MIXED, 1, !MIXED && !WARPS>(g, team, src.prop_m + (size_t)col * 9, r, acc);
        if (team.l == 0)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                a.state[(kHist + col * 3 + j) * n + o] = acc[0][j];
    }
}

// ---- corrector ----
// Corrector pass `it` of every object that is not done: lists the columns whose accelerations the next
// evaluation must renew. The rule is correct_position's, over the eight columns at once:
// - no column's position moves by a bit: every further pass would repeat this one, done;
// - the passes left would not converge (the change of the last one, followed with J through all of them,
//   is above the last bits) or a column is below the model's radius: the plain pass;
// - else the fixed point of the passes under a + J y; columns within `near` of it take a + J y for their
//   acceleration, the others are evaluated there.
template <bool BATCH> __global__ void __launch_bounds__(128) startup_correct_kernel(CorrModel cm, StartupArgs a, int it)
{
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= a.n)
        return;
    const size_t n = (size_t)a.n;
    int* flags = reinterpret_cast<int*>(a.state + (size_t)kSflag * n);
    int flag = flags[o];
    double* st = a.state + o;
    double* before = a.pass_pos ? a.pass_pos + (size_t)it * 27 * n + o : nullptr;
    if (flag & kFlagDone) { // the passes left repeat the last one
        if (before && !(flag & kFlagFast))
            for (int i = 0; i < 27; ++i)
                before[i * n] = st[(kSr + i) * n];
        return;
    }
    const double h = source<BATCH>(a, o, 0).h;
    double acc[9][3], pos[9][3], v4[3];
    for (int c = 0; c < 9; ++c)
        for (int j = 0; j < 3; ++j) {
            acc[c][j] = st[(kHist + c * 3 + j) * n];
            pos[c][j] = st[(kSr + c * 3 + j) * n];
        }
    for (int j = 0; j < 3; ++j)
        v4[j] = st[(kSv4 + j) * n];
    PassResult p;
    corrector_pass(h, acc, pos[4], v4, p);
    unsigned moved = 0;
    float d[9][3];
    for (int c = 0; c < 9; ++c)
        for (int j = 0; j < 3; ++j) {
            d[c][j] = 0.f;
            if (c == 4)
                continue;
            if (!same_bits(p.r[c][j], pos[c][j]))
                moved |= 1u << c;
            d[c][j] = (float)(p.r[c][j] - pos[c][j]);
        }
    unsigned todo = moved;
    if (moved) {
        CorrJacobian jac[9];
        bool high = true;
        float len = 3.4e38f;
        for (int c = 0; c < 9; ++c) {
            jac[c] = CorrJacobian(cm, pos[c]);
            high = high && jac[c].len >= cm.low;
            len = fminf(len, jac[c].len);
        }
        const float h2 = (float)(h * h);
        float y[9][3];
        for (int c = 0; c < 9; ++c)
            for (int j = 0; j < 3; ++j)
                y[c][j] = d[c][j];
        // the passes after this one, as the linear map y -> d + h^2 (S and GJ rows) J y
        float change = 0.f;
        const int left = a.ncorr - 1 - it;
        for (int q = 0; q < left && q < 12 && high && (it == 0 || (flag & kFlagFast)); ++q) {
            float da[9][3];
            for (int c = 0; c < 9; ++c)
                jac[c].apply(y[c], da[c]);
            change = 0.f;
            for (int c = 0; c < 9; ++c) {
                if (c == 4)
                    continue;
                for (int j = 0; j < 3; ++j) {
                    float t = 0.f;
                    for (int k = 0; k < 9; ++k)
                        if (k != 4)
                            t = fmaf((float)c_GJ[c][k] + c_pass.m[c][k], da[k][j], t);
                    t = fmaf(h2, t, d[c][j]);
                    change = fmaxf(change, fabsf(t - y[c][j]));
                    y[c][j] = t;
                }
            }
        }
        if (it == 0 && high && a.ncorr > 2 && change <= 0x1p-54f * len)
            flag |= kFlagFast;
        if (flag & kFlagFast) {
            todo = 0;
            double ac[9][3];
            for (int c = 0; c < 9; ++c) {
                float da[3];
                jac[c].apply(y[c], da);
                const float m = fmaxf(fmaxf(fabsf(y[c][0]), fabsf(y[c][1])), fabsf(y[c][2]));
                if (!(m <= cm.near * jac[c].len))
                    todo |= 1u << c;
                for (int j = 0; j < 3; ++j)
                    ac[c][j] = acc[c][j] + (double)da[j];
            }
            todo &= ~(1u << 4);
            corrector_pass(h, ac, pos[4], v4, p);
            for (int c = 0; c < 9; ++c)
                for (int j = 0; j < 3; ++j)
                    if (c != 4)
                        st[(kHist + c * 3 + j) * n] = ac[c][j];
        }
    }
    if (before && !(flag & kFlagFast))
        for (int i = 0; i < 27; ++i)
            before[i * n] = pos[i / 3][i % 3];
    else if (before && it == 0)
        before[0] = __longlong_as_double(0x7ff8000000000000ll);
    for (int j = 0; j < 3; ++j) {
        for (int c = 0; c < 9; ++c)
            if (c != 4)
                st[(kSr + c * 3 + j) * n] = p.r[c][j];
        for (int c = 0; c < 4; ++c)
            st[(kSv + c * 3 + j) * n] = p.v[c][j];
        st[(kSs + j) * n] = p.s8[j];
        st[(kSb + j) * n] = p.S8[j];
    }
    if (!todo)
        flag |= kFlagDone;
    flags[o] = flag;
    if (todo) {
        unsigned* list = reinterpret_cast<unsigned*>(a.state);
        int at = atomicAdd(a.counters + it, __popc(todo));
        for (int c = 0; c < 9; ++c)
            if (todo >> c & 1)
                list[at++] = (unsigned)o * 8u + (unsigned)(c < 4 ? c : c - 1);
    }
}

// The propagation's state from the startup's matrices (GpuPropagator::Step at step 1,
// gpu_propagator.cu:31-47, and the replay of steps 1..4, CopyStartupStateKernel).
__global__ void __launch_bounds__(128) startup_finish_kernel(StartupArgs a)
{
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= a.n)
        return;
    const size_t n = (size_t)a.n;
    double* st = a.state + o;
    const bool fix_q3 = (a.flags & 2u) != 0;
    double r[4][3], v[4][3], e[4][3];
    if (a.col_pos)
        for (int i = 0; i < 27; ++i)
            a.col_pos[(size_t)i * n + o] = st[(kSr + i) * n];
    for (int k = 0; k < 4; ++k)
        for (int j = 0; j < 3; ++j) {
            r[k][j] = st[(kSr + (5 + k) * 3 + j) * n];
            v[k][j] = st[(kSv + k * 3 + j) * n];
            e[k][j] = st[(kHist + (fix_q3 ? 5 + k : 8) * 3 + j) * n];
        }
    for (int j = 0; j < 3; ++j) {
        st[(kR + j) * n] = r[3][j];
        st[(kV + j) * n] = v[3][j];
        for (int k = 0; k < 4; ++k) {
            st[(kRep + k * 6 + j) * n] = r[k][j];
            st[(kRep + k * 6 + 3 + j) * n] = v[k][j];
            st[(kRepA + k * 3 + j) * n] = e[k][j];
        }
    }
}

// ---- launch ----
template <class Kern> cudaError_t smem_of(Kern kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Lanes per evaluation of `items` independent evaluations: the warps that hold a column per lane while
// every SM has at most one such group, else the most lanes (<= 32) that leave one block of 256 threads
// (255 registers: at 168 the walk waits on its table loads, 1.7 times as long) per SM; 0 where one evaluation per thread (plain kernels) is the better walk.
struct TeamShape {
    int P = 0; // threads per group (0: plain kernels)
    bool warps = false;
};
TeamShape team_shape(int64_t items, int L, int num_sms)
{
    TeamShape t;
    const int W = (L + 32) / 32;
    if (W > 1 && items <= num_sms) {
        t.P = 32 * W;
        t.warps = true;
        return t;
    }
    if (items > (int64_t)num_sms * 96)
        return t;
    t.P = 2;
    while (t.P < 32 && items * 2 * t.P <= (int64_t)num_sms * 256)
        t.P *= 2;
    return t;
}
// Threads per block and blocks for `items` groups of P threads, at least a warp.
void team_grid(int64_t items, int P, int num_sms, int& block, unsigned& grid)
{
    const int64_t per_sm = (items + num_sms - 1) / num_sms;
    const int64_t groups = std::max<int64_t>(std::max(1, 32 / P), std::min<int64_t>(per_sm, 256 / P));
    block = (int)groups * P;
    grid = (unsigned)((items + groups - 1) / groups);
}

// The team kernels take the precision of the lane table, the others MIXED.
template <bool MIXED, bool BATCH>
cudaError_t launch_rk8(const TableSrc& plain, const TableSrc& lanes, const StartupArgs& a, int num_sms, cudaStream_t s)
{
    const TeamShape t = team_shape(2 * a.n, lanes.L, num_sms);
    cudaError_t e;
    if (t.P > 0) {
        int block;
        unsigned grid;
        team_grid(2 * a.n, t.P, num_sms, block, grid);
        const size_t bytes = stage_offset(lanes) + (size_t)(block / t.P) * (30 + (t.warps ? t.P / 4 : 0)) * 8;
        if (bytes <= max_smem_optin()) {
            auto launch = [&](auto kernel) {
                if ((e = smem_of(kernel, bytes)) != cudaSuccess)
                    return e;
                kernel<<<grid, block, bytes, s>>>(lanes, a, t.P);
                return cudaGetLastError();
            };
            if (lanes.mixed)
                return t.warps ? launch(startup_rk8_team_kernel<true, true, BATCH>)
                               : launch(startup_rk8_team_kernel<true, false, BATCH>);
            return t.warps ? launch(startup_rk8_team_kernel<false, true, BATCH>)
                           : launch(startup_rk8_team_kernel<false, false, BATCH>);
        }
    }
    // two objects per thread where that still leaves a block of four warps per SM
    const size_t bytes = table_smem_bytes(plain);
    if (!BATCH && a.n >= (int64_t)num_sms * 128) {
        const LaunchShape ls = pick_shape(2 * ((a.n + 1) / 2), 256, num_sms);
        if ((e = smem_of(startup_rk8_kernel<MIXED, 2, false>, bytes)) != cudaSuccess)
            return e;
        startup_rk8_kernel<MIXED, 2, false><<<ls.grid, ls.block, bytes, s>>>(plain, a);
    } else {
        const LaunchShape ls = pick_shape(2 * a.n, 256, num_sms);
        if ((e = smem_of(startup_rk8_kernel<MIXED, 1, BATCH>, bytes)) != cudaSuccess)
            return e;
        startup_rk8_kernel<MIXED, 1, BATCH><<<ls.grid, ls.block, bytes, s>>>(plain, a);
    }
    return cudaGetLastError();
}

template <bool MIXED, bool BATCH>
cudaError_t launch_eval(const TableSrc& plain, const TableSrc& lanes, const StartupArgs& a, int pass, int num_sms,
    cudaStream_t s)
{
    const int64_t items = (pass < 0 ? 5 : 8) * a.n;
    const TeamShape t = team_shape(items, lanes.L, num_sms);
    cudaError_t e;
    if (t.P > 0) {
        int block;
        unsigned grid;
        team_grid(items, t.P, num_sms, block, grid);
        const size_t bytes = stage_offset(lanes) + (t.warps ? (size_t)(block / t.P) * (t.P / 4) * 8 : 0);
        auto launch = [&](auto kernel) {
            if ((e = smem_of(kernel, bytes)) != cudaSuccess)
                return e;
            kernel<<<grid, block, bytes, s>>>(lanes, a, pass, t.P);
            return cudaGetLastError();
        };
        if (lanes.mixed)
            return t.warps ? launch(startup_eval_team_kernel<true, true, BATCH>)
                           : launch(startup_eval_team_kernel<true, false, BATCH>);
        return t.warps ? launch(startup_eval_team_kernel<false, true, BATCH>)
                       : launch(startup_eval_team_kernel<false, false, BATCH>);
    }
    const size_t bytes = table_smem_bytes(plain);
    if (!BATCH && items >= (int64_t)num_sms * 384) {
        const unsigned grid = (unsigned)std::min<int64_t>(num_sms, ((items + 1) / 2 + 255) / 256);
        if ((e = smem_of(startup_eval_kernel<MIXED, 2, false>, bytes)) != cudaSuccess)
            return e;
        startup_eval_kernel<MIXED, 2, false><<<grid, 256, bytes, s>>>(plain, a, pass);
    } else {
        const unsigned grid = (unsigned)std::min<int64_t>(num_sms, (items + 255) / 256);
        if ((e = smem_of(startup_eval_kernel<MIXED, 1, BATCH>, bytes)) != cudaSuccess)
            return e;
        startup_eval_kernel<MIXED, 1, BATCH><<<grid, 256, bytes, s>>>(plain, a, pass);
    }
    return cudaGetLastError();
}

template <bool MIXED, bool BATCH>
cudaError_t run(const TableSrc& plain, const TableSrc& lanes, const StartupArgs& a, int num_sms, cudaStream_t s)
{
    cudaError_t e;
    if ((e = launch_rk8<MIXED, BATCH>(plain, lanes, a, num_sms, s)) != cudaSuccess
        || (e = launch_eval<MIXED, BATCH>(plain, lanes, a, -1, num_sms, s)) != cudaSuccess)
        return e;
    const unsigned blocks = (unsigned)((a.n + 127) / 128);
    for (int it = 0; it < a.ncorr; ++it) {
        startup_correct_kernel<BATCH><<<blocks, 128, 0, s>>>(plain.corr, a, it);
        if ((e = cudaGetLastError()) != cudaSuccess
            || (e = launch_eval<MIXED, BATCH>(plain, lanes, a, it, num_sms, s)) != cudaSuccess)
            return e;
    }
    startup_finish_kernel<<<blocks, 128, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_startup_gravity(const TableSrc& plain, const TableSrc& lanes, const StartupArgs& a,
    int num_sms, cudaStream_t s)
{
    if (a.n <= 0)
        return cudaSuccess;
    if (a.reqs)
        return plain.mixed ? run<true, true>(plain, lanes, a, num_sms, s) : run<false, true>(plain, lanes, a, num_sms, s);
    return plain.mixed ? run<true, false>(plain, lanes, a, num_sms, s) : run<false, false>(plain, lanes, a, num_sms, s);
}

} // namespace gpop
