// variational.cu -- forward variational equations (6x6 STM), the adjoint (reverse sweep) of the
// GJ8 propagation, and the closest approach of listed pairs with miss-distance seeds.
//
// Tangents and adjoints are the derivatives of the discrete map of the forward propagation (startup, GJ8
// steps: gpu_propagator.cu:28-119) with one simplification: the Jacobian of a step's corrector passes is
// taken once, at the position of the last evaluation (the corrector converges, so the passes' iterates differ by
// far less than the truncation error); of the startup's passes likewise where they converge, else in front of each
// (pass_tangent_kernel). Forward tangents and the reverse sweep make the same choice, so they are exact transposes of
// each other. With few passes the last evaluation is not at the step's position: found from its acceleration
// (evaluation_point). Transition matrices of 40 steps of 120 s against differences in long double, largest error of a
// block with 1, 2 and 3 passes: with one Jacobian per step and column at the last positions 7e-7, 9e-9 and 2e-10,
// with those of the evaluations 1.1e-13, 7e-10 and 7e-13.
//
// The Jacobians depend on the positions alone, not on the tangents. So the forward propagation runs with
// the propagation's own kernels and keeps its positions (per step, and of the startup's 80 stages and nine
// columns); one kernel makes all the Jacobians, a (point, object) per thread with the table read by
// broadcast; and the tangents or the adjoint follow as short linear recurrences, a thread per direction or
// unit. One kernel of 8 lanes per object that walked primal, Jacobian and tangents in turn (and ran the
// segments of the reverse sweep twice) measured, with the corrector's early end: 1,000 STMs over 360 steps
// 43.8 ms, 1,200 miss gradients over 720 steps 75 ms for the sweep alone; now the Jacobians take 2.0 and 4.4 ms
// (bound by the FP64 pipe) and the recurrences 0.18 and 0.53 ms.
//
// Adjoint of one GJ8 step n (K = number of corrector passes, iterates r(0..K-1), a(i) = f(r(i))):
//   S' = S + s + h8/2,  r(0) = h^2 (sum_c GJ[9][c] h_c + S'),  s1 = sum_c SA[8][c] h_(c+1),
//   s2 = sum_c GJ[8][c] h_(c+1),  r(i+1) = h^2 (s2 + GJ[8][8] a(i) + S'),
//   s_n = s + (a(K-1) + h8)/2,  v_n = h (s1 + SA[8][8] a(K-1) + s_n),  history <- (h_1..h_8, a(K-1)).
// The reverse pass below applies the transposes of these maps in the opposite order.
#include "common.cuh"
#include "gj8_tables.cuh"
#include "hermite.cuh"
#include "integrator.cuh"
#include "jacobian.cuh"
#include "variational.cuh"

#include <algorithm>

namespace gpop {

namespace {

__device__ __forceinline__ bool bind_plain64(uint8_t* smem, const TableSrc& ts, unsigned* err, GravSmem& g)
{
    const bool ok = stage_to_smem(smem + 128, ts.src, ts.bytes, reinterpret_cast<uint64_t*>(smem), err, ts.wait_spins);
    g.L = ts.L;
    g.Lt = ts.L;
    g.radius = ts.radius;
    g.gm = ts.gm;
    g.t64 = reinterpret_cast<const GravEntry64*>(smem + 128);
    g.t32 = nullptr;
    return ok;
}

} // namespace

// Moves r to where gravity, with Jacobian J, is larger by d. False, with r as it was, where that is at rounding
// (2^-46 of r: a converged corrector, some 1e-15) or not near. J has no trace, so it is far from singular.
__device__ __forceinline__ bool evaluation_point(const double (&J)[3][3], const double (&d)[3], double (&r)[3])
{
    double x[3], c0[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) { // cofactors of column j
        const int k = (j + 1) % 3, l = (j + 2) % 3;
        double c[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            c[i] = J[(i + 1) % 3][k] * J[(i + 2) % 3][l] - J[(i + 2) % 3][k] * J[(i + 1) % 3][l];
        x[j] = c[0] * d[0] + c[1] * d[1] + c[2] * d[2];
        if (j == 0)
            for (int i = 0; i < 3; ++i)
                c0[i] = c[i];
    }
    const double det = fabs(c0[0] * J[0][0] + c0[1] * J[1][0] + c0[2] * J[2][0]);
    const double move = fmax(fmax(fabs(x[0]), fabs(x[1])), fabs(x[2]));
    const double size = fmax(fmax(fabs(r[0]), fabs(r[1])), fabs(r[2])) * det;
    if (!(move > 0x1p-46 * size) || !(move < 0x1p-4 * size))
        return false;
    const double inv = 1.0 / (c0[0] * J[0][0] + c0[1] * J[1][0] + c0[2] * J[2][0]);
#pragma unroll
    for (int j = 0; j < 3; ++j)
        r[j] = fma(x[j], inv, r[j]);
    return true;
}

// ---- Jacobians of many points ----
__global__ void __launch_bounds__(256, 1) jac_points_kernel(TableSrc ts, JacPoints a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    GravSmem g;
    if (!bind_plain64(smem, ts, a.err, g))
        return;
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.total; t += T) {
        int64_t i, u;
        if (a.offset) { // the item whose range holds t
            int lo = 0, hi = a.items - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (a.offset[mid] <= t)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            i = lo;
            u = t - a.offset[lo];
        } else {
            i = t / a.width;
            u = t - i * a.width;
        }
        const int64_t o = a.obj ? a.obj[u] : u;
        if (a.mark && isnan(a.mark[o]))
            continue;
        const double* M = a.M + (size_t)(a.frames ? i % a.frames : i) * 9;
        double r[3], acc[3], J[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
            r[j] = a.pos[(i * 3 + j) * a.n + o];
#pragma unroll 1
        for (int it = 0;; ++it) {
            gravity_jac_gcrs<false>(g, 0, 1, M, r, acc, J, 0u);
            if (!a.acc || it == 4)
                break;
            double d[3];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                d[j] = a.acc[(i * 3 + j) * a.n + o] - acc[j];
            if (!evaluation_point(J, d, r))
                break;
        }
#pragma unroll
        for (int k = 0; k < 9; ++k)
            a.jac[(int64_t)k * a.total + t] = J[k / 3][k % 3];
    }
}

namespace {

__device__ __forceinline__ void load_jac(const double* __restrict__ jac, int64_t total, int64_t t, double (&J)[3][3])
{
#pragma unroll
    for (int k = 0; k < 9; ++k)
        J[k / 3][k % 3] = __ldg(jac + (int64_t)k * total + t);
}

__device__ __forceinline__ void mul(const double (&J)[3][3], const double (&x)[3], double (&y)[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
        y[i] = J[i][0] * x[0] + J[i][1] * x[1] + J[i][2] * x[2];
}

} // namespace

// ---- startup tangents ----
// RK8 (gpu_startup.cu:108-144) of direction dir and chain: thread t = ((chain 6 + dir) n + o). The stage
// states as in rk8_step; the columns' position tangents go to out slot (col 3 + j).
__global__ void __launch_bounds__(128) rk8_tangent_kernel(StartupTangentArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 12 * a.n)
        return;
    const int64_t n = a.n, o = t % n;
    const int cd = (int)(t / n), chain = cd / 6, dir = cd % 6;
    const double hh = chain == 0 ? a.h : -a.h;
    double r[3], v[3], Kx[10][3], Kv[10][3];
    for (int j = 0; j < 3; ++j) {
        r[j] = dir == j ? 1.0 : 0.0;
        v[j] = dir == 3 + j ? 1.0 : 0.0;
        if (chain == 0)
            a.out[((int64_t)(4 * 3 + j) * 6 + dir) * n + o] = r[j];
    }
    for (int i = 1; i <= 4; ++i) {
        const int s = chain == 0 ? i - 1 : -i;
        for (int k = 0; k < 10; ++k) {
            double x[3];
            for (int j = 0; j < 3; ++j) {
                double sx = 0.0, sv = 0.0;
                for (int p = 0; p < k; ++p) {
                    sx = fma(c_RKA[k - 1][p], Kx[p][j], sx);
                    sv = fma(c_RKA[k - 1][p], Kv[p][j], sv);
                }
                x[j] = fma(hh, sx, r[j]);
                Kx[k][j] = fma(hh, sv, v[j]);
            }
            double J[3][3];
            load_jac(a.stage_jac, 80 * n, (int64_t)((s + 4) * 10 + k) * n + o, J);
            mul(J, x, Kv[k]);
        }
        const int col = chain == 0 ? 4 + i : 4 - i;
        for (int j = 0; j < 3; ++j) {
            double sx = 0.0, sv = 0.0;
            for (int k = 0; k < 10; ++k) {
                sx = fma(Kx[k][j], c_RKB[k], sx);
                sv = fma(Kv[k][j], c_RKB[k], sv);
            }
            v[j] = fma(hh, sv, v[j]);
            r[j] = fma(hh, sx, r[j]);
            a.out[((int64_t)(col * 3 + j) * 6 + dir) * n + o] = r[j];
        }
    }
}

// The mid-corrector of direction dir. Position tangents of the columns in out slots 0..26 become, at the end, those
// of the accelerations; 27..32 s and S of column 8, 33..44 and 45..56 positions and velocities of columns 5..8.
struct ColumnTangents {
    double* out;
    int64_t stride;
    double dr[9][3], da[9][3], r4[3], v4[3];
    PassResult p;
    __device__ __forceinline__ ColumnTangents(const StartupTangentArgs& a, int64_t t)
        : out(a.out + t)
        , stride(6 * a.n)
    {
        const int dir = (int)(t / a.n);
        for (int c = 0; c < 9; ++c)
            for (int j = 0; j < 3; ++j)
                dr[c][j] = slot(c * 3 + j);
        for (int j = 0; j < 3; ++j) {
            r4[j] = dir == j ? 1.0 : 0.0;
            v4[j] = dir == 3 + j ? 1.0 : 0.0;
        }
    }
    __device__ __forceinline__ double& slot(int k) const { return out[(int64_t)k * stride]; }
    __device__ __forceinline__ void accelerations(const double* jac, int64_t total, int64_t n, int64_t first)
    {
        for (int c = 0; c < 9; ++c) {
            double J[3][3];
            load_jac(jac, total, first + (int64_t)c * n, J);
            mul(J, dr[c], da[c]);
        }
    }
    // a pass; whether it left every position as it was
    __device__ __forceinline__ bool pass(double h)
    {
        corrector_pass(h, da, r4, v4, p);
        bool same = true;
        for (int c = 0; c < 9; ++c) {
            if (c == 4)
                continue;
            for (int j = 0; j < 3; ++j) {
                same = same && same_bits(dr[c][j], p.r[c][j]);
                dr[c][j] = p.r[c][j];
            }
        }
        return same;
    }
    __device__ __forceinline__ void put_end(const double (&x)[9][3]) const
    {
        for (int j = 0; j < 3; ++j) {
            for (int c = 0; c < 9; ++c)
                slot(c * 3 + j) = x[c][j];
            slot(27 + j) = p.s8[j];
            slot(30 + j) = p.S8[j];
            for (int k = 0; k < 4; ++k) {
                slot(33 + k * 3 + j) = dr[5 + k][j];
                slot(45 + k * 3 + j) = p.v[k][j];
            }
        }
    }
};

// Passes of the objects that take them one by one (few passes, long steps), each with the Jacobians in front of it.
__global__ void __launch_bounds__(128) pass_tangent_kernel(StartupTangentArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * a.n)
        return;
    const int64_t n = a.n, o = t % n;
    if (isnan(a.mark[o]))
        return;
    ColumnTangents q(a, t);
    for (int it = a.pass_lo; it < a.pass_hi; ++it) {
        q.accelerations(a.pass_jac, (int64_t)(a.pass_hi - a.pass_lo) * 9 * n, n, (int64_t)(it - a.pass_lo) * 9 * n + o);
        q.pass(a.h);
    }
    q.put_end(q.dr);
}

// The end: the accelerations at the last positions, behind the passes of the others, which have converged: one
// Jacobian per column serves them all.
__global__ void __launch_bounds__(128) corrector_tangent_kernel(StartupTangentArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * a.n)
        return;
    const int64_t n = a.n, o = t % n;
    ColumnTangents q(a, t);
    q.accelerations(a.col_jac, 9 * n, n, o);
    if (!isnan(a.mark[o])) {
        for (int c = 0; c < 9; ++c)
            for (int j = 0; j < 3; ++j)
                q.slot(c * 3 + j) = q.da[c][j];
        return;
    }
    for (int it = 0; it < a.ncorr; ++it) {
        const bool same = q.pass(a.h);
        q.accelerations(a.col_jac, 9 * n, n, o);
        if (same) // every further pass repeats this one
            break;
    }
    q.put_end(q.da);
}

// ---- forward variational equations: steps [step_lo, step_hi] of every (direction, object) ----
__global__ void __launch_bounds__(128) stm_sweep_kernel(StmArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = a.n, W = 6 * n;
    if (t >= W)
        return;
    const int64_t o = t % n;
    const int dir = (int)(t / n);
    const double h = a.h;
    double hist[9][3], s[3], S[3], r[3], v[3];
    double* st = a.sweep + t; // 39 arrays of 6 n: history, s, S, r, v
    if (a.first) {
        const double* T = a.startup + t;
        const int rep = a.steps < 4 ? a.steps : 4; // steps 1..4 replay the startup columns
        for (int j = 0; j < 3; ++j) {
            for (int c = 0; c < 9; ++c)
                hist[c][j] = T[(int64_t)(c * 3 + j) * W];
            s[j] = T[(int64_t)(27 + j) * W];
            S[j] = T[(int64_t)(30 + j) * W];
            r[j] = T[(int64_t)(33 + (rep - 1) * 3 + j) * W];
            v[j] = T[(int64_t)(45 + (rep - 1) * 3 + j) * W];
        }
    } else {
        for (int j = 0; j < 3; ++j) {
            for (int c = 0; c < 9; ++c)
                hist[c][j] = st[(int64_t)(c * 3 + j) * W];
            s[j] = st[(int64_t)(27 + j) * W];
            S[j] = st[(int64_t)(30 + j) * W];
            r[j] = st[(int64_t)(33 + j) * W];
            v[j] = st[(int64_t)(36 + j) * W];
        }
    }
    const int64_t total = (int64_t)(a.step_hi - a.step_lo + 1) * n;
    double Jn[3][3];
    if (a.step_lo <= a.step_hi)
        load_jac(a.jac, total, o, Jn);
    for (int step = a.step_lo; step <= a.step_hi; ++step) {
        double J[3][3];
#pragma unroll
        for (int k = 0; k < 9; ++k)
            J[k / 3][k % 3] = Jn[k / 3][k % 3];
        if (step < a.step_hi) // the next step's Jacobian loads during this step
            load_jac(a.jac, total, (int64_t)(step + 1 - a.step_lo) * n + o, Jn);
        double s1[3], s2[3], prev[3], a7[3], a8[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) { // as gj8_kernel
            double rt = 0.0;
#pragma unroll
            for (int c = 0; c < 9; ++c)
                rt = fma(hist[c][j], c_GJ[9][c], rt);
            S[j] += s[j] + hist[8][j] / 2;
            r[j] = (rt + S[j]) * h * h;
            double c1 = 0.0, c2 = 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                c1 = fma(hist[c + 1][j], c_SA[8][c], c1);
                c2 = fma(hist[c + 1][j], c_GJ[8][c], c2);
            }
            s1[j] = c1;
            s2[j] = c2;
            prev[j] = s[j];
            a7[j] = hist[8][j];
            a8[j] = 0.0;
        }
        for (int it = 0; it < a.ncorr; ++it) {
            mul(J, r, a8);
            bool same = true;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const double rn = h * h * (s2[j] + a8[j] * c_GJ[8][8] + S[j]);
                same = same && same_bits(rn, r[j]);
                r[j] = rn;
            }
            if (same) // every further pass repeats this one
                break;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            s[j] = prev[j] + (a8[j] + a7[j]) / 2;
            v[j] = h * (s1[j] + a8[j] * c_SA[8][8] + s[j]);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                hist[c][j] = hist[c + 1][j];
            hist[8][j] = a8[j];
        }
    }
    for (int j = 0; j < 3; ++j) {
        for (int c = 0; c < 9; ++c)
            st[(int64_t)(c * 3 + j) * W] = hist[c][j];
        st[(int64_t)(27 + j) * W] = s[j];
        st[(int64_t)(30 + j) * W] = S[j];
        st[(int64_t)(33 + j) * W] = r[j];
        st[(int64_t)(36 + j) * W] = v[j];
        if (a.last) {
            a.phi[(o * 6 + j) * 6 + dir] = r[j];
            a.phi[(o * 6 + 3 + j) * 6 + dir] = v[j];
        }
    }
}

// ---- adjoint: steps [step_lo, step_hi] of every unit, in reverse ----
// hb: history adjoints in logical order after the step on entry, before it on exit; sb, Sb: adjoints of
// s and S likewise. Units are in rank order (the latest last step first): at a step the ranks whose last
// step is not before it take part, and its Jacobians lie at offset[step - step_lo] + rank.
__global__ void __launch_bounds__(64) adjoint_sweep_kernel(AdjSweepArgs a)
{
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; // rank
    if (u >= a.n_units)
        return;
    const int64_t U = a.n_units, unit = a.unit ? a.unit[u] : u;
    const double h = a.h, h2 = h * h;
    const int k0 = a.seed_step0[unit];
    const int kend = min(k0 + 2, a.steps);
    const double* seeds = a.seeds + unit * 27;
    double hb[9][3], sb[3], Sb[3];
    double* st = a.sweep + u;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int c = 0; c < 9; ++c)
            hb[c][j] = a.first ? 0.0 : st[(c * 3 + j) * U];
        sb[j] = a.first ? 0.0 : st[(27 + j) * U];
        Sb[j] = a.first ? 0.0 : st[(30 + j) * U];
    }
    auto at = [&](int step) {
        const int i = step - a.step_lo;
        return a.offset ? a.offset[i] + u : (int64_t)i * U + u;
    };
    const int top = min(kend, a.step_hi);
    double Jn[3][3];
    if (top >= a.step_lo)
        load_jac(a.jac, a.total, at(top), Jn);
    for (int step = top; step >= a.step_lo; --step) {
        double J[3][3];
#pragma unroll
        for (int k = 0; k < 9; ++k)
            J[k / 3][k % 3] = Jn[k / 3][k % 3];
        if (step > a.step_lo) // the next Jacobian loads during this step
            load_jac(a.jac, a.total, at(step - 1), Jn);
        const int node = step - k0;
        const double* seed = (node >= 0 && node < 3) ? seeds + node * 9 : nullptr;
        double abar[3], s1b[3], s2b[3], Spb[3], prevb[3], a7b[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
            abar[j] = hb[8][j] + (seed ? seed[6 + j] : 0.0);
#pragma unroll
        for (int c = 8; c >= 1; --c)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                hb[c][j] = hb[c - 1][j];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            hb[0][j] = 0.0;
            const double rb = seed ? seed[j] : 0.0, vb = seed ? seed[3 + j] : 0.0;
            const double sK = sb[j] + h * vb; // s_n feeds v_n = h (s1 + SA88 a + s_n)
            s1b[j] = h * vb;
            abar[j] += h * c_SA[8][8] * vb + sK / 2;
            prevb[j] = sK;
            a7b[j] = sK / 2;
            s2b[j] = h2 * rb;
            abar[j] += h2 * c_GJ[8][8] * rb;
            Spb[j] = Sb[j] + h2 * rb;
        }
        for (int it = a.ncorr - 1; it >= 0; --it) {
            double rb[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                rb[k] = J[0][k] * abar[0] + J[1][k] * abar[1] + J[2][k] * abar[2];
            if (it >= 1) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    s2b[j] += h2 * rb[j];
                    Spb[j] += h2 * rb[j];
                    abar[j] = h2 * c_GJ[8][8] * rb[j];
                }
            } else {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
#pragma unroll
                    for (int c = 0; c < 9; ++c)
                        hb[c][j] += h2 * c_GJ[9][c] * rb[j];
                    Spb[j] += h2 * rb[j];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
                hb[c + 1][j] += c_SA[8][c] * s1b[j] + c_GJ[8][c] * s2b[j];
            hb[8][j] += a7b[j] + Spb[j] / 2; // a7 = h8, and S' = S + s + h8/2
            Sb[j] = Spb[j];
            sb[j] = prevb[j] + Spb[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int c = 0; c < 9; ++c)
            st[(c * 3 + j) * U] = hb[c][j];
        st[(27 + j) * U] = sb[j];
        st[(30 + j) * U] = Sb[j];
    }
}

// Gradient of the units whose object lies in [obj_lo, obj_lo + n): the startup's outputs along each
// initial-state direction, contracted with their adjoints. Thread t = rank 6 + dir.
__global__ void __launch_bounds__(128) adjoint_finish_kernel(AdjFinishArgs a)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 6 * a.n_units)
        return;
    const int64_t u = t / 6, U = a.n_units, unit = a.unit ? a.unit[u] : u;
    const int dir = (int)(t % 6);
    const int64_t o = a.unit_obj[unit] - a.obj_lo;
    if (o < 0 || o >= a.n)
        return;
    const double* T = a.startup + (int64_t)dir * a.n + o;
    const int64_t W = 6 * a.n;
    const double* st = a.sweep + u;
    double g = 0.0; // history, s and S adjoints are those of the step-5 inputs (zero if none)
    for (int j = 0; j < 3; ++j) {
        for (int c = 0; c < 9; ++c)
            g += st[(c * 3 + j) * U] * T[(int64_t)(c * 3 + j) * W];
        g += st[(27 + j) * U] * T[(int64_t)(27 + j) * W] + st[(30 + j) * U] * T[(int64_t)(30 + j) * W];
    }
    const bool fix_q3 = (a.flags & 2u) != 0;
    const int k0 = a.seed_step0[unit];
    for (int node = 0; node < 3; ++node) { // seeds on the replayed steps 1..4
        const int step = k0 + node;
        if (step < 1 || step > 4 || step > a.steps)
            continue;
        const double* sd = a.seeds + unit * 27 + node * 9;
        for (int j = 0; j < 3; ++j) {
            g += sd[j] * T[(int64_t)(33 + (step - 1) * 3 + j) * W]
                + sd[3 + j] * T[(int64_t)(45 + (step - 1) * 3 + j) * W];
            g += sd[6 + j] * T[(int64_t)((fix_q3 ? 4 + step : 8) * 3 + j) * W];
        }
    }
    a.grad[unit * 6 + dir] = g;
}

// ---- closest approach of listed pairs, with the seeds of d(miss) ----
__global__ void __launch_bounds__(128) pair_approach_kernel(PairArgs a)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n_pairs)
        return;
    const int64_t oa = a.pairs[2 * p], ob = a.pairs[2 * p + 1], n = a.n_obj;
    const int N = a.steps;
    const double h = a.h;
    // running minimum of the sampled distance (UpdateClosestApproachKernel, device.cu:56-91)
    double best = __longlong_as_double(0x7ff0000000000000ll); // +inf
    int bk = -1;
    for (int k = 0; k < N; ++k) {
        double d2 = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double d = a.traj_r[((int64_t)k * 3 + c) * n + oa] - a.traj_r[((int64_t)k * 3 + c) * n + ob];
            d2 += d * d;
        }
        if (d2 < best) {
            best = d2;
            bk = k;
        }
    }
    double seed[27];
#pragma unroll
    for (int i = 0; i < 27; ++i)
        seed[i] = 0.0;
    double tca, miss;
    int step0;
    if (bk <= 0 || bk >= N - 1) {
        // first or last sample: not refined (device.cu:100-110); miss = the sampled distance
        const int k = bk < 0 ? 0 : bk;
        tca = k == 0 ? 0.0 : (double)N * h;
        double D[3], d2 = 0.0;
        for (int c = 0; c < 3; ++c) {
            D[c] = a.traj_r[((int64_t)k * 3 + c) * n + oa] - a.traj_r[((int64_t)k * 3 + c) * n + ob];
            d2 += D[c] * D[c];
        }
        miss = sqrt(d2);
        step0 = k + 1;
        if (miss > 0.0)
            for (int c = 0; c < 3; ++c)
                seed[c] = D[c] / miss;
    } else {
        // Hermite through trajectory indices bk-1, bk, bk+1 (steps bk .. bk+2), secant TCA
        // (CalculateClosestApproachesKernel, device.cu:111-173)
        Pair6 H;
        H.dt = h;
        for (int c = 0; c < 3; ++c) {
            double qa[9], qb[9];
            for (int node = 0; node < 3; ++node) {
                const int64_t base = ((int64_t)(bk - 1 + node) * 3 + c) * n;
                qa[node * 3 + 0] = a.traj_r[base + oa];
                qa[node * 3 + 1] = a.traj_v[base + oa];
                qa[node * 3 + 2] = a.traj_a[base + oa];
                qb[node * 3 + 0] = a.traj_r[base + ob];
                qb[node * 3 + 1] = a.traj_v[base + ob];
                qb[node * 3 + 2] = a.traj_a[base + ob];
            }
            herm_build(H.A[c], qa[0], qa[1], qa[2], qa[3], qa[4], qa[5], qa[6], qa[7], qa[8], h);
            herm_build(H.B[c], qb[0], qb[1], qb[2], qb[3], qb[4], qb[5], qb[6], qb[7], qb[8], h);
        }
        const double t = find_root(H, 0.0, h);
        tca = t + (double)bk * h;
        double D[3], D1[3], D2[3], d2 = 0.0, f = 0.0, ft = 0.0;
        for (int c = 0; c < 3; ++c) {
            D[c] = herm_eval(H.A[c], h, t) - herm_eval(H.B[c], h, t);
            D1[c] = herm_deriv(H.A[c], h, t) - herm_deriv(H.B[c], h, t);
            D2[c] = herm_deriv2(H.A[c], h, t) - herm_deriv2(H.B[c], h, t);
            d2 += D[c] * D[c];
            f += D[c] * D1[c];
            ft += D1[c] * D1[c] + D[c] * D2[c];
        }
        miss = sqrt(d2);
        step0 = bk;
        if (miss > 0.0) {
            // miss = |D(t*)|, f(t*) = D . D' = 0 defines t*: d miss = (D . dD + f dt*) / miss,
            // dt* = -(D' . dD + D . dD') / f_t (implicit function at the computed root). The
            // interpolant is linear in the node data, so dD = sum_i beta_i(t*) d(data_i).
            for (int i = 0; i < 9; ++i) {
                Herm B;
                double e[9];
                for (int k = 0; k < 9; ++k)
                    e[k] = k == i ? 1.0 : 0.0;
                herm_build(B, e[0], e[1], e[2], e[3], e[4], e[5], e[6], e[7], e[8], h);
                const double beta = herm_eval(B, h, t), dbeta = herm_deriv(B, h, t);
                for (int c = 0; c < 3; ++c) {
                    const double df = beta * D1[c] + D[c] * dbeta;
                    const double dt = ft != 0.0 ? -df / ft : 0.0;
                    // node i/3, kind i%3 (r, v, a) -> seed layout [node][r3 | v3 | a3]
                    seed[(i / 3) * 9 + (i % 3) * 3 + c] = (D[c] * beta + f * dt) / miss;
                }
            }
        }
    }
    a.tca[p] = tca;
    a.miss[p] = miss;
    a.closest[p] = bk;
    a.unit_obj[2 * p] = (int)oa;
    a.unit_obj[2 * p + 1] = (int)ob;
    a.seed_step0[2 * p] = step0;
    a.seed_step0[2 * p + 1] = step0;
    for (int i = 0; i < 27; ++i) {
        a.seeds[(2 * p) * 27 + i] = seed[i];
        a.seeds[(2 * p + 1) * 27 + i] = -seed[i];
    }
}

// ---- launchers ----
cudaError_t launch_jac_points(const TableSrc& plain64, const JacPoints& a, int num_sms, cudaStream_t s)
{
    if (a.total <= 0)
        return cudaSuccess;
    const size_t smem = 128 + (size_t)plain64.bytes;
    const cudaError_t e
        = cudaFuncSetAttribute(jac_points_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    // few points spread over the SMs in blocks of a warp or more, many take a block of 8 warps per SM
    const int64_t per_sm = (a.total + num_sms - 1) / num_sms;
    const int block = (int)std::min<int64_t>(256, std::max<int64_t>(32, (per_sm + 31) / 32 * 32));
    const unsigned grid = (unsigned)std::min<int64_t>(num_sms, (a.total + block - 1) / block);
    jac_points_kernel<<<grid, block, smem, s>>>(plain64, a);
    return cudaGetLastError();
}

cudaError_t launch_rk8_tangents(const StartupTangentArgs& a, cudaStream_t s)
{
    rk8_tangent_kernel<<<(unsigned)((12 * a.n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pass_tangents(const StartupTangentArgs& a, cudaStream_t s)
{
    pass_tangent_kernel<<<(unsigned)((6 * a.n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_corrector_tangents(const StartupTangentArgs& a, cudaStream_t s)
{
    corrector_tangent_kernel<<<(unsigned)((6 * a.n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_stm_sweep(const StmArgs& a, cudaStream_t s)
{
    if (a.n <= 0)
        return cudaSuccess;
    stm_sweep_kernel<<<(unsigned)((6 * a.n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_sweep(const AdjSweepArgs& a, cudaStream_t s)
{
    if (a.n_units <= 0)
        return cudaSuccess;
    adjoint_sweep_kernel<<<(unsigned)((a.n_units + 63) / 64), 64, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_finish(const AdjFinishArgs& a, cudaStream_t s)
{
    if (a.n_units <= 0)
        return cudaSuccess;
    adjoint_finish_kernel<<<(unsigned)((6 * a.n_units + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pair_approach(const PairArgs& a, cudaStream_t s)
{
    if (a.n_pairs <= 0)
        return cudaSuccess;
    pair_approach_kernel<<<(unsigned)((a.n_pairs + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

// ---- acceleration Jacobian of many positions (gpop_gravity_jacobian) ----
// LANE: P lanes per point on the lane-layout table (few points), else a point per thread on the plain one.
template <bool LANE>
__global__ void __launch_bounds__(256, 1) jacobian_kernel(TableSrc ts, int64_t n, int P, const double* r,
    const double* M, double* acc, double* jac, unsigned* err)
{
    extern __shared__ __align__(128) uint8_t smem[];
    GravSmem g;
    if constexpr (LANE) {
        if (!bind_lane_table(smem, ts, err, g))
            return;
    } else {
        if (!bind_plain64(smem, ts, err, g))
            return;
    }
    const int lane = (int)threadIdx.x & 31, l = LANE ? (int)threadIdx.x % P : 0;
    const unsigned mask = !LANE ? 0u : P == 32 ? 0xffffffffu : ((1u << P) - 1u) << (lane & ~(P - 1));
    const int64_t T = ((int64_t)gridDim.x * blockDim.x) / P;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / P; i < n; i += T) {
        const double ri[3] = { r[i * 3], r[i * 3 + 1], r[i * 3 + 2] };
        double a[3], J[3][3];
        if (M)
            gravity_jac_gcrs<LANE>(g, l, P, M, ri, a, J, mask);
        else
            gravity_jac_itrs<LANE>(g, l, P, ri[0], ri[1], ri[2], a, J, mask);
        if (l == 0)
            for (int k = 0; k < 3; ++k) {
                if (acc)
                    acc[i * 3 + k] = a[k];
                for (int m = 0; m < 3; ++m)
                    jac[(i * 3 + k) * 3 + m] = J[k][m];
            }
    }
}

// Lanes per point: the most (<= 32) that keep all points in one block of 8 warps per SM; one thread per
// point once every scheduler has a warp of them (n >= 128 per SM).
cudaError_t launch_jacobian(const TableSrc& plain64, const TableSrc& lane64, int64_t n, const double* r,
    const double* M, double* acc, double* jac, unsigned* err, int num_sms, cudaStream_t s)
{
    if (n <= 0)
        return cudaSuccess;
    int P = 1;
    if (n < (int64_t)num_sms * 128)
        for (P = 2; P < 32 && n * 2 * P <= (int64_t)num_sms * 256;)
            P *= 2;
    const TableSrc& ts = P > 1 ? lane64 : plain64;
    const size_t smem = 128 + (size_t)ts.bytes;
    const int64_t threads = n * P, per_sm = (threads + num_sms - 1) / num_sms;
    const int block = (int)std::min<int64_t>(256, std::max<int64_t>(32, (per_sm + 31) / 32 * 32));
    const unsigned grid = (unsigned)std::min<int64_t>(num_sms, (threads + block - 1) / block);
    cudaError_t e;
    if (P > 1) {
        if ((e = cudaFuncSetAttribute(jacobian_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
            return e;
        jacobian_kernel<true><<<grid, block, smem, s>>>(ts, n, P, r, M, acc, jac, err);
    } else {
        if ((e = cudaFuncSetAttribute(jacobian_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
            return e;
        jacobian_kernel<false><<<grid, block, smem, s>>>(ts, n, P, r, M, acc, jac, err);
    }
    return cudaGetLastError();
}

} // namespace gpop
