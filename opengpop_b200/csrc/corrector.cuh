// corrector.cuh -- end of the GJ8 corrector iteration of one object under gravity.
#pragma once
#include "common.cuh"
#include "gj8_tables.cuh"
#include "model.h"

namespace gpop {

// J of a position: the Jacobian of
//   a = -GM/r^2 u - GM b/r^2 [(1 - 5 s^2) u + 2 s e],  b = 1.5 J2 R^2/r^2, s = u . e,
// e the polar axis (the frame's z: off the Earth's axis by some 1e-3, which J2 turns into 1e-6 of J).
struct CorrJacobian {
    float u[3], len, g, b; // unit vector, r, GM / r^3
    __device__ __forceinline__ CorrJacobian() {}
    __device__ __forceinline__ CorrJacobian(const CorrModel& cm, const double (&r)[3])
    {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            u[j] = (float)r[j];
        const float r2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        const float ri = rsqrtf(r2);
        len = r2 * ri;
        g = (cm.gm * ri) * ri * ri;
        b = cm.j2 * ri * ri;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            u[j] *= ri;
    }
    __device__ __forceinline__ void apply(const float (&y)[3], float (&o)[3]) const
    {
        const float s = u[2], c5 = 1.f - 5.f * s * s;
        const float dr = u[0] * y[0] + u[1] * y[1] + u[2] * y[2];
        const float t = s * (y[2] - s * dr); // r/2 times the change of s^2
        const float pu = 3.f * dr + b * (5.f * dr * c5 + 10.f * t);
        const float py = 1.f + b * c5;
        const float pz = b * (10.f * dr * s - 2.f * y[2]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            o[j] = g * (pu * u[j] - py * y[j] + (j == 2 ? pz : 0.f));
    }
};

// The corrector iterates the position to the fixed point of
//   F(r) = h^2 (s2 + GJ[8][8] a(r) + S)   (gpu_propagator.cu:86-119),
// one gravity evaluation per pass; s and v of the step follow from the last acceleration. Each pass
// shrinks the distance to the fixed point by rho = h^2 |GJ[8][8]| |da/dr|, 1.6e-4 in LEO at 30 s, so
// the seven passes of the method end far below the last bit. correct_position takes the acceleration
// at r and moves r on:
// - the bits of F(r) are those of r: the passes left would return them again, done;
// - the passes left would not settle r (few passes, long steps), or r lies below 1.02 R: the plain
//   pass r = F(r);
// - else the fixed point under a(r) + J y, J the Jacobian of the central term and J2 and y the
//   distance to that point: the next evaluation is three digits nearer than that of a plain pass.
//   When |F(r) - r| is at most `near` of r (corrector_model: 9.6e-15 for JGM3, 7e-8 m in LEO), what J
//   leaves out of the acceleration is below a tenth of its last bit: a + J y is the acceleration at
//   the fixed point to rounding, and no evaluation follows.
// Positions, sums and the acceleration stay FP64; J y, a correction of their last digits, is FP32.
// Bounds a propagation (every other cost is per evaluation). Evaluations of a step by a warp of 64
// objects, which waits for the slowest: 7 as the method states them; 4.0 when passes end on equal
// bits alone (LEO and the mixed population at 30 s; 4.5 at 60 s); 2.7 with the central term for J
// and eight last bits for `near`; 2.0 with J2 and `near` as here. Position error against a long double
// propagation, rms of 160 LEO objects after 1,000 steps, seven passes / this rule: 10 s 2.49e-7 / 2.23e-7 m, 30 s
// 5.35e-7 / 5.77e-7, 60 s 1.13e-6 / 1.05e-6 (the sums of rounded accelerations; such figures scatter by 6 %; the
// tests hold them to the oracle's seven passes). 18,501 objects, 240 steps, FP64, the call:
// 85.6 -> 30.2 ms; 65,536 mixed, 320 steps: 147.2 -> 54.5 ms.
//
// it, ncorr: this pass and the passes of the method. fast: kept by the caller between the passes of
// a step. Returns whether the object's step is done; r and a are then its position and acceleration.
__device__ __forceinline__ bool correct_position(const CorrModel& cm, double h, int it, int ncorr,
    const double (&s2)[3], const double (&S)[3], double (&a)[3], double (&r)[3], bool& fast)
{
    double rn[3];
    bool same = true;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        rn[j] = h * h * (fma(a[j], c_GJ[8][8], s2[j]) + S[j]);
        same = same && same_bits(rn[j], r[j]);
    }
    if (same)
        return true;
    float d[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        d[j] = (float)(rn[j] - r[j]);
    const CorrJacobian jac(cm, r);
    const float hg = (float)(h * h * c_GJ[8][8]);
    const float dmax = fmaxf(fmaxf(fabsf(d[0]), fabsf(d[1])), fabsf(d[2]));
    if (it == 0) {
        // change of the plain iteration after its last pass, with one power of rho to spare
        const float rho = 2.2f * fabsf(hg * jac.g);
        float left = dmax;
        for (int i = 2; i < ncorr && i < 10; ++i)
            left *= rho;
        fast = ncorr > 2 && rho < 0.1f && left <= 0x1p-54f * jac.len && jac.len >= cm.low;
    }
    const bool near = dmax <= cm.near * jac.len;
    if (!fast || (it == ncorr - 1 && !near)) {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            r[j] = rn[j];
        return it == ncorr - 1;
    }
    // y = (I - h^2 GJ[8][8] J)^-1 d to second order
    float y[3] = { d[0], d[1], d[2] }, o[3];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        jac.apply(y, o);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            y[j] = d[j] + hg * o[j];
    }
    jac.apply(y, o);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const double aj = a[j] + (double)o[j];
        r[j] = h * h * (fma(aj, c_GJ[8][8], s2[j]) + S[j]);
        if (near)
            a[j] = aj;
    }
    return near;
}

} // namespace gpop
