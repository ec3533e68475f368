// jacobian.cuh -- gravity acceleration and its 3x3 Jacobian (FP64), by one thread or a lane group.
//
// The column sums are functions of q = R/r and eps = z/r only, and Q(n,m) = q^n P(n,m)(eps) is
// homogeneous of degree n in q, so q dQ/dq = n Q and dQ/deps follows the recursion
//   E(n) = q Q(n-1) + u E(n-1) - c w E(n-2),  E(m) = 0   (from Q(n) = u Q(n-1) - c w Q(n-2)).
// The longitude enters through z^m, z = C1 + i S1. G, J, K, H of eq. 4-11 and their partials in
// (q, eps, C1, S1) are chained to the Earth-fixed position. Of the 18 sums per column that this takes
// as it stands (Q, n Q and E with g, j and h) twelve are enough:
// - g = (1 + n + m) j, so the g sums are j sums of Q, n Q and n^2 Q;
// - the E sums of column m - 1 with j are the Q sums of column m with h (the derivative of column m - 1
//   is column m), those with g the Q and n Q sums with h.
// For the same reason dJ/deps = dH/dC1, dK/deps = dH/dS1, dK/dC1 = dJ/dS1 and dK/dS1 = -dJ/dC1: 16
// totals. A term takes 21 FP64 operations and three 16-byte table reads (26 and four before).
#pragma once
#include "gravity.cuh"
#include "lanes.cuh"

namespace gpop {

struct JacTotals {
    double Gv = 0, Gq = 0, Ge = 0, Gc = 0, Gs = 0, Jv = 0, Jq = 0, Jc = 0, Js = 0, Kv = 0, Kq = 0;
    double Hv = 0, Hq = 0, He = 0, Hc = 0, Hs = 0;
};

// Column m (entries e[0..L - m]) into the totals; (Cm, Sm), (Cp, Sp), (Cq, Sq) = z^m, z^(m-1), z^(m-2)
// (zero for negative powers), qm = q^m.
__device__ __forceinline__ void jac_column(const GravEntry64* __restrict__ e, int m, int L, double q, double u,
    double w, double qm, double Cm, double Sm, double Cp, double Sp, double Cq, double Sq, JacTotals& t)
{
    double j0[2], j1[2], j2[2], h0[2], h1[2], he[2] = { 0.0, 0.0 };
    double dn = (double)m;
    {
        const double2* p = reinterpret_cast<const double2*>(e);
        const double2 j = p[2], h = p[3];
        const double nQ = dn * qm, n2 = dn * nQ;
        j0[0] = j.x * qm;
        j0[1] = j.y * qm;
        j1[0] = j.x * nQ;
        j1[1] = j.y * nQ;
        j2[0] = j.x * n2;
        j2[1] = j.y * n2;
        h0[0] = h.x * qm;
        h0[1] = h.y * qm;
        h1[0] = h.x * nQ;
        h1[1] = h.y * nQ;
    }
    // tq, te hold c(n) w Q(n-2) and c(n) w E(n-2), formed one term ahead (c(m + 1) = 0)
    double Q1 = qm, E1 = 0.0, tq = 0.0, te = 0.0;
#pragma unroll 4
    for (int i = 1; i <= L - m; ++i) {
        const double2* p = reinterpret_cast<const double2*>(e + i);
        const double2 j = p[2], h = p[3];
        const double cw = reinterpret_cast<const double2*>(e + i + 1)[0].x * w;
        const double Q = fma(u, Q1, -tq);
        const double E = fma(q, Q1, fma(u, E1, -te));
        tq = cw * Q1;
        te = cw * E1;
        dn += 1.0;
        const double nQ = dn * Q, n2 = dn * nQ;
        j0[0] = fma(j.x, Q, j0[0]);
        j0[1] = fma(j.y, Q, j0[1]);
        j1[0] = fma(j.x, nQ, j1[0]);
        j1[1] = fma(j.y, nQ, j1[1]);
        j2[0] = fma(j.x, n2, j2[0]);
        j2[1] = fma(j.y, n2, j2[1]);
        h0[0] = fma(h.x, Q, h0[0]);
        h0[1] = fma(h.y, Q, h0[1]);
        h1[0] = fma(h.x, nQ, h1[0]);
        h1[1] = fma(h.y, nQ, h1[1]);
        he[0] = fma(h.x, E, he[0]);
        he[1] = fma(h.y, E, he[1]);
        Q1 = Q;
        E1 = E;
    }
    const double dm = (double)m, dm1 = dm - 1.0, mm = dm * dm1;
    const double g0[2] = { fma(dm + 1.0, j0[0], j1[0]), fma(dm + 1.0, j0[1], j1[1]) };
    const double g1[2] = { fma(dm + 1.0, j1[0], j2[0]), fma(dm + 1.0, j1[1], j2[1]) };
    const double ge[2] = { fma(dm, h0[0], h1[0]), fma(dm, h0[1], h1[1]) }; // of column m - 1
    t.Gv += Cm * g0[0] + Sm * g0[1];
    t.Gq += Cm * g1[0] + Sm * g1[1];
    t.Ge += Cp * ge[0] + Sp * ge[1];
    t.Gc += dm * (Cp * g0[0] + Sp * g0[1]);
    t.Gs += dm * (Cp * g0[1] - Sp * g0[0]);
    t.Jv += dm * (Cp * j0[0] + Sp * j0[1]);
    t.Jq += dm * (Cp * j1[0] + Sp * j1[1]);
    t.Jc += mm * (Cq * j0[0] + Sq * j0[1]);
    t.Js += mm * (Cq * j0[1] - Sq * j0[0]);
    t.Kv += dm * (Cp * j0[1] - Sp * j0[0]);
    t.Kq += dm * (Cp * j1[1] - Sp * j1[0]);
    t.Hv += Cp * h0[0] + Sp * h0[1];
    t.Hq += Cp * h1[0] + Sp * h1[1];
    t.He += Cp * he[0] + Sp * he[1];
    t.Hc += dm1 * (Cq * h0[0] + Sq * h0[1]);
    t.Hs += dm1 * (Cq * h0[1] - Sq * h0[0]);
}

// Acceleration a and Jacobian Jm[i][j] = d a_i / d p_j in the Earth-fixed frame with the columns over the
// P lanes of a group (lane l takes l, l + P, ...; mask: the group's lanes). LANE: lane-layout table; P = 1
// with the plain table is one thread per point.
template <bool LANE>
__device__ __forceinline__ void gravity_jac_itrs(const GravSmem& gs, int l, int P, double x, double y, double z,
    double* a, double (*Jm)[3], unsigned mask)
{
    const int L = gs.L;
    const double invr = inv_norm(x, y, z);
    const double eps = z * invr, q = gs.radius * invr;
    const double u = q * eps, w = q * q;
    const double C1 = x * invr, S1 = y * invr;
    JacTotals t;
    if constexpr (LANE) {
        double CP, SP, qP = 1.0, qm = 1.0;
        cpow(C1, S1, P, CP, SP);
        for (int i = 0; i < P; ++i)
            qP *= q;
        for (int i = 0; i < l; ++i)
            qm *= q;
        double Cm = 0, Sm = 0, Cp = 0, Sp = 0, Cq = 0, Sq = 0;
        for (int m = l; m <= L; m += P) {
            if (m == l || m - P < 2) { // first column of the lane, or a zero power to restart
                cpow(C1, S1, m, Cm, Sm);
                Cp = Sp = Cq = Sq = 0.0;
                if (m >= 1)
                    cpow(C1, S1, m - 1, Cp, Sp);
                if (m >= 2)
                    cpow(C1, S1, m - 2, Cq, Sq);
            } else {
                cmul(Cm, Sm, CP, SP, Cm, Sm);
                cmul(Cp, Sp, CP, SP, Cp, Sp);
                cmul(Cq, Sq, CP, SP, Cq, Sq);
            }
            jac_column(lane_col64(gs, m), m, L, q, u, w, qm, Cm, Sm, Cp, Sp, Cq, Sq, t);
            qm *= qP;
        }
        lane_sum4(t.Gv, t.Gq, t.Ge, t.Gc, l, P, mask);
        lane_sum4(t.Gs, t.Jv, t.Jq, t.Jc, l, P, mask);
        lane_sum4(t.Js, t.Kv, t.Kq, t.Hv, l, P, mask);
        lane_sum4(t.Hq, t.He, t.Hc, t.Hs, l, P, mask);
    } else {
        double qm = 1.0, Cm = 1.0, Sm = 0.0, Cp = 0.0, Sp = 0.0, Cq = 0.0, Sq = 0.0;
#pragma unroll 1
        for (int m = 0; m <= L; ++m) {
            jac_column(gs.t64 + grav_col_offset(m, gs.Lt), m, L, q, u, w, qm, Cm, Sm, Cp, Sp, Cq, Sq, t);
            Cq = Cp;
            Sq = Sp;
            Cp = Cm;
            Sp = Sm;
            cmul(Cm, Sm, C1, S1, Cm, Sm);
            qm *= q;
        }
    }
    // value and partials in q, eps, C1, S1 of G, J, K, H (the q sums are q d/dq)
    const double qi = 1.0 / q;
    const double F[4][5] = { { t.Gv, t.Gq * qi, t.Ge, t.Gc, t.Gs }, { t.Jv, t.Jq * qi, t.Hc, t.Jc, t.Js },
        { t.Kv, t.Kq * qi, t.Hs, t.Js, -t.Jc }, { t.Hv, t.Hq * qi, t.He, t.Hc, t.Hs } };
    const double ph[3] = { C1, S1, eps };
    double gq[3], ge[3], gc[3], gsn[3]; // gradients of q, eps, C1, S1
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        gq[j] = -q * invr * ph[j];
        ge[j] = ((j == 2 ? 1.0 : 0.0) - eps * ph[j]) * invr;
        gc[j] = ((j == 0 ? 1.0 : 0.0) - C1 * ph[j]) * invr;
        gsn[j] = ((j == 1 ? 1.0 : 0.0) - S1 * ph[j]) * invr;
    }
    double dF[4][3];
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            dF[f][j] = F[f][1] * gq[j] + F[f][2] * ge[j] + F[f][3] * gc[j] + F[f][4] * gsn[j];
    // a = c (Lambda p^ - P), P = (J, K, H), Lambda = 1 + G + eps H, c = -GM / r^2
    const double Lambda = t.Gv + 1.0 + eps * t.Hv;
    const double e = norm_error(x, y, z, invr), c0 = -gs.gm * (invr * invr);
    const double c = fma(c0, 1.5 * e, c0); // as central()
    const double pe[3] = { fma(ph[0], e, ph[0]), fma(ph[1], e, ph[1]), fma(ph[2], e, ph[2]) }; // and of its p^ p^
    double dL[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        dL[j] = dF[0][j] + eps * dF[3][j] + t.Hv * ge[j];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double base = Lambda * ph[i] - F[i + 1][0];
        a[i] = c * base;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            Jm[i][j] = -2.0 * c * pe[j] * invr * base
                + c * (dL[j] * ph[i] + Lambda * ((i == j ? 1.0 : 0.0) - ph[i] * pe[j]) * invr - dF[i + 1][j]);
    }
}

// GCRS acceleration and Jacobian for the ITRS<-GCRS matrix M of gravity_gcrs: p = A r with
// A[i][k] = M[3 i + k], a = A^T a_itrs, J = A^T J_itrs A.
template <bool LANE>
__device__ __forceinline__ void gravity_jac_gcrs(const GravSmem& gs, int l, int P, const double* __restrict__ M,
    const double* r, double* a, double (*Jg)[3], unsigned mask)
{
    double p[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        p[i] = __ldg(M + 3 * i) * r[0] + __ldg(M + 3 * i + 1) * r[1] + __ldg(M + 3 * i + 2) * r[2];
    double ai[3], Ji[3][3];
    gravity_jac_itrs<LANE>(gs, l, P, p[0], p[1], p[2], ai, Ji, mask);
    double A[3][3];
#pragma unroll
    for (int i = 0; i < 9; ++i)
        A[i / 3][i % 3] = __ldg(M + i);
    double T[3][3]; // J_itrs A
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            T[i][k] = Ji[i][0] * A[0][k] + Ji[i][1] * A[1][k] + Ji[i][2] * A[2][k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = A[0][k] * ai[0] + A[1][k] * ai[1] + A[2][k] * ai[2];
#pragma unroll
        for (int l2 = 0; l2 < 3; ++l2)
            Jg[k][l2] = A[0][k] * T[0][l2] + A[1][k] * T[1][l2] + A[2][k] * T[2][l2];
    }
}

} // namespace gpop
