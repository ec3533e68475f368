// lanes.cuh -- gravity with the columns of the triangle split over the P lanes of an object
// (lane l of P takes m = l, l + P, ...); the per-object sums are added with warp shuffles among
// the lanes named by `mask` (the whole warp, or the object's aligned group of P lanes), so every
// lane of the object ends with the same result. Used where one object per thread leaves
// the GPU idle: calls with few objects, long requests of a batch, Jacobians of few points. The tables
// are in the lane layout (build_lane_blob), so the lanes' simultaneous reads of different columns
// fall in different shared-memory banks.
#pragma once
#include "gravity.cuh"
#include "kernels.h"

namespace gpop {

// Stages a lane-layout blob into shared memory (after a 128-byte mbarrier slot) and binds it.
__device__ __forceinline__ bool bind_lane_table(uint8_t* smem, const TableSrc& ts, unsigned* err, GravSmem& g)
{
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);
    uint8_t* tab = smem + 128;
    const bool ok = stage_to_smem(tab, ts.src, ts.bytes, mbar, err, ts.wait_spins);
    g.L = ts.L;
    g.Lt = ts.L;
    g.radius = ts.radius;
    g.gm = ts.gm;
    g.cb64 = reinterpret_cast<const int*>(tab);
    g.cb32 = reinterpret_cast<const int*>(tab + 512);
    g.t64 = reinterpret_cast<const GravEntry64*>(tab + kLaneOff64);
    g.t32 = reinterpret_cast<const GravEntry32*>(tab + ts.off32);
    return ok;
}

__device__ __forceinline__ void cmul(double ac, double as, double bc, double bs, double& rc, double& rs)
{
    const double c = ac * bc - as * bs;
    const double s = as * bc + ac * bs;
    rc = c;
    rs = s;
}

#ifndef GPOP_LANE_PAIR_COLUMNS
#define GPOP_LANE_PAIR_COLUMNS 1
#endif
constexpr bool kLanePairColumns = GPOP_LANE_PAIR_COLUMNS != 0;

// Eq. 4-11 for column m of a lane walk, then the lane's cos/sin(m lambda) and q^m recursions step
// P columns on (z^P; from column 0 the m - 1 values jump to z^(P-1)).
template <int K>
__device__ __forceinline__ void lane_combine(int m, const ColSums64<K>& s, const double (&CP)[K],
    const double (&SP)[K], const double (&CPm1)[K], const double (&SPm1)[K], const double (&qP)[K],
    double (&Cm)[K], double (&Sm)[K], double (&Cp)[K], double (&Sp)[K], double (&qm)[K],
    double (&G)[K], double (&H)[K], double (&J)[K], double (&KK)[K])
{
    const double dm = (double)m;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        G[k] += Cm[k] * s.g1[k] + Sm[k] * s.g2[k];
        J[k] += dm * (Cp[k] * s.j1[k] + Sp[k] * s.j2[k]);
        KK[k] -= dm * (Sp[k] * s.j1[k] - Cp[k] * s.j2[k]);
        H[k] += Cp[k] * s.h1[k] + Sp[k] * s.h2[k];
        if (m == 0) {
            Cp[k] = CPm1[k];
            Sp[k] = SPm1[k];
        } else {
            cmul(Cp[k], Sp[k], CP[k], SP[k], Cp[k], Sp[k]);
        }
        cmul(Cm[k], Sm[k], CP[k], SP[k], Cm[k], Sm[k]);
        qm[k] *= qP[k];
    }
}

// (C1 + i S1)^p by binary powering (p >= 0).
__device__ __forceinline__ void cpow(double c1, double s1, int p, double& rc, double& rs)
{
    double xc = 1.0, xs = 0.0, bc = c1, bs = s1;
    while (p > 0) {
        if (p & 1)
            cmul(xc, xs, bc, bs, xc, xs);
        p >>= 1;
        if (p)
            cmul(bc, bs, bc, bs, bc, bs);
    }
    rc = xc;
    rs = xs;
}

// What a lane's columns m, m + P, ... start from and step by: z = C1 + i S1 and q to the powers m, m - 1 (none
// for column 0), P and P - 1 (the m - 1 values of column P, for the lane that starts at column 0). P is a
// power of two, or beyond the last column (one round: only the first three are made). top: the largest m - 1
// of the group. The powers come from the squares z^2, z^4, ... that every lane forms (two dependent
// operations per bit, where a scan over the lanes adds a shuffle to each).
struct LanePowers {
    double Cm, Sm, Cp, Sp, qm, CP, SP, CPm1, SPm1, qP;
};
__device__ __forceinline__ LanePowers lane_powers(double C1, double S1, double q, int m, int top, int P, bool steps)
{
    LanePowers w;
    const int e = m > 0 ? m - 1 : 0;
    double bc = C1, bs = S1, bq = q, xc = 1.0, xs = 0.0, xq = 1.0;
    w.CPm1 = 1.0;
    w.SPm1 = 0.0;
    w.CP = C1;
    w.SP = S1;
    w.qP = q;
    for (int o = 1; o <= top || (steps && o < P); o <<= 1) {
        double tc, ts;
        cmul(xc, xs, bc, bs, tc, ts);
        const bool on = (e & o) != 0;
        xc = on ? tc : xc;
        xs = on ? ts : xs;
        xq = on ? xq * bq : xq;
        if (steps && o < P)
            cmul(w.CPm1, w.SPm1, bc, bs, w.CPm1, w.SPm1);
        cmul(bc, bs, bc, bs, bc, bs);
        bq *= bq;
        if (2 * o == P) {
            w.CP = bc;
            w.SP = bs;
            w.qP = bq;
        }
    }
    cmul(xc, xs, C1, S1, w.Cm, w.Sm);
    w.qm = xq * q;
    w.Cp = m > 0 ? xc : 0.0;
    w.Sp = m > 0 ? xs : 0.0;
    w.Cm = m > 0 ? w.Cm : 1.0;
    w.Sm = m > 0 ? w.Sm : 0.0;
    w.qm = m > 0 ? w.qm : 1.0;
    return w;
}

// Totals of four values over the P lanes (a power of two) of each aligned group, in every lane. From
// four lanes the first two levels halve what a lane still carries: 2 + 1 + log2 P - 2 exchanges and
// four broadcasts of a value instead of 4 log2 P exchanges.
__device__ __forceinline__ void lane_sum4(double& a, double& b, double& c, double& d, int l, int P,
    unsigned mask)
{
    if (P >= 4) {
        const int h = P >> 1, f = P >> 2;
        const bool hi = (l & h) != 0, hf = (l & f) != 0;
        double x = hi ? c : a, y = hi ? d : b;
        x += __shfl_xor_sync(mask, hi ? a : c, h);
        y += __shfl_xor_sync(mask, hi ? b : d, h);
        double t = hf ? y : x;
        t += __shfl_xor_sync(mask, hf ? x : y, f);
        for (int o = P >> 3; o > 0; o >>= 1)
            t += __shfl_xor_sync(mask, t, o);
        a = __shfl_sync(mask, t, 0, P);
        b = __shfl_sync(mask, t, f, P);
        c = __shfl_sync(mask, t, h, P);
        d = __shfl_sync(mask, t, h + f, P);
    } else if (P == 2) {
        a += __shfl_xor_sync(mask, a, 1);
        b += __shfl_xor_sync(mask, b, 1);
        c += __shfl_xor_sync(mask, c, 1);
        d += __shfl_xor_sync(mask, d, 1);
    }
}

// The lanes of a group inside one warp: lane l of P, the group's lanes of the warp.
struct WarpTeam {
    int l, P;
    unsigned mask;
    __device__ __forceinline__ int top() const { return P - 2; } // LanePowers
    __device__ __forceinline__ void sum4(double& a, double& b, double& c, double& d) const
    {
        lane_sum4(a, b, c, d, l, P, mask);
    }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
};

// A group of whole warps (T = 32 warps threads, at least one per column): lane sums in each warp, then
// over the warps through shared memory. buf holds 2 x 4 x warps doubles of this group; the two halves
// take turns, so that one barrier per sum is enough (a warp that is a sum ahead writes the other half,
// and cannot be two ahead). bar: the group's named barrier.
struct BlockTeam {
    int l, P, warps, bar;
    double* buf;
    mutable int half;
    __device__ __forceinline__ int top() const { return (l | 31) - 1; } // of the warp: the first has the longest columns
    __device__ __forceinline__ void sync() const
    {
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(P) : "memory");
    }
    __device__ __forceinline__ void sum4(double& a, double& b, double& c, double& d) const
    {
        const int lane = l & 31;
        lane_sum4(a, b, c, d, lane, 32, 0xffffffffu);
        double* h = buf + half * 4 * warps;
        if (lane < 4)
            h[(l >> 5) * 4 + lane] = lane == 0 ? a : lane == 1 ? b : lane == 2 ? c : d;
        sync();
        a = b = c = d = 0.0;
        for (int w = 0; w < warps; ++w) {
            a += h[w * 4];
            b += h[w * 4 + 1];
            c += h[w * 4 + 2];
            d += h[w * 4 + 3];
        }
        half ^= 1;
    }
};

// Lanes per group as gravity_itrs_team takes them: P <= 32 lanes of a warp, or whole warps.
template <bool WARPS> struct TeamOf;
template <> struct TeamOf<false> {
    using type = WarpTeam;
};
template <> struct TeamOf<true> {
    using type = BlockTeam;
};
template <bool WARPS>
__device__ __forceinline__ typename TeamOf<WARPS>::type make_team(int P, double* buf)
{
    const int l = (int)threadIdx.x % P;
    if constexpr (WARPS) {
        return BlockTeam { l, P, P / 32, 1 + (int)threadIdx.x / P, buf, 0 };
    } else {
        const int lane = (int)threadIdx.x & 31;
        return WarpTeam { l, P, P == 32 ? 0xffffffffu : ((1u << P) - 1u) << (lane & ~(P - 1)) };
    }
}

// Doubles of shared memory per group of gj8_team_kernel: the history, then the sums of a group of warps.
inline __host__ __device__ int team_doubles(int P, bool warps) { return 28 + (warps ? P / 4 : 0); }

// Columns first, first + P, ... up to `last` of K objects, added into G, H, J, KK. As gravity_itrs in mixed
// mode: the head columns m <= 8 are combined in FP64 (their terms of degree > 8 summed in FP32 per column),
// the columns m > 8 are walked, combined and summed in FP32 and added to the FP64 totals once. PAIRS: FP64
// lanes walk two of their columns side by side (kernels with few registers to spare keep one at a time).
template <bool MIXED, int K, bool PAIRS>
__device__ __forceinline__ void lane_walk(const GravSmem& gs, int first, int P, int last, const LanePowers (&lp)[K],
    const double (&u)[K], const double (&w)[K], double (&G)[K], double (&H)[K], double (&J)[K], double (&KK)[K])
{
    const int L = gs.L, top = MIXED && L > kMixedSplit ? kMixedSplit : L; // last degree of the FP64 terms
    double CP[K], SP[K], Cm[K], Sm[K], Cp[K], Sp[K], CPm1[K], SPm1[K], qm[K], qP[K];
    float uf[K], wf[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        uf[k] = (float)u[k];
        wf[k] = (float)w[k];
        Cm[k] = lp[k].Cm;
        Sm[k] = lp[k].Sm;
        Cp[k] = lp[k].Cp;
        Sp[k] = lp[k].Sp;
        qm[k] = lp[k].qm;
        CP[k] = lp[k].CP;
        SP[k] = lp[k].SP;
        CPm1[k] = lp[k].CPm1;
        SPm1[k] = lp[k].SPm1;
        qP[k] = lp[k].qP;
    }
    const int Lhead = min(last, MIXED && L > kMixedSplit ? kMixedSplit : L);
    // column bases of the lane's next column are read one column ahead (they are shared-memory
    // loads the walk's first table read depends on)
    int b64 = gs.cb64[min(first, 127)], b32 = gs.cb32[min(first, 127)];
    int m = first;
    if constexpr (!MIXED && PAIRS && kLanePairColumns) {
        // FP64: two of this lane's columns (m and m + P) side by side, so each object carries two
        // independent recursions; each column's sums, and their combination, in the order of the
        // one-column loop below (bit-identical accelerations)
        for (; m + P <= Lhead; m += 2 * P) {
            const int mb = m + P;
            const int mn = mb + P < 127 ? mb + P : 127;
            const int bb64 = gs.cb64[mb], nb64 = gs.cb64[mn];
            ColSums64<K> sa, sb;
            sa.zero();
            sb.zero();
            double Qa1[K], Qa2[K], Qb1[K], Qb2[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                Qa1[k] = qm[k];
                Qa2[k] = 0.0;
                Qb1[k] = qm[k] * qP[k]; // the q^m the one-column loop carries into column m + P
                Qb2[k] = 0.0;
            }
            const GravEntry64* ea = reinterpret_cast<const GravEntry64*>(reinterpret_cast<const uint4*>(gs.t64) + b64);
            const GravEntry64* eb = reinterpret_cast<const GravEntry64*>(reinterpret_cast<const uint4*>(gs.t64) + bb64);
            sa.add(ea, Qa1);
            sb.add(eb, Qb1);
            column64_pair<K>(ea + 1, eb + 1, top - mb, u, w, Qa1, Qa2, sa, Qb1, Qb2, sb);
            column64<K>(ea, top - mb + 1, top - m, u, w, Qa1, Qa2, sa);
            lane_combine<K>(m, sa, CP, SP, CPm1, SPm1, qP, Cm, Sm, Cp, Sp, qm, G, H, J, KK);
            lane_combine<K>(mb, sb, CP, SP, CPm1, SPm1, qP, Cm, Sm, Cp, Sp, qm, G, H, J, KK);
            b64 = nb64;
        }
    }
    for (; m <= Lhead; m += P) {
        const int mn = m + P < 127 ? m + P : 127;
        const int nb64 = gs.cb64[mn], nb32 = gs.cb32[mn];
        ColSums64<K> s;
        s.zero();
        double Q1[K], Q2[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            Q1[k] = qm[k];
            Q2[k] = 0.0;
        }
        const GravEntry64* e = reinterpret_cast<const GravEntry64*>(reinterpret_cast<const uint4*>(gs.t64) + b64);
        s.add(e, Q1);
        column64<K>(e, 1, top - m, u, w, Q1, Q2, s);
        if constexpr (MIXED) {
            if (L > kMixedSplit) {
                ColSums32<K> f;
                f.zero();
                float Q1f[K], Q2f[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    Q1f[k] = (float)Q1[k];
                    Q2f[k] = (float)Q2[k];
                }
                column32k<K>(reinterpret_cast<const GravEntry32*>(reinterpret_cast<const uint4*>(gs.t32) + b32),
                    kMixedSplit + 1 - m, L - m, uf, wf, Q1f, Q2f, f);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    s.g1[k] += (double)f.g[k].x;
                    s.g2[k] += (double)f.g[k].y;
                    s.j1[k] += (double)f.j[k].x;
                    s.j2[k] += (double)f.j[k].y;
                    s.h1[k] += (double)f.h[k].x;
                    s.h2[k] += (double)f.h[k].y;
                }
            }
        }
        const double dm = (double)m; // eq. 4-11
#pragma unroll
        for (int k = 0; k < K; ++k) {
            G[k] += Cm[k] * s.g1[k] + Sm[k] * s.g2[k];
            J[k] += dm * (Cp[k] * s.j1[k] + Sp[k] * s.j2[k]);
            KK[k] -= dm * (Sp[k] * s.j1[k] - Cp[k] * s.j2[k]);
            H[k] += Cp[k] * s.h1[k] + Sp[k] * s.h2[k];
            if (m == 0) {
                Cp[k] = CPm1[k];
                Sp[k] = SPm1[k];
            } else {
                cmul(Cp[k], Sp[k], CP[k], SP[k], Cp[k], Sp[k]);
            }
            cmul(Cm[k], Sm[k], CP[k], SP[k], Cm[k], Sm[k]);
            qm[k] *= qP[k];
        }
        b64 = nb64;
        b32 = nb32;
    }
    if constexpr (MIXED) {
        if (m <= last) { // this lane's columns m > 8, in FP32
            float cf[K], sf[K], cpf[K], spf[K], CPf[K], SPf[K], qmf[K], qPf[K];
            float Gf[K], Hf[K], Jf[K], Kf[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                cf[k] = (float)Cm[k];
                sf[k] = (float)Sm[k];
                cpf[k] = (float)Cp[k];
                spf[k] = (float)Sp[k];
                CPf[k] = (float)CP[k];
                SPf[k] = (float)SP[k];
                qmf[k] = (float)qm[k];
                qPf[k] = (float)qP[k];
                Gf[k] = Hf[k] = Jf[k] = Kf[k] = 0.f;
            }
            for (; m <= last; m += P) {
                const int nb = gs.cb32[m + P < 127 ? m + P : 127];
                ColSums32<K> f;
                const GravEntry32* e32 = reinterpret_cast<const GravEntry32*>(reinterpret_cast<const uint4*>(gs.t32) + b32);
                const float4* p = reinterpret_cast<const float4*>(e32);
                const float4 a = p[0], b = p[1];
                float Q1f[K], Q2f[K];
#pragma unroll
                for (int k = 0; k < K; ++k) { // n = m term (Q = q^m)
                    const float2 QQ = make_float2(qmf[k], qmf[k]);
                    f.g[k] = __fmul2_rn(QQ, make_float2(a.z, a.w));
                    f.j[k] = __fmul2_rn(QQ, make_float2(b.x, b.y));
                    f.h[k] = __fmul2_rn(QQ, make_float2(b.z, b.w));
                    Q1f[k] = qmf[k];
                    Q2f[k] = 0.f;
                }
                column32k<K>(e32, 1, L - m, uf, wf, Q1f, Q2f, f);
                const float dmf = (float)m;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    Gf[k] += cf[k] * f.g[k].x + sf[k] * f.g[k].y;
                    Jf[k] += dmf * (cpf[k] * f.j[k].x + spf[k] * f.j[k].y);
                    Kf[k] -= dmf * (spf[k] * f.j[k].x - cpf[k] * f.j[k].y);
                    Hf[k] += cpf[k] * f.h[k].x + spf[k] * f.h[k].y;
                    const float c1 = cf[k] * CPf[k] - sf[k] * SPf[k], s1 = sf[k] * CPf[k] + cf[k] * SPf[k];
                    const float c2 = cpf[k] * CPf[k] - spf[k] * SPf[k], s2 = spf[k] * CPf[k] + cpf[k] * SPf[k];
                    cf[k] = c1;
                    sf[k] = s1;
                    cpf[k] = c2;
                    spf[k] = s2;
                    qmf[k] *= qPf[k];
                }
                b32 = nb;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                G[k] += (double)Gf[k];
                H[k] += (double)Hf[k];
                J[k] += (double)Jf[k];
                KK[k] += (double)Kf[k];
            }
        }
    }
}

// Gravity in the Earth-fixed frame of K objects with the columns split over the P lanes of each object's
// group (lane l takes columns l, l + P, ...; P a power of two, or more than the columns); the per-object
// totals are added across the group.
template <bool MIXED, int K, bool PAIRS = false, class Team = WarpTeam>
__device__ __forceinline__ void gravity_itrs_team(const GravSmem& gs, const Team& team, const double (&x)[K],
    const double (&y)[K], const double (&z)[K], double (&ax)[K], double (&ay)[K], double (&az)[K])
{
    double ri[K], gr2[K], u[K], w[K], G[K], H[K], J[K], KK[K];
    LanePowers lp[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        ri[k] = inv_norm(x[k], y[k], z[k]);
        const double q = gs.radius * ri[k];
        u[k] = q * (z[k] * ri[k]);
        w[k] = q * q;
        gr2[k] = central(gs.gm, x[k], y[k], z[k], ri[k]); // here it hides behind the walk
        G[k] = H[k] = J[k] = KK[k] = 0.0;
        lp[k] = lane_powers(x[k] * ri[k], y[k] * ri[k], q, team.l, team.top(), team.P, team.P <= gs.L);
    }
    lane_walk<MIXED, K, PAIRS>(gs, team.l, team.P, gs.L, lp, u, w, G, H, J, KK);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        team.sum4(G[k], H[k], J[k], KK[k]);
        assemble_itrs(gr2[k], x[k], y[k], z[k], ri[k], G[k], H[k], J[k], KK[k], ax[k], ay[k], az[k]);
    }
}

template <bool MIXED, int K, bool PAIRS = false>
__device__ __forceinline__ void gravity_itrs_lk(const GravSmem& gs, int l, int P, const double (&x)[K],
    const double (&y)[K], const double (&z)[K], double (&ax)[K], double (&ay)[K], double (&az)[K],
    unsigned mask)
{
    gravity_itrs_team<MIXED, K, PAIRS>(gs, WarpTeam { l, P, mask }, x, y, z, ax, ay, az);
}

// K objects: GCRS positions r[k] with the ITRS<-GCRS matrix M of gravity_gcrs.
template <bool MIXED, int K, bool PAIRS = false, class Team = WarpTeam>
__device__ __forceinline__ void gravity_gcrs_team(const GravSmem& gs, const Team& team, const double (&m)[9],
    const double (&r)[K][3], double (&a)[K][3])
{
    double px[K], py[K], pz[K], ax[K], ay[K], az[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        px[k] = m[0] * r[k][0] + m[1] * r[k][1] + m[2] * r[k][2];
        py[k] = m[3] * r[k][0] + m[4] * r[k][1] + m[5] * r[k][2];
        pz[k] = m[6] * r[k][0] + m[7] * r[k][1] + m[8] * r[k][2];
    }
    gravity_itrs_team<MIXED, K, PAIRS>(gs, team, px, py, pz, ax, ay, az);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        a[k][0] = m[0] * ax[k] + m[3] * ay[k] + m[6] * az[k];
        a[k][1] = m[1] * ax[k] + m[4] * ay[k] + m[7] * az[k];
        a[k][2] = m[2] * ax[k] + m[5] * ay[k] + m[8] * az[k];
    }
}

template <bool MIXED, int K, bool PAIRS = false, class Team = WarpTeam>
__device__ __forceinline__ void gravity_gcrs_team(const GravSmem& gs, const Team& team,
    const double* __restrict__ M, const double (&r)[K][3], double (&a)[K][3])
{
    double m[9];
#pragma unroll
    for (int i = 0; i < 9; ++i)
        m[i] = __ldg(M + i);
    gravity_gcrs_team<MIXED, K, PAIRS>(gs, team, m, r, a);
}

template <bool MIXED, int K, bool PAIRS = false>
__device__ __forceinline__ void gravity_gcrs_lk(const GravSmem& gs, int l, int P, const double* __restrict__ M,
    const double (&r)[K][3], double (&a)[K][3], unsigned mask)
{
    gravity_gcrs_team<MIXED, K, PAIRS>(gs, WarpTeam { l, P, mask }, M, r, a);
}

} // namespace gpop
