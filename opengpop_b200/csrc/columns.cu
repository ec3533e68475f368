// columns.cu -- GJ8 steps of many objects per SM with the gravity columns split over a block's warps.
//
// A block of 8 warps, one per SM, carries up to 512 objects in sets of 64. Every evaluation goes set by set:
// a lane takes two objects of the set and each warp walks its own range of columns for all 64 of them, the
// eight totals of an object are added through shared memory, and the thread that owns the object assembles
// the acceleration and corrects. So
// - a table entry is read once per warp and broadcast to 64 objects (lanes that walk different columns read
//   one entry each);
// - all warps have the same work whatever the number of objects (two objects per thread fill 8 warps at 512
//   objects per SM only, and at 64 objects per SM one);
// - a set whose objects are all done takes no part in the next corrector pass.
// What is left of a set (rem <= 32 objects per block) gives its pairs of objects P = 2, 4, 8 or 16 lanes of a
// warp each, whose columns m, m + P, ... lie next to each other and so are nearly as long.
// An object's corrector state lies in shared memory for up to 64 objects per block, else in its state arrays
// (L2): nothing of it is held through the walks, which have the registers to themselves.
//
// Bounds: dependent FMAs with two warps per scheduler, then the FP64 (mixed: FMA) pipe. Captured at 70x70, FP64: 17
// objects per SM (the pair's lanes) FP64 pipe 52 % busy, shared-memory loads 37 % of their port, waits per issued
// instruction 1.35 on fixed latency, 0.87 at barriers, 0.70 on the pipe; 64 and 128 per SM 62 % and 63 %, 46 %, 1.3,
// 0.3 to 0.5, 0.85; mixed at 128 per SM FMA pipe 30 %, 40 %. Measured on B200, 70x70 FP64 / mixed, us per step
// against the best of the other walks: 2,368 objects 18.6 / 15.3 (24.7 / 19.4), 9,472: 40.6 / 25.1 (51.5 / 42.0),
// 18,944: 78.7 / 45.7 (91 / 66), 37,888: 152 / 87 (156 / 96); two evaluations of a set take 70,500 of its 80,300
// cycles. From 6 sets on, two objects per thread are as good or better: no barriers there.
#include "common.cuh"
#include "corrector.cuh"
#include "gj8_tables.cuh"
#include "gravity.cuh"
#include "kernels.h"
#include "lanes.cuh"

#include <algorithm>

namespace gpop {

namespace {

constexpr int kWarps = kColumnWarps;
constexpr int kBlock = 32 * kWarps;
constexpr int kSet = 64;

// An object's values, array i at base[i * stride]: the state arrays, with s2, s1 and the acceleration of a
// finished object from `work` on.
struct Desk {
    double* base;
    int64_t stride;
    int work;
    __device__ __forceinline__ double& at(int i) const { return base[i * stride]; }
};
constexpr int kDeskArrays = kHist + 27 + 9; // in shared memory: r, v, s, S, history, then the work values

// Walk of a range of columns for the objects of a set; start values q, u, C1, S1 and totals G, H, J, K.
template <bool MIXED>
__device__ __forceinline__ void walk_two(const GravSmem& g, int m0, int m1, const WalkStart& ws, SplitTotals& t)
{
    LanePowers p[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
        p[k] = lane_powers(ws.C1[k], ws.S1[k], ws.q[k], m0, m0 - 1, 1, false);
    auto set = [&](auto& W) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            W.Cm[k] = p[k].Cm;
            W.Sm[k] = p[k].Sm;
            W.Cp[k] = p[k].Cp;
            W.Sp[k] = p[k].Sp;
            W.qm[k] = p[k].qm;
        }
    };
    auto get = [&](const auto& W) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            t.G[k] = W.G[k];
            t.H[k] = W.H[k];
            t.J[k] = W.J[k];
            t.K[k] = W.KK[k];
        }
    };
    if constexpr (MIXED) {
        MixedWalk2<true, kSplitPairUnroll> W(g, ws);
        set(W);
        walk_groups(W, m0, m1 - 1);
        get(W);
    } else {
        PairWalk64<true, 2> W(g, ws);
        set(W);
        W.walk(m0, m1);
        get(W);
    }
}

// full: sets of 64 objects per block; rem: objects of its last set (P lanes per pair of them, plan kind). Object k of set s of block
// b is lo + (s grid + b) 64 + k, object k of the last set lo + 64 full grid + b rem + k. bufs: buffers of
// warp totals; local: the desks lie in shared memory.
struct ColumnArgs {
    int full = 0, rem = 0, P = 1, kind = 0, bufs = 1;
    bool local = false;
};

template <bool MIXED>
__global__ void __launch_bounds__(kBlock, 1) gj8_columns_kernel(TableSrc ts, PropArgs a, ColumnPlan plan, ColumnArgs c)
{
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ unsigned need[2]; // sets with objects that are not done, for even and odd passes
    GravSmem g;
    if (!bind_lane_table(smem, ts, a.err, g))
        return;
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t n = a.n, lo = a.obj_lo, hi = a.obj_hi < 0 ? n : a.obj_hi;
    const int o = c.full * kSet + c.rem; // objects of this block
    const int pad = c.full * kSet + (c.rem ? 32 : 0);
    const int sets = c.full + (c.rem ? 1 : 0);
    // start values, then totals, of every object; totals of each warp for one set; desks
    double* xs = reinterpret_cast<double*>(smem + stage_offset(ts));
    double* part = xs + 4 * pad;
    double* desks = part + c.bufs * kWarps * 4 * kSet;
    auto object = [&](int j) -> int64_t {
        const int s = j / kSet;
        const int64_t i = s < c.full ? ((int64_t)s * gridDim.x + blockIdx.x) * kSet + (j - s * kSet)
                                     : (int64_t)c.full * kSet * gridDim.x + (int64_t)blockIdx.x * c.rem + (j - c.full * kSet);
        return lo + i;
    };
    auto desk = [&](int j, int64_t obj) -> Desk {
        return c.local ? Desk { desks + j, o, kHist + 27 } : Desk { a.state + obj, n, kX0 };
    };
    for (int j = tid; j < pad; j += kBlock) { // idle places walk something harmless
        xs[j] = 0.5;
        xs[pad + j] = 0.0;
        xs[2 * pad + j] = 1.0;
        xs[3 * pad + j] = 0.0;
    }
    if (c.local)
        for (int j = tid; j < o; j += kBlock) {
            const int64_t obj = object(j);
            if (obj < hi)
                for (int i = 0; i < kHist + 27; ++i)
                    desks[i * o + j] = a.state[i * n + obj];
        }
    const double h = a.h;
    for (int step = a.step_begin; step < a.step_end; ++step) {
        const int64_t t = step - a.traj_step0;
        auto trajectory = [&](int64_t obj, const double (&r)[3], const double (&v)[3], const double (&ae)[3]) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                if (a.traj_r)
                    a.traj_r[(t * 3 + j) * n + obj] = r[j];
                if (a.traj_v)
                    a.traj_v[(t * 3 + j) * n + obj] = v[j];
                if (a.traj_a)
                    a.traj_a[(t * 3 + j) * n + obj] = ae[j];
            }
        };
        if (step <= 4) {
            for (int j = tid; j < o; j += kBlock) {
                const int64_t obj = object(j);
                if (obj >= hi)
                    continue;
                const Desk d = desk(j, obj);
                const double* st = a.state + obj;
                double r[3], v[3], ae[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    r[k] = st[(kRep + (step - 1) * 6 + k) * n];
                    v[k] = st[(kRep + (step - 1) * 6 + 3 + k) * n];
                    ae[k] = st[(kRepA + (step - 1) * 3 + k) * n];
                    d.at(kR + k) = r[k];
                    d.at(kV + k) = v[k];
                }
                trajectory(obj, r, v, ae);
            }
            continue;
        }
        const int ring0 = (step - 5) % 9;
        const double* M = a.prop_m + (size_t)(step + 4) * 9;
        unsigned done = 0, fast = 0; // bits of this thread's objects j = tid, tid + 256
        // start values of an evaluation at r
        auto start = [&](int j, const double (&r)[3]) {
            const double x = __ldg(M + 0) * r[0] + __ldg(M + 1) * r[1] + __ldg(M + 2) * r[2];
            const double y = __ldg(M + 3) * r[0] + __ldg(M + 4) * r[1] + __ldg(M + 5) * r[2];
            const double z = __ldg(M + 6) * r[0] + __ldg(M + 7) * r[1] + __ldg(M + 8) * r[2];
            const double ri = inv_norm(x, y, z), q = g.radius * ri;
            xs[j] = q;
            xs[pad + j] = q * (z * ri);
            xs[2 * pad + j] = x * ri;
            xs[3 * pad + j] = y * ri;
        };
        for (int j = tid, b = 0; j < o; j += kBlock, ++b) {
            const int64_t obj = object(j);
            if (obj >= hi) {
                done |= 1u << b;
                continue;
            }
            const Desk d = desk(j, obj);
            double r[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) { // as gj8_kernel
                double q[9];
#pragma unroll
                for (int i = 0; i < 9; ++i) {
                    int slot = ring0 + i;
                    slot -= slot >= 9 ? 9 : 0;
                    q[i] = d.at(kHist + slot * 3 + k);
                }
                double rt = 0.0, c1 = 0.0, c2 = 0.0;
#pragma unroll
                for (int i = 0; i < 9; ++i)
                    rt = fma(q[i], c_GJ[9][i], rt);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    c1 = fma(q[i + 1], c_SA[8][i], c1);
                    c2 = fma(q[i + 1], c_GJ[8][i], c2);
                }
                const double S = d.at(kSb + k) + (d.at(kSs + k) + q[8] / 2);
                r[k] = (rt + S) * h * h;
                d.at(kSb + k) = S;
                d.at(kR + k) = r[k];
                d.at(d.work + k) = c2;
                d.at(d.work + 3 + k) = c1;
            }
            start(j, r);
        }
        if (tid == 0) {
            need[0] = (1u << sets) - 1u;
            need[1] = 0;
        }
        int buf = 0;
        for (int it = 0; it < a.ncorr; ++it) {
            __syncthreads(); // start values and the sets that need them
            const unsigned mask = need[it & 1];
            if (mask == 0)
                break; // the same for every thread
            for (int s = 0; s < sets; ++s) {
                if (!(mask >> s & 1))
                    continue;
                double* mine = part + (buf * kWarps + warp) * 4 * kSet;
                if (s < c.full) {
                    const double* x = xs + s * kSet + lane;
                    WalkStart ws;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        ws.q[k] = x[32 * k];
                        ws.u[k] = x[pad + 32 * k];
                        ws.w[k] = ws.q[k] * ws.q[k];
                        ws.C1[k] = x[2 * pad + 32 * k];
                        ws.S1[k] = x[3 * pad + 32 * k];
                    }
                    SplitTotals p;
                    walk_two<MIXED>(g, plan.b[0][warp], plan.b[0][warp + 1], ws, p);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        mine[lane + 32 * k] = p.G[k];
                        mine[kSet + lane + 32 * k] = p.H[k];
                        mine[2 * kSet + lane + 32 * k] = p.J[k];
                        mine[3 * kSet + lane + 32 * k] = p.K[k];
                    }
                } else {
                    const int per = 32 / c.P, l = lane / per; // pairs of objects, this lane of a pair's
                    const double* x = xs + c.full * kSet + lane % per;
                    const int m0 = plan.b[c.kind][warp], m1 = plan.b[c.kind][warp + 1];
                    double u[2], w[2], G[2] = { 0.0, 0.0 }, H[2] = { 0.0, 0.0 }, J[2] = { 0.0, 0.0 }, K[2] = { 0.0, 0.0 };
                    LanePowers lp[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const double q = x[per * k];
                        u[k] = x[pad + per * k];
                        w[k] = q * q;
                        lp[k] = lane_powers(x[2 * pad + per * k], x[3 * pad + per * k], q, m0 + l, m0 + c.P - 2, c.P,
                            m0 + c.P < m1);
                    }
                    lane_walk<MIXED, 2, true>(g, m0 + l, c.P, m1 - 1, lp, u, w, G, H, J, K);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        for (int d = per; d < 32; d <<= 1) { // over the lanes of the pair
                            G[k] += __shfl_xor_sync(0xffffffffu, G[k], d);
                            H[k] += __shfl_xor_sync(0xffffffffu, H[k], d);
                            J[k] += __shfl_xor_sync(0xffffffffu, J[k], d);
                            K[k] += __shfl_xor_sync(0xffffffffu, K[k], d);
                        }
                        if (l == 0) {
                            double* to = mine + k * per + lane;
                            to[0] = G[k];
                            to[kSet] = H[k];
                            to[2 * kSet] = J[k];
                            to[3 * kSet] = K[k];
                        }
                    }
                }
                __syncthreads(); // the set's totals of every warp; its start values are free
                const double* all = part + buf * kWarps * 4 * kSet;
                const int k = tid & (kSet - 1), v = tid / kSet;
                if (s < c.full || k < kSet / c.P) {
                    double sum = 0.0;
#pragma unroll
                    for (int w = 0; w < kWarps; ++w)
                        sum += all[(w * 4 + v) * kSet + k];
                    xs[v * pad + s * kSet + k] = sum;
                }
                buf = c.bufs > 1 ? buf ^ 1 : 0;
                if (c.bufs == 1 && s + 1 < sets)
                    __syncthreads(); // one buffer: its readers finish before it is written again
            }
            if (tid == 0)
                need[(it + 1) & 1] = 0; // (its last readers passed the barriers of a set since)
            __syncthreads(); // totals of every set
            unsigned more = 0;
            for (int j = tid, b = 0; j < o; j += kBlock, ++b) {
                if (done >> b & 1)
                    continue;
                const Desk d = desk(j, object(j));
                double r[3], s2[3], S[3], a8[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    r[k] = d.at(kR + k);
                    S[k] = d.at(kSb + k);
                    s2[k] = d.at(d.work + k);
                }
                {
                    const double x = __ldg(M + 0) * r[0] + __ldg(M + 1) * r[1] + __ldg(M + 2) * r[2];
                    const double y = __ldg(M + 3) * r[0] + __ldg(M + 4) * r[1] + __ldg(M + 5) * r[2];
                    const double z = __ldg(M + 6) * r[0] + __ldg(M + 7) * r[1] + __ldg(M + 8) * r[2];
                    const double ri = inv_norm(x, y, z);
                    double ax, ay, az;
                    assemble_itrs(central(g.gm, x, y, z, ri), x, y, z, ri, xs[j], xs[pad + j], xs[2 * pad + j], xs[3 * pad + j],
                        ax, ay, az);
                    a8[0] = __ldg(M + 0) * ax + __ldg(M + 3) * ay + __ldg(M + 6) * az;
                    a8[1] = __ldg(M + 1) * ax + __ldg(M + 4) * ay + __ldg(M + 7) * az;
                    a8[2] = __ldg(M + 2) * ax + __ldg(M + 5) * ay + __ldg(M + 8) * az;
                }
                bool f = (fast >> b & 1) != 0;
                const bool end = correct_position(ts.corr, h, it, a.ncorr, s2, S, a8, r, f);
                fast = f ? fast | 1u << b : fast & ~(1u << b);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    d.at(kR + k) = r[k];
                    if (end)
                        d.at(d.work + 6 + k) = a8[k];
                }
                if (end) {
                    done |= 1u << b;
                } else {
                    start(j, r);
                    more |= 1u << (j < c.full * kSet ? j / kSet : c.full);
                }
            }
            more = __reduce_or_sync(0xffffffffu, more);
            if (lane == 0 && more)
                atomicOr(&need[(it + 1) & 1], more);
        }
        // the finished step
        for (int j = tid; j < o; j += kBlock) {
            const int64_t obj = object(j);
            if (obj >= hi)
                continue;
            const Desk d = desk(j, obj);
            double r[3], v[3], a8[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                a8[k] = d.at(d.work + 6 + k);
                const double s = d.at(kSs + k) + (a8[k] + d.at(kHist + (ring0 + 8 - (ring0 > 0 ? 9 : 0)) * 3 + k)) / 2;
                d.at(kSs + k) = s;
                v[k] = h * (d.at(d.work + 3 + k) + a8[k] * c_SA[8][8] + s);
                d.at(kV + k) = v[k];
                d.at(kHist + ring0 * 3 + k) = a8[k];
                r[k] = d.at(kR + k);
            }
            trajectory(obj, r, v, a8);
        }
        __syncthreads(); // every thread has read the last `need` before the next step sets it
    }
    for (int j = tid; j < o; j += kBlock) {
        const int64_t obj = object(j);
        if (obj >= hi)
            continue;
        if (c.local)
            for (int i = 0; i < kHist + 27; ++i)
                a.state[i * n + obj] = desks[i * o + j];
        const Desk d = desk(j, obj);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (a.out_r)
                a.out_r[obj * 3 + k] = d.at(kR + k);
            if (a.out_v)
                a.out_v[obj * 3 + k] = d.at(kV + k);
        }
    }
}

} // namespace

cudaError_t launch_gj8_columns(const TableSrc& lanes, const PropArgs& a, int num_sms, cudaStream_t s)
{
    const int64_t lo = a.obj_lo, hi = a.obj_hi < 0 ? a.n : a.obj_hi, cnt = hi - lo;
    if (cnt <= 0 || cnt > (int64_t)num_sms * 512)
        return cudaErrorInvalidValue;
    const int per = (int)((cnt + num_sms - 1) / num_sms);
    ColumnArgs c;
    c.full = per / kSet;
    c.rem = per % kSet;
    if (c.rem > 32) {
        ++c.full;
        c.rem = 0;
    }
    c.kind = c.rem > 16 ? 1 : c.rem > 8 ? 2 : c.rem > 4 ? 3 : 4;
    c.P = 1 << c.kind;
    const int o = c.full * kSet + c.rem, pad = c.full * kSet + (c.rem ? 32 : 0);
    // two buffers of totals where they fit beside the table and the start values
    const size_t base = stage_offset(lanes) + (size_t)4 * pad * 8, buf = (size_t)kWarps * 4 * kSet * 8;
    const size_t limit = max_smem_optin() - 64; // (need[] is static)
    c.bufs = c.full + (c.rem ? 1 : 0) > 1 && base + 2 * buf <= limit ? 2 : 1;
    size_t bytes = base + c.bufs * buf;
    const size_t desks = (size_t)kDeskArrays * o * 8;
    c.local = bytes + desks <= limit;
    if (c.local)
        bytes += desks;
    const unsigned grid = (unsigned)std::min<int64_t>(num_sms, (cnt + o - 1) / o);
    const ColumnPlan& plan = lanes.plan;
    cudaError_t e;
    if (lanes.mixed) {
        if ((e = cudaFuncSetAttribute(gj8_columns_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) != cudaSuccess)
            return e;
        gj8_columns_kernel<true><<<grid, kBlock, bytes, s>>>(lanes, a, plan, c);
    } else {
        if ((e = cudaFuncSetAttribute(gj8_columns_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) != cudaSuccess)
            return e;
        gj8_columns_kernel<false><<<grid, kBlock, bytes, s>>>(lanes, a, plan, c);
    }
    return cudaGetLastError();
}

} // namespace gpop
