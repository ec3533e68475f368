// frames_block.cuh -- one epoch's ITRS->GCRS matrix by a block of kFrameThreads threads (frames.cu, batch.cu).
#pragma once
#include "frames.cuh"
#include "kernels.h"

namespace gpop {

// The 2,414 nutation terms (IERS 2010 Tables 5.3a/b, both j = 0 and j = 1 series for longitude and obliquity) are
// split across the threads and combined in a fixed order; thread 0 then evaluates precession, GAST and the matrix
// chain. Bounds: the latency of an epoch, since most calls have few (a sine, a cosine and 14 products per term),
// then thread 0's chain. The tables of a call of 120 steps (80 + 125 epochs) took 208 us as two launches with a
// warp per epoch, 37 as one launch with four, and take 28 with the coefficients' division by the unit done when
// the table is loaded; 11,000 epochs of a batch 620 -> 590 us. Every epoch of every call is summed in the same order.
constexpr int kFrameThreads = 128;

__device__ __forceinline__ double series_part(const NutTerm* terms, int count, const double* F)
{
    double acc = 0.0;
    for (int i = threadIdx.x; i < count; i += kFrameThreads)
        acc += frames::nutation_term(terms[i], F);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// Writes M at m_out and the UTC MJD at mjd_out (may be NULL).
__device__ __forceinline__ void frames_epoch(const FrameData& fd, int y, int mo, int d, int hh, int mi, double sec,
    double* __restrict__ m_out, double* __restrict__ mjd_out)
{
    __shared__ double part[4][kFrameThreads / 32];
    // UTC MJD, EOP, UT1 and TT of this epoch (TimePointParamsKernel, time_points.cu:44-52)
    const double mjd_utc = frames::calendar_to_mjd(y, mo, d, hh, mi, sec);
    const double mjd_tt
        = mjd_utc + (frames::leap_at(fd.leap_mjd, fd.leap_val, fd.n_leap, mjd_utc) + frames::kTtTai) / 86400.0;
    const double t = (mjd_tt - frames::kMjdJ2000) / 36525.0;
    double F[14];
    frames::fundamental_args(t, F);
    const NutTerm* lon1 = fd.nut + fd.n_lon0;
    const NutTerm* obl0 = lon1 + fd.n_lon1;
    const NutTerm* obl1 = obl0 + fd.n_obl0;
    const double s[4] = { series_part(fd.nut, fd.n_lon0, F), series_part(lon1, fd.n_lon1, F),
        series_part(obl0, fd.n_obl0, F), series_part(obl1, fd.n_obl1, F) };
    if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 4; ++q)
            part[q][threadIdx.x >> 5] = s[q];
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum[4];
        for (int q = 0; q < 4; ++q) {
            sum[q] = 0.0;
            for (int w = 0; w < kFrameThreads / 32; ++w)
                sum[q] += part[q][w];
        }
        const EopRec eop = frames::eop_at(fd.eop, fd.n_eop, mjd_utc);
        const double mjd_ut1 = mjd_utc + eop.ut1 / 86400.0;
        double M[9];
        frames::assemble(t, F, sum[0] + sum[1] * t, sum[2] + sum[3] * t, mjd_ut1, mjd_tt, eop, M);
        for (int k = 0; k < 9; ++k)
            m_out[k] = M[k];
        if (mjd_out)
            *mjd_out = mjd_utc;
    }
}

} // namespace gpop
