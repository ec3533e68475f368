// common.cuh -- device constants and helpers shared by the propagation and screening kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gpop {

// gpop_config.flags bit (GPOP_MIXED_COMPENSATED in gpop.h): compensated FP32 sums in mixed mode.
constexpr unsigned kFlagMixedCompensated = 1u << 3;

// Error bits a kernel may raise in the context's device error word.
enum : unsigned {
    kErrTmaTimeout = 1u, // the bounded wait on the gravity-table bulk copy gave up
    kErrBadInput = 2u, // a state with a non-finite component, or a position at the origin
    kErrTmaUnfinished = 4u, // a staging copy had still not landed when its block gave up and left
};

// first_spins of stage_to_smem with this bit set: warp (first_spins without it) polls not once, the
// others as usual (a test setting).
constexpr uint32_t kWaitOneWarp = 1u << 31;

// ---- bulk-copy (TMA, cp.async.bulk) staging of a read-only table into shared memory ----
__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Copies `bytes` (multiple of 16, both addresses 16-byte aligned) from global to shared memory with
// one elected thread issuing cp.async.bulk chunks that complete on an mbarrier. Every thread of the
// block waits with a bounded spin of first_spins polls; a thread whose polls run out raises
// kErrTmaTimeout and waits a second bounded time for the copies still in flight (kErrTmaUnfinished if
// they have not landed by then either: the caller's results are void). The copy may land between the
// last polls of two warps, so the answer is the block's: false in every thread as soon as one gave up.
// A block that returns on it leaves as one, and no barrier or full-warp exchange behind it waits for
// threads that have left. Every thread of the block makes the call.
__device__ __forceinline__ bool stage_to_smem(void* smem_dst, const void* gsrc, uint32_t bytes,
    uint64_t* mbar, unsigned* err_word, uint32_t first_spins)
{
    const uint32_t bar = smem_u32(mbar);
    if (first_spins & kWaitOneWarp)
        first_spins = (threadIdx.x >> 5) == (first_spins & ~kWaitOneWarp) ? 0u : 1u << 22;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                     : "memory");
        const uint32_t chunk = 32768u;
        uint32_t dst = smem_u32(smem_dst);
        const char* src = static_cast<const char*>(gsrc);
        for (uint32_t off = 0; off < bytes; off += chunk) {
            uint32_t len = (bytes - off) < chunk ? (bytes - off) : chunk;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                         "[%0], [%1], %2, [%3];" ::"r"(dst + off),
                         "l"(src + off), "r"(len), "r"(bar)
                         : "memory");
        }
    }
    // bounded wait on phase 0 (about a second at the sleep below before giving up)
    uint32_t done = 0;
    for (uint32_t it = 0; it < first_spins && !done; ++it) {
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
                     " selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(bar)
                     : "memory");
        if (!done)
            __nanosleep(64);
    }
    const bool in_time = done != 0;
    if (!in_time) {
        atomicOr(err_word, kErrTmaTimeout);
        // give the copies in flight a second bounded window before the block leaves
        for (int it = 0; it < (1 << 22) && !done; ++it) {
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
                         " selp.u32 %0, 1, 0, p;\n}"
                         : "=r"(done)
                         : "r"(bar)
                         : "memory");
            if (!done)
                __nanosleep(64);
        }
        if (!done)
            atomicOr(err_word, kErrTmaUnfinished);
    }
    return __syncthreads_and(in_time) != 0;
}

// Stores and loads of per-thread values parked in shared memory across a long computation. The
// asm keeps the compiler from forwarding the stored value (which would keep it in a register).
__device__ __forceinline__ void st_stage(double* p, double v)
{
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(smem_u32(p)), "d"(v) : "memory");
}
__device__ __forceinline__ double ld_stage(const double* p)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}

// Whether two values have the same bit pattern (NaN equals itself, +0 differs from -0).
__device__ __forceinline__ bool same_bits(double a, double b)
{
    return __double_as_longlong(a) == __double_as_longlong(b);
}

} // namespace gpop
