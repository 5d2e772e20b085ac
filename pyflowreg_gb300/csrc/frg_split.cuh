// Parts of the split chained SOR (k_sor_split, frg_split_sor.cuh): the work of 32 rows
// is divided among update warps (one per pipelined iteration), fold warps that run
// ahead of them and one warp that waits for both and for the neighbouring CTAs.
//
// Every wait is bounded: a wait that runs out is given up, and so is every later
// one of that warp, so that the kernel ends; the frame's result is then NaN.
#pragma once

#include "frg_internal.h"
#include "frg_split_schedule.h"

#include <cooperative_groups.h>

namespace frg {

namespace {

constexpr unsigned kMaxTries = 500000u;  // tries of a wait, of at most 2 us each

constexpr int kPkZero = 1, kPkTick = 2, kPkCoef = 4, kPkStore = 8;

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned mb, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mb), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned mb)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.release.cta.shared::cta.b64 t, [%0];\n\t}" ::"r"(mb) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned mb, unsigned bytes)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.relaxed.cta.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(mb),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect(unsigned mb, unsigned bytes)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.release.cta.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(mb),
                 "r"(bytes)
                 : "memory");
}

// A word into the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ void st_cluster(unsigned addr, int rank, int v)
{
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.b32 [a], %2;\n\t}" ::"r"(addr), "r"(rank),
                 "r"(v)
                 : "memory");
}

// 16 bytes into another CTA's shared memory, counted by a barrier there.  A
// predicated instruction: a branch around it costs the step about 50 clocks.
__device__ __forceinline__ void st_async_if(bool p, unsigned addr, int4 v, unsigned mb)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %6, 0;\n\t"
                 "@p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n\t}" ::"r"(addr),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mb), "r"((int)p)
                 : "memory");
}

__device__ __forceinline__ void st_async_if(bool p, unsigned addr, double2 v, unsigned mb)
{
    st_async_if(p, addr, *reinterpret_cast<const int4*>(&v), mb);
}

__device__ __forceinline__ void st_async_if(bool p, unsigned addr, float2 v, unsigned mb)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t"
                 "@p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];\n\t}" ::"r"(addr),
                 "r"(__float_as_int(v.x)), "r"(__float_as_int(v.y)), "r"(mb), "r"((int)p)
                 : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned mb, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 2000;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(mb), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Waits for the phase with this parity to complete.  After one wait has run
// out no further one is made.
__device__ __forceinline__ void mbar_wait(unsigned mb, unsigned parity, bool& dead)
{
    if (dead) return;
    for (unsigned i = 0; i < kMaxTries; ++i)
        if (mbar_test(mb, parity)) return;
    dead = true;
}

// Which warp does what.  Warp i runs on scheduler i % 4, and with five update
// warps two share one: that scheduler gets the waiting warp besides and no fold
// (one idle warp fills its place when there are more than six).
template <int M, int NU, int FC>
struct SplitRoles {
    static constexpr int WU = M * NU;
    static constexpr bool spread = M == 1 && NU == 5 && FC >= 3;  // warp 8 waits: it has to be there
    static constexpr int wait = spread ? 8 : WU;
    static constexpr int idle = spread && FC > 6 ? 12 : -1;
    static constexpr int warps = WU + 1 + M * FC + (idle >= 0 ? 1 : 0);
    static_assert(FC >= 1 && NU >= 1 && NU <= kGMax && wait < warps && idle < warps && warps <= 32, "every role has its warps");
    __device__ static int fold(int warp) { return spread ? warp - (warp < 8 ? 5 : (warp < 12 ? 6 : 7)) : warp - WU - 1; }
};

}  // namespace

}  // namespace frg
