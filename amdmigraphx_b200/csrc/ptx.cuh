// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 (TMEM alloc / mma / commit / ld) and the descriptor encoders they need.
// Only plain (non-multicast) TMA loads are used anywhere in this library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mgx {

// Status word written by kernels whose bounded waits expire.  One copy per
// translation unit (no relocatable device code is needed); the library's
// mgx_cuda_device_status() collects them through read_and_clear_status().
static __device__ unsigned int g_device_status;

static inline int read_and_clear_status(unsigned int* out)
{
    unsigned int v = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_device_status, sizeof(v));
    if(e != cudaSuccess)
        return static_cast<int>(e);
    if(v != 0)
    {
        e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(zero));
        if(e != cudaSuccess)
            return static_cast<int>(e);
    }
    *out = v;
    return 0;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool elect_one()
{
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(pred));
    return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    // Without a time hint: the hardware parks the thread for a while by itself.  With one (20 us) it polled, with a
    // sleep in between: twice the wait instructions, 15 % of what the int4 prompt kernel executed (512 rows of
    // 12288 x 4096: 50.2 us, without the hint 47.7).
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Bounded wait.  Returns true when the phase completed.  Gives up (false) when
// *abort_flag becomes non-zero or after limit_ns nanoseconds; in the second case
// it raises *abort_flag and records `code` in the device status word, so that
// every other role of the CTA leaves its own wait too and the kernel can free
// its tensor memory and return instead of hanging.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  volatile uint32_t* abort_flag, uint32_t code,
                                                  uint64_t limit_ns = 2000000000ull)
{
    if(mbar_try_wait(bar, parity))
        return true;
    uint64_t t0 = 0;
    for(uint32_t it = 0;; ++it)
    {
        if(mbar_try_wait(bar, parity))
            return true;
        if((it & 63u) == 63u)
        {
            if(*abort_flag != 0)
                return false;
            uint64_t now = globaltimer_ns();
            if(t0 == 0)
                t0 = now;
            else if(now - t0 > limit_ns)
            {
                *abort_flag = code;
                atomicCAS(&g_device_status, 0u, code);
                return false;
            }
        }
    }
}

// The same for a whole warp, with one answer for all its lanes.  The roles that issue TMA requests and
// tcgen05 instructions run their loops as whole warps and elect a lane only around the instructions:
// loop counters, addresses and descriptors are then uniform to the compiler, which the operands of
// those instructions have to be.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t code)
{
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag, code)) != 0;
}

// The same wait on a barrier that other CTAs of the cluster arrive on: what they wrote to their
// shared memory before arriving is visible after it.
__device__ __forceinline__ bool mbar_wait_cluster_bounded(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                                          uint32_t code, uint64_t limit_ns = 2000000000ull)
{
    uint64_t t0 = 0;
    for(uint32_t it = 0;; ++it)
    {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(smem_u32(bar)), "r"(parity)
                     : "memory");
        if(ok != 0)
            return true;
        if((it & 63u) == 63u)
        {
            if(*abort_flag != 0)
                return false;
            const uint64_t now = globaltimer_ns();
            if(t0 == 0)
                t0 = now;
            else if(now - t0 > limit_ns)
            {
                *abort_flag = code;
                atomicCAS(&g_device_status, 0u, code);
                return false;
            }
        }
    }
}

// Arrive on the barrier at the same place in CTA `rank` of the cluster.
__device__ __forceinline__ void cluster_arrive(uint64_t* bar, uint32_t rank)
{
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\t"
                 "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(smem_u32(bar)),
                 "r"(rank)
                 : "memory");
}

// The value at the same place in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_load(const void* p, uint32_t rank)
{
    uint32_t v;
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.u32 %0, [r];\n\t}"
                 : "=r"(v)
                 : "r"(smem_u32(p)), "r"(rank)
                 : "memory");
    return v;
}

__device__ __forceinline__ uint4 cluster_load_uint4(const void* p, uint32_t rank)
{
    uint4 v;
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %4, %5;\n\t"
                 "ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [r];\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(smem_u32(p)), "r"(rank)
                 : "memory");
    return v;
}

__device__ __forceinline__ void cluster_load4(const float* p, uint32_t rank, float (&v)[4])
{
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %4, %5;\n\t"
                 "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [r];\n\t}"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(smem_u32(p)), "r"(rank)
                 : "memory");
}

// Barriers of whole warps (.aligned): the lanes of a warp have to execute one together, which after code that divided
// them is only sure behind __syncwarp().
__device__ __forceinline__ void cluster_barrier_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_barrier_wait()
{
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Every thread of the cluster's CTAs passes both halves.
__device__ __forceinline__ void cluster_barrier()
{
    cluster_barrier_arrive();
    cluster_barrier_wait();
}

// ---------------------------------------------------------------- programmatic dependent launch
// A kernel launched with cudaLaunchAttributeProgrammaticStreamSerialization may start while the
// previous kernel of its stream still runs; it must call grid_dependency_wait() before it reads
// anything that kernel writes, and before it writes anything that kernel may still read.  The
// wait returns at once when the kernel was launched without the attribute.
__device__ __forceinline__ void grid_dependency_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Allows the next kernel of the stream (if it was launched with the attribute) to start now; without it that
// kernel starts when this one is complete and its results can be seen.  The int4 decode linears request packed
// weights before they wait: kernels whose results packed weights may be (8-bit integers, mgx_cuda.h) do not call it.
__device__ __forceinline__ void grid_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The two together, first thing in a short kernel: its successor may take up its place on the SMs at
// once, and nothing is touched before the predecessor is done.
__device__ __forceinline__ void grid_chain()
{
    grid_launch_dependents();
    grid_dependency_wait();
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// 3-D tiled load global -> shared, completion on an mbarrier.  c0 is the
// innermost coordinate (elements); c0 * element size must be a multiple of 16 B.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int32_t c0, int32_t c1, int32_t c2)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1),
                 "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int32_t c0, int32_t c1)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
                 : "memory");
}

// 3-D tiled store shared -> global (bulk async-group completion).  Elements of the box
// that fall outside the tensor are not written.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem_src,
                                             int32_t c0, int32_t c1, int32_t c2)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::
                     "l"(reinterpret_cast<uint64_t>(map)),
                 "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(smem_slot)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before_sync()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after_sync()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Arrive on an mbarrier when all tcgen05.mma issued so far by this thread finish.
__device__ __forceinline__ void tc_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::
                     "r"(smem_u32(bar))
                 : "memory");
}

// D[tmem] (+)= A[smem] * B[smem], 8-bit integer operands, int32 accumulate.
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                       uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// Same with the A operand read from tensor memory (row i of A in lane i, four K bytes per
// 32-bit column) instead of shared memory.
__device__ __forceinline__ void mma_i8_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                              uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// Registers -> tensor memory: lane = the warp's lane quarter * 32 + thread lane, 32 columns.
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void tmem_st_wait()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// fp8 (e4m3/e5m2) operands, fp32 accumulate.
__device__ __forceinline__ void mma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                       uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// fp16 / bf16 operands, fp32 accumulate.
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                        uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// Same with the A operand in tensor memory (row i in lane i, two K elements per 32-bit column).
__device__ __forceinline__ void mma_f16_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives
// lane (base_lane + t), columns col .. col+31.  A warp may only touch the lane
// quarter (warp_id % 4) * 32 .. +31.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// Same shape, 16 columns.
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// Narrow forms of the same shape: 2, 4 and 8 columns.
__device__ __forceinline__ void tmem_ld_32x32b_x2(uint32_t taddr, uint32_t (&r)[2])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld_32x32b_x4(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// N columns (2, 4, 8, 16 or 32) of the warp's lane quarter.
template <int N>
__device__ __forceinline__ void tmem_ld_32x32b(uint32_t taddr, uint32_t (&r)[N])
{
    static_assert(N == 2 or N == 4 or N == 8 or N == 16 or N == 32, "unsupported width");
    if constexpr(N == 2)
        tmem_ld_32x32b_x2(taddr, r);
    else if constexpr(N == 4)
        tmem_ld_32x32b_x4(taddr, r);
    else if constexpr(N == 8)
        tmem_ld_32x32b_x8(taddr, r);
    else if constexpr(N == 16)
        tmem_ld_32x32b_x16(taddr, r);
    else
        tmem_ld_32x32b_x32(taddr, r);
}

// Two floats -> packed half2 with round-toward-zero (lo in the low half).
__device__ __forceinline__ uint32_t cvt_rz_f16x2(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ void tmem_ld_wait()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------------- pairs of CTAs (cta_group::2)
// The two CTAs of a cluster of two work on one accumulator of 256 rows: CTA r holds rows 128 r .. 128 r + 127 of D in
// its own tensor memory, and in its own shared memory the same rows of A and the r-th half of the rows of B, at the
// same offsets as the other.  CTA 0 issues.  Allocation and release take a warp of each.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Into this CTA's shared memory, completion on CTA 0's barrier (the one at the same place as `bar`).
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int32_t c0, int32_t c1,
                                                 int32_t c2)
{
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %2, 0;\n\t"
                 "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
                 " [%0], [%1, {%3, %4, %5}], [r];\n\t}" ::"r"(smem_u32(smem_dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

// Arrive on the barrier of both CTAs when all tcgen05.mma issued so far by this thread finish.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar)
{
    const uint16_t both = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "h"(both)
                 : "memory");
}

#define MGX_MMA_PAIR(NAME, KIND)                                                                                       \
    __device__ __forceinline__ void NAME(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,            \
                                         uint32_t accumulate)                                                          \
    {                                                                                                                  \
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"                                               \
                     "tcgen05.mma.cta_group::2.kind::" KIND " [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),                \
                     "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)                                             \
                     : "memory");                                                                                      \
    }
MGX_MMA_PAIR(mma_i8_pair, "i8")
MGX_MMA_PAIR(mma_f8_pair, "f8f6f4")
MGX_MMA_PAIR(mma_f16_pair, "f16")
#undef MGX_MMA_PAIR

// ------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor for a K-major operand tile stored as rows of
// 128 bytes with the 128-byte swizzle (what a TMA box {128 B, rows} with
// CU_TENSOR_MAP_SWIZZLE_128B writes): 8-row groups are 1024 B apart (stride
// byte offset), the leading byte offset is unused for swizzled K-major layouts.
// Bits: [0,14) start>>4, [16,30) LBO>>4, [32,46) SBO>>4, [46,48) version = 1,
// [49,52) base offset (0: tiles are 1024-B aligned), [61,64) layout 2 = SWIZZLE_128B.
__host__ __device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// Instruction descriptor (kind::i8 / f8f6f4 / f16): [4,6) D format (0 f16, 1 f32,
// 2 s32), [7,10) A format, [10,13) B format, bit 15 / 16 A / B major (0 = K-major),
// [17,23) N>>3, [24,29) M>>4.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t d_fmt, uint32_t a_fmt, uint32_t b_fmt,
                                                  uint32_t m, uint32_t n)
{
    return (d_fmt << 4) | (a_fmt << 7) | (b_fmt << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

} // namespace mgx
