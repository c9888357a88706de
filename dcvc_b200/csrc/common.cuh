// Shared device/host helpers for the sm_100a kernels of dcvc_b200.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef DCVC_HOST_DEVICE
#define DCVC_HOST_DEVICE __host__ __device__ __forceinline__
#endif

namespace dcvc {

// Error flag slots written by kernels whose bounded waits gave up.  The host reads them after a
// synchronisation point (dcvc_check_device_errors); a non-zero slot turns into an error status.
enum DeviceError : int {
    kErrNone = 0,
    kErrGemmProducerTimeout = 1,
    kErrGemmMmaTimeout = 2,
    kErrGemmEpilogueTimeout = 3,
};

// One global word per device holds the first error seen (see errors.cu).
__device__ __forceinline__ void report_error(int* flag, int code)
{
    if (flag != nullptr) {
        atomicCAS(flag, 0, code);
    }
}

// ---------------------------------------------------------------- programmatic dependent launch
//
// Kernels are launched with programmatic stream serialisation: a kernel may start while its
// predecessor in the stream drains.  Each kernel signals early that its dependents may launch and
// waits for the full completion (and memory flush) of its predecessor before touching any data
// the predecessor produces.

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void griddep_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------- shared-memory helpers

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16 bytes of shared memory by address: pointers into the aligned dynamic buffer are generic to the
// compiler.
__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// The same for data that nothing writes while `addr` is known: free to move and to be issued early.
__device__ __forceinline__ float4 lds128_const(uint32_t addr)
{
    float4 v;
    asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

__device__ __forceinline__ void sts128(uint32_t addr, uint4 v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// 32 bytes to 32-byte aligned global memory.
__device__ __forceinline__ void st_global_256(void* p, const uint32_t (&r)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// ---------------------------------------------------------------- mbarrier (bounded waits)

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete.  Gives up after `limit_cycles` SM
// clock cycles and returns false (the caller records an error and winds down).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  long long limit_cycles)
{
    if (mbar_try_wait(bar, parity)) {
        return true;
    }
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > limit_cycles) {
            return false;
        }
    }
    return true;
}

// One look at a barrier, without waiting (CLUSTER: one that also receives arrivals of the other CTA of a pair,
// acquired at cluster scope).
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    if constexpr (CLUSTER) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    }
    return ok != 0;
}

// The same for a barrier that also receives arrivals from the other CTA of a pair: acquires at
// cluster scope.
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// mbar_wait_bounded by a whole converged warp with one answer for all lanes.  The warps that feed
// the tensor cores and the copy engine run their loops on all 32 lanes and let one elected lane
// issue: with the loop inside `if (lane == 0)` a stage of four MMAs costs its issuer 565 clocks
// whatever their width, with uniform control flow 400 (measured with everything else in place
// taken away), and four 256-wide MMAs run for 512.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, long long limit_cycles)
{
    auto ready = [&] { return CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
    if (__all_sync(0xffffffffu, ready())) {
        return true;
    }
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, ready())) {
        if (__any_sync(0xffffffffu, clock64() - t0 > limit_cycles)) {
            return false;
        }
    }
    return true;
}

// One answer for a whole converged warp.
__device__ __forceinline__ bool warp_any(bool b) { return __any_sync(0xffffffffu, b); }

// True in one lane of a converged warp (always the same one).
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// ---------------------------------------------------------------- TMA

__device__ __forceinline__ void tma_prefetch_desc(const void* tmap)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// 2D tiled load, no multicast.  c0 is the innermost (contiguous) coordinate in elements.
__device__ __forceinline__ void tma_load_2d(void* dst, const void* tmap, uint64_t* bar, int c0,
                                            int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}

// Brings a tile of a 2D tensor into L2.
__device__ __forceinline__ void tma_prefetch_2d(const void* tmap, int c0, int c1)
{
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(
                     reinterpret_cast<uint64_t>(tmap)),
                 "r"(c0), "r"(c1)
                 : "memory");
}

// 2D tiled store from shared memory (bulk-group completion), no multicast.
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* src, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
            reinterpret_cast<uint64_t>(tmap)),
        "r"(smem_u32(src)), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

// Waits until the shared-memory sources of all committed bulk stores have been read.
__device__ __forceinline__ void bulk_wait_read0()
{
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Waits until all committed bulk stores have completed.
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Orders this thread's generic-proxy shared-memory writes before later async-proxy (TMA) reads.
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- tcgen05

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst_smem)),
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

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, both operands K-major, described by smem descriptors.
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                           uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same for 8-bit operands (kind::f8f6f4; the instruction descriptor's A/B format 0 is
// E4M3): one instruction covers K = 32, i.e. 32 bytes of each K-major row as in the 16-bit form.
__device__ __forceinline__ void tc_mma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives on the mbarrier once all previously issued tcgen05 ops of this thread complete.
__device__ __forceinline__ void tc_commit(uint64_t* bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tc_wait_ld()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane (base + t).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
}

// Four consecutive 32-bit columns of this warp's 32 lanes (thread t writes lane base + t).
__device__ __forceinline__ void tmem_st_32x32b_x4(uint32_t taddr, const uint32_t (&r)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3])
                 : "memory");
}

__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major operand tile written by TMA with 128-byte
// swizzle: rows of 64 16-bit elements (128 B), 8-row groups 1024 B apart.
DCVC_HOST_DEVICE uint64_t make_sw128_kmajor_desc(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);  // start address, bits 0-13
    d |= static_cast<uint64_t>(1) << 16;                      // leading byte offset (unused)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;              // stride byte offset, bits 32-45
    d |= static_cast<uint64_t>(1) << 46;                      // descriptor version (sm_100)
    d |= static_cast<uint64_t>(2) << 61;                      // layout: 128-byte swizzle
    return d;
}

// Instruction descriptor for kind::f16 with FP32 accumulation, both operands K-major.
// ab_format: 0 = f16, 1 = bf16.
DCVC_HOST_DEVICE uint32_t make_idesc_f16(int m, int n, int ab_format)
{
    uint32_t d = 0;
    d |= 1u << 4;                                  // D format: f32
    d |= static_cast<uint32_t>(ab_format) << 7;    // A format
    d |= static_cast<uint32_t>(ab_format) << 10;   // B format
    d |= static_cast<uint32_t>(n >> 3) << 17;      // N / 8
    d |= static_cast<uint32_t>(m >> 4) << 24;      // M / 16
    return d;
}

// ---------------------------------------------------------------- CTA pairs (cta_group::2)
// A cluster of two CTAs computes one 256-row MMA tile: each CTA stages its 128 rows of A and half
// of the tile's B columns, the even CTA issues the MMAs, and each CTA's tensor memory receives its
// 128 rows of the accumulator.  No TMA multicast: every load goes to the issuing CTA's own shared
// memory.

__device__ __forceinline__ uint32_t cluster_cta_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// All threads of both CTAs; orders shared-memory writes (barrier initialisation) before the peer's
// accesses.
__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();  // the barrier instructions are for converged warps
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The address of this CTA's shared variable `p` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}

// Predicated forms: a branch around one lane's instruction costs its warp some hundred clocks.
__device__ __forceinline__ void mbar_arrive_if(bool pred, uint64_t* bar)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(
                     smem_u32(bar)),
                 "r"(static_cast<int>(pred))
                 : "memory");
}

// Arrivals of a pair's CTAs on a barrier of the even one, which its MMA warp waits for with acquire at cluster
// scope.  Without a scope an arrival orders nothing outside its own CTA, so each says what crosses:
//
// Tensor memory alone (an accumulator has been read, values have been written to it): the loads and stores are
// complete (tcgen05.wait) and tcgen05.fence::before_thread_sync orders them before the arrival, ::after_thread_sync
// the MMA behind the wait.  No other memory is involved, so the arrival itself need not release any: relaxed, at
// cluster scope.  `n` arrivals at once (address from cluster_map).
__device__ __forceinline__ void mbar_arrive_tmem_if(bool pred, uint32_t cluster_addr, uint32_t n)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
        "@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0], %1;\n\t}" ::"r"(cluster_addr),
        "r"(n), "r"(static_cast<int>(pred))
        : "memory");
}

// Shared memory (the odd CTA's part of an operand that the MMA reads from both CTAs): a release at cluster scope.  It
// waits for all that its thread has in flight, and the next step of the MMA warp waits for it (tail kernel, us at
// 32640 pixels and 512 channels: 49.2 without an order between the CTAs, 65.4 with a release in every arrival, 51.6
// with one per warp and 64 columns of x, 51.0 as here).  So the writing warps arrive on a barrier of their own CTA,
// and one warp that has nothing in flight, the odd CTA's idle MMA warp, waits for it and arrives once, for all of
// them, on the even CTA's barrier at the same place, which counts the even CTA's warps and that one arrival.
// `even`: the distance from this CTA's shared memory to the even CTA's.
__device__ __forceinline__ bool pair_pass(uint64_t* bar, uint32_t parity, uint32_t even, long long limit_cycles)
{
    if (!mbar_wait_warp(bar, parity, limit_cycles)) {
        return false;
    }
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(smem_u32(bar) + even),
        "r"(static_cast<int>(elect_one()))
        : "memory");
    return true;
}

__device__ __forceinline__ void tma_store_2d_if(bool pred, const void* tmap, uint32_t src, int c0, int c1)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@p cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n\t}" ::"l"(
            reinterpret_cast<uint64_t>(tmap)),
        "r"(src), "r"(c0), "r"(c1), "r"(static_cast<int>(pred))
        : "memory");
}

// 2D tiled load into this CTA's shared memory whose completion is counted on a barrier of the
// pair's even CTA (`bar`: its address from cluster_map), no multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tmap, uint32_t bar, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

// A CTA that holds tensor memory asks for more than half of an SM's shared memory, so that no two of them meet on one
// SM and an allocation never waits for a kernel that waits for something else.
constexpr int kTmemCtaMinSmem = 232448 / 2 + 1;

// Tensor memory of a CTA pair.  tcgen05.alloc and tcgen05.dealloc with cta_group::2 are made by a warp of each
// CTA together and act on the tensor memory of both SMs.  Nothing but a barrier of the cluster shows that the
// other CTA has started, or that it is still there: without one, a CTA that asks for the pair's columns before its
// peer runs, or leaves while the peer still gives its columns back, has no bound on when that operation ends.
// Hence pair_begin() and pair_end(); the two meetings cost a launch 0.2 to 0.4 us (tail of 8160 to 14400 rows).

// All threads of both CTAs, once the barriers of the CTA are initialised; the warp of each CTA for which `alloc_warp`
// holds allocates.
__device__ __forceinline__ uint32_t pair_begin(uint32_t* dst_smem, uint32_t ncols, bool alloc_warp)
{
    cluster_sync();  // both CTAs run; their barriers are initialised before any copy or arrive reaches them
    if (alloc_warp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *dst_smem;
}

// All threads of both CTAs, last.
__device__ __forceinline__ void pair_end(uint32_t taddr, uint32_t ncols, bool alloc_warp)
{
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs are done with the pair's accumulators and each other's barriers
    if (alloc_warp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
    }
    cluster_sync();  // and have both given the columns back
}

// M = 256 MMA over both CTAs' operands (issued by the even CTA).
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same with A in tensor memory: each CTA's 128 rows in its lanes, 16-bit K elements packed two
// to a column.
__device__ __forceinline__ void tc_mma_f16_pair_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                   uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same for E4M3 operands (see tc_mma_f8).
__device__ __forceinline__ void tc_mma_f8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on the barrier at this offset in both CTAs of the pair once the issued MMAs complete.
__device__ __forceinline__ void tc_commit_pair_both(uint64_t* bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}

// Arrive on this CTA's barrier once the issued MMAs complete.
__device__ __forceinline__ void tc_commit_pair_local(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------- math

__device__ __forceinline__ float tanh_approx(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// WSiLU(x) = x * sigmoid(4x) (src/layers/layers.py:106-111), evaluated through the identity
// sigmoid(4x) = (1 + tanh(2x)) / 2 with the hardware tanh approximation (relative error about
// 2^-11, the FP16 rounding step of the stored result).
__device__ __forceinline__ float wsilu(float x)
{
    const float h = 0.5f * x;
    return fmaf(h, tanh_approx(2.0f * x), h);
}

// wsilu() of two values with packed f32x2 arithmetic (sm_100 FMUL2 / FADD2 / FFMA2): each lane is
// rounded to nearest on its own, so each result is bitwise equal to wsilu() of that lane, with
// half the FP32-pipe instructions.  x + x is the exact doubling 2.0f * x.
__device__ __forceinline__ float2 wsilu2(float2 x)
{
    const float2 h = __fmul2_rn(x, make_float2(0.5f, 0.5f));
    const float2 d = __fadd2_rn(x, x);
    return __ffma2_rn(h, make_float2(tanh_approx(d.x), tanh_approx(d.y)), h);
}

}  // namespace dcvc
