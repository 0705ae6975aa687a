// Thin inline-PTX wrappers for the Blackwell (sm_100a) primitives the kernels
// in this directory are built from: mbarrier, TMA tiled loads
// (cp.async.bulk.tensor), tensor memory (tcgen05.alloc / ld / st) and the
// 5th-generation tensor-core MMA (tcgen05.mma) with its shared-memory and
// instruction descriptors.
//
// Every wait in this file is bounded: a wait that runs out sets a status bit
// and returns false so the caller can unwind (drain its copies, free its
// tensor memory) and leave the kernel normally.
#pragma once

#include <cstdint>
#include <mutex>
#include <vector>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace bdattn {

// Status bits written by kernels into the per-device status word.
enum : int {
    kStatusWaitTimeout = 1,   // a bounded mbarrier wait ran out
    kStatusBadArgs = 2,       // device-side argument check failed
};

// Per-device status word (one copy per device that loads the module).  The
// library is built as a single translation unit, so this definition is the
// only one.
__device__ int g_device_status = 0;

// ------------------------------------------------------------ host helpers
// Raises a kernel's dynamic shared-memory limit to `bytes` once per (kernel,
// device) instead of on every launch; a later request for more raises it again.
inline cudaError_t set_max_smem_once_impl(const void* func, int bytes) {
    struct Seen { const void* func; int dev; int bytes; };
    static std::mutex mu;
    static std::vector<Seen> seen;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    for (Seen& s : seen) {
        if (s.func == func && s.dev == dev) {
            if (s.bytes >= bytes) return cudaSuccess;
            e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e == cudaSuccess) s.bytes = bytes;
            return e;
        }
    }
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) seen.push_back({func, dev, bytes});
    return e;
}
template <class Kernel>
inline cudaError_t set_max_smem_once(Kernel kernel, int bytes) {
    return set_max_smem_once_impl(reinterpret_cast<const void*>(kernel), bytes);
}
// Streaming-multiprocessor count of the current device, looked up once per device.
inline int sm_count() {
    static std::mutex mu;
    static int count[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    std::lock_guard<std::mutex> lock(mu);
    if (count[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        count[dev] = n;
    }
    return count[dev];
}

// Programmatic dependent launch.  A kernel launched through launch_dependent() may
// become resident while the kernel before it in the stream is still running (as that
// one's CTAs retire, once all of them have passed dependents_may_launch()); it does
// its set-up and then holds at wait_for_prior_grid() until the earlier grid has
// completed and its writes are visible.  A kernel launched this way reads and writes no global memory ahead of
// wait_for_prior_grid(); what may come before it are requests that bring data into the L2
// (tma_prefetch_l2_2d).  CTAs and threads that have nothing to do may end without the wait: the grid is complete
// only when those that have have waited, so that a grid behind it still finds all earlier ones complete.
// With a cluster of more than one CTA, `cluster` gives its size.
template <class... KArgs, class... Args>
inline cudaError_t launch_dependent_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                            cudaStream_t stream, dim3 cluster, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster.x;
    attr[1].val.clusterDim.y = cluster.y;
    attr[1].val.clusterDim.z = cluster.z;
    cfg.attrs = attr;
    cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <class... KArgs, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                    cudaStream_t stream, Args&&... args) {
    return launch_dependent_cluster(kernel, grid, block, smem, stream, dim3(1), static_cast<Args&&>(args)...);
}
__device__ __forceinline__ void dependents_may_launch() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_prior_grid() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a converged warp, the same one every time.  tcgen05 instructions take descriptors,
// addresses and barriers from uniform registers.  In a branch that the compiler can tell is taken by a
// single, elected thread, of a warp whose number it knows to be the same in all lanes
// (warp_index), their operands can be computed there; behind `lane == 0` an MMA took its thread 46-64 cycles,
// as long as the tensor pipe needs for 128 columns and longer than for 64.
// 576 x 1280 x 1280 9.9 -> 6.5 us, 2240 x 1024 x 2240 16.6 -> 11.9, 4096 x 3 x 3072 x 3072 with norm + RoPE
// 172 -> 163, attention 4096 x 4096, 8 heads of 40, 54.9 -> 52.6.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n"
        ".reg .b32 rx;\n"
        ".reg .pred px;\n"
        "elect.sync rx|px, 0xffffffff;\n"
        "@px mov.s32 %0, 1;\n"
        "}\n"
        : "+r"(pred));
    return pred != 0;
}
// The warp's number, known to be the same in all of its lanes.
__device__ __forceinline__ int warp_index() {
    return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0);
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait for the phase with the given parity to complete.  The limit is
// wall time (two seconds), checked every 4096 polls.  On expiry the timeout
// bit is set in the device status word and false is returned.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 4096; ++i) {
            if (mbar_try_wait(bar, parity)) return true;
        }
        if (global_timer_ns() - t0 > 2000000000ull) {
            atomicOr(&g_device_status, kStatusWaitTimeout);
            return false;
        }
    }
}
// The same for a converged warp: one answer for all of its lanes, so that they stay together.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0;
}

// -------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 3-D tiled load (x = innermost element coordinate; x * elem_size must be a
// multiple of 16 bytes), completing on an mbarrier of this CTA.  No multicast.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)),
          "r"(x), "r"(y), "r"(z)
        : "memory");
}
// 3-D tiled store shared -> global (bulk group completion).  Coordinates must not
// be negative; x * element size must be a multiple of 16 bytes; elements past
// the tensor's extent are not written.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Waits until the bulk stores of this thread have finished READING shared memory.
__device__ __forceinline__ void tma_store_wait_read_all() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// Waits until the bulk stores of this thread have completed.
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Makes this thread's shared-memory writes visible to the async proxy (TMA).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// 4-D tiled load (d, head, row, batch).  Elements outside a dimension are
// zero-filled, which pads a head narrower than the box on the fly.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)),
          "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)),
          "r"(x), "r"(y)
        : "memory");
}

// Asks for a box to be brought into the L2, where every later access sees it, whoever wrote it last: so this may
// run ahead of wait_for_prior_grid().
__device__ __forceinline__ void tma_prefetch_l2_2d(const CUtensorMap* m, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y)
                 : "memory");
}

// Asynchronous copy of kBytes (4 or 16) to shared memory, zeros where `on` is false (src is then not read).
template <int kBytes>
__device__ __forceinline__ void cp_async_zfill(void* dst, const void* src, bool on) {
    const int n = on ? kBytes : 0;
    if constexpr (kBytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// 32 x 32 values of an FP32 matrix to 4 KB of a warp's shared memory (cp.async), rows [row, row + 32) from column 0
// of `src`, zeros outside rows [0, n_rows) and columns [0, n_cols).  The 16-byte pieces of a row are permuted by
// the row, so that a copy takes whole rows and a lane reads its own without bank conflicts (row_piece32): a
// load with a row per lane touches 32 cache lines.
__device__ __forceinline__ void copy_rows32(uint8_t* dst, const float* src, long long ld, int row, int n_rows, int n_cols,
                                            int lane) {
    if ((n_cols >= 32 || (n_cols & 3) == 0) && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3), p = lane & 7;
            const bool on = row + r >= 0 && row + r < n_rows && p * 4 < n_cols;
            cp_async_zfill<16>(dst + r * 128 + ((p ^ (r & 7)) << 4), on ? src + (row + r) * ld + p * 4 : src, on);
        }
    } else {
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
            const bool on = row + r >= 0 && row + r < n_rows && lane < n_cols;
            cp_async_zfill<4>(dst + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4,
                              on ? src + (row + r) * ld + lane : src, on);
        }
    }
}
// Values 4 i .. 4 i + 3 of the lane's row.
__device__ __forceinline__ float4 row_piece32(const uint8_t* rows, int lane, int i) {
    return *reinterpret_cast<const float4*>(rows + lane * 128 + ((i ^ (lane & 7)) << 4));
}

// ---------------------------------------------------------- tensor memory
// Allocate ncols (power of two, 32..512) TMEM columns; the base address is
// written to *smem_slot.  Executed by one full warp.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(smem_slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives
// lane (lane_base + t), columns [col, col + 32).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
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
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
          "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
          "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
          "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
          "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// ------------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs of a cluster, one tile: both allocate, the even CTA issues the MMAs, whose
// operands lie at the same shared-memory offsets in both.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same without ordering memory: for the start (behind fence_mbar_init) and for the end of a
// kernel whose CTAs have waited for every arrival and read every value that comes from a peer, and only
// have to outlive the peers' accesses to them.  The release of the other form waits for the global
// stores in flight.
__device__ __forceinline__ void cluster_sync_relaxed() {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this CTA's shared-memory address `addr` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled load into this CTA's shared memory that completes on a barrier of either CTA
// of the pair (`bar`: shared::cluster address).  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive (count 1) on the barrier at this offset in both CTAs once all MMAs issued so far
// by this thread have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}

// ------------------------------------------------------------ descriptors
// Shared-memory matrix descriptor, 128-byte swizzle (layout type 2), for a
// tile whose rows are 128 bytes (64 16-bit elements) and whose 8-row groups
// are `sbo_bytes` apart.  Bits: [0,14) start>>4, [16,30) LBO>>4, [32,46)
// SBO>>4, [46,48) version=1, [61,64) layout type.
//   K-major operand : LBO unused (1), SBO = 1024.
//   MN-major operand: LBO = distance between 64-element column chunks,
//                     SBO = distance between 8-row (K) groups = 1024.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes,
                                                         uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

// Instruction descriptor for kind::f16 with BF16 (fmt=1) or F16 (fmt=0)
// operands and an FP32 accumulator.
//   bits [4,6) D format (1 = F32), [7,10) A format, [10,13) B format,
//   bit 15 A major (0 = K), bit 16 B major (0 = K, 1 = MN),
//   [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc_f16(int fmt, int M, int N, int a_mn_major,
                                                      int b_mn_major) {
    return (1u << 4) | (static_cast<uint32_t>(fmt) << 7) | (static_cast<uint32_t>(fmt) << 10) |
           (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
           (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] . B[smem]      (issued by one thread)
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem]      (A: 16-bit elements, two per column)
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive (count 1) on an mbarrier once all MMAs issued so far by this thread
// have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// ---------------------------------------------------------------- numerics
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// x * Phi(x), the exact (erf) GELU.  Phi(-a) = exp(-a^2 / 2) * g(a) for a >= 0 with
// g(a) = erfcx(a / sqrt(2)) / 2, here a polynomial in t = 1 / (1 + 0.21 a) (the form of
// Abramowitz & Stegun 7.1.26; degree 9, coefficients from a weighted least-squares fit to 1.6e-8
// relative over a in [0, 14]).  No branch, about 20 instructions: the epilogues of the GEGLU
// layers were bound by erff.  Largest error over [-12, 12] in FP32: 3.8e-7 (4.5e-7 for
// 0.5 x (1 + erff(x / sqrt(2)))).
__device__ __forceinline__ float gelu_exact(float x) {
    const float a = fabsf(x);
    const float t = __fdividef(1.0f, fmaf(0.21f, a, 1.0f));
    float h = -0.0716563025f;
    h = fmaf(h, t, 0.283588519f);
    h = fmaf(h, t, -0.33025326f);
    h = fmaf(h, t, 0.349400848f);
    h = fmaf(h, t, -0.0939250888f);
    h = fmaf(h, t, 0.124872676f);
    h = fmaf(h, t, 0.0691921831f);
    h = fmaf(h, t, 0.0850688561f);
    h = fmaf(h, t, 0.0837115758f);
    h *= t * fast_exp2(a * a * -0.72134752f);
    return x * (x >= 0.0f ? 1.0f - h : h);
}
// Packs two floats to 16-bit halves of a word: `lo` in bits [0,16).
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    uint32_t r;
    if constexpr (kBf16) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    } else {
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    }
    return r;
}

// v + bias of N columns (bias in shared memory, read by all lanes alike).
template <int N>
__device__ __forceinline__ void add_bias(const uint32_t (&v)[N], const float* bias_w, float (&f)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bias_w + i);
        f[i] = __uint_as_float(v[i]) + b.x;
        f[i + 1] = __uint_as_float(v[i + 1]) + b.y;
        f[i + 2] = __uint_as_float(v[i + 2]) + b.z;
        f[i + 3] = __uint_as_float(v[i + 3]) + b.w;
    }
}

// Stores a warp's 32 x 32 tile (thread = row) of 16-bit values, two to a word: through `stg` (2 KB of this
// warp's shared memory), so that four lanes write 64 consecutive bytes of a row.  Straight
// from the registers a store instruction touches 32 rows, 32 cache lines.
// base: element (first row, first column); rows / cols: how many of each exist.
__device__ __forceinline__ void store_words32(const uint32_t (&w)[16], uint8_t* stg, int lane, uint16_t* base,
                                              long long ld, int rows, int cols) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(stg + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
            make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    __syncwarp();
    const int c = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = i * 8 + (lane >> 2);
        if (r < rows && c * 8 < cols)
            *reinterpret_cast<uint4*>(base + r * ld + c * 8) =
                *reinterpret_cast<const uint4*>(stg + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
    }
    __syncwarp();
}
template <bool kBf16>
__device__ __forceinline__ void store_tile32(const float (&f)[32], uint8_t* stg, int lane, uint16_t* base,
                                             long long ld, int rows, int cols) {
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = pack2<kBf16>(f[2 * i], f[2 * i + 1]);
    store_words32(w, stg, lane, base, ld, rows, cols);
}

}  // namespace bdattn
