/*
 * tc_common.cuh -- sm_100a building blocks written directly in PTX:
 * mbarriers with bounded waits, TMA tile loads (no cluster multicast),
 * tcgen05 MMA / TMEM allocation / TMEM loads, and the shared-memory matrix
 * and instruction descriptors of the 5th-generation tensor cores.
 *
 * Descriptor bit layouts follow the PTX ISA ("tcgen05 matrix descriptors",
 * "instruction descriptor"): they were cross-checked against the field
 * definitions in CUTLASS's cute/arch/mma_sm100_desc.hpp.
 *
 * Every wait on an mbarrier is bounded: after the wait limit of
 * %globaltimer time the wait records an error code in a device flag and
 * returns false, and the kernel unwinds (frees TMEM, exits) instead of
 * hanging the GPU.
 *
 * The flag is the first int of the device error block each tensor-core
 * kernel receives as `err` (16 bytes, 8-byte aligned): err[0] the error code
 * (0 = none), err[2..3] the wait limit in nanoseconds as one 64-bit value
 * (0 = HCBK_WAIT_TIMEOUT_NS).  The limit is read once per wait, when the
 * first try finds the phase incomplete.
 */
#ifndef HCBLAS_B200_TC_COMMON_CUH_
#define HCBLAS_B200_TC_COMMON_CUH_

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef HCBK_WAIT_TIMEOUT_NS
#define HCBK_WAIT_TIMEOUT_NS 2000000000ull /* 2 s */
#endif

namespace hcbk {
namespace tc {

/* error codes written to the device error flag */
enum : int {
  ERR_NONE = 0,
  ERR_TIMEOUT_PRODUCER = 1,
  ERR_TIMEOUT_MMA_FULL = 2,
  ERR_TIMEOUT_MMA_TMEM = 3,
  ERR_TIMEOUT_EPILOGUE = 4,
  ERR_TIMEOUT_COMBINE = 5,
  ERR_LAUNCH_SHAPE = 6, /* a kernel was launched with a block shape it does not support */
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

/* ------------------------------------------------------------ mbarrier -- */

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

/* the same with cluster-scope acquire: for barriers that the peer CTA of
 * a pair arrives on */
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

/* Wait for the phase with the given parity to complete.  Bounded: returns
 * false (after recording `code` in *err) on timeout, or when another thread
 * has already recorded an error. */
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err, int code) {
  auto try_once = [&]() {
    return CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity);
  };
  if (try_once()) return true;
  const uint64_t t0 = globaltimer();
  const uint64_t set = *reinterpret_cast<volatile unsigned long long *>(err + 2);
  const uint64_t limit = set ? set : HCBK_WAIT_TIMEOUT_NS;
  uint32_t n = 0;
  while (true) {
    if (try_once()) return true;
    if ((++n & 1023u) == 0) {
      if (*reinterpret_cast<volatile int *>(err) != 0) return false;
      if (globaltimer() - t0 > limit) {
        atomicCAS(err, 0, code);
        return false;
      }
    }
  }
}

/* --------------------------------------- programmatic dependent launch -- */

/* A kernel launched with the programmatic-serialization attribute may start
 * while the kernel before it in the stream still runs; all its threads wait
 * here, before the first access to global memory, until that kernel is done
 * and its writes are visible (at once when launched the ordinary way).  What
 * overlaps is the launch itself and the prologue (barriers, TMEM). */
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
/* the launch attribute of such a kernel */
inline cudaLaunchAttribute pdl_attribute() {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}
/* in the kernel before: the next one may be scheduled once every block has
 * passed here (or ended) */
__device__ __forceinline__ void grid_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

/* ------------------------------------------------- CTA pair (cluster) -- */

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

/* every thread of every CTA in the cluster; release/acquire ordering */
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* shared::cluster address of the variable at `p` in CTA `rank` of the cluster */
__device__ __forceinline__ uint32_t mapa_shared(const void *p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}

/* arrive on an mbarrier given by its shared::cluster address (possibly in
 * the peer CTA) */
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}

/* ---------------------------------------------------------------- TMA -- */

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

/* 1-D bulk copy from global memory into this CTA's shared memory: both
 * addresses 16-byte aligned, `bytes` a multiple of 16; completion is
 * signalled on `bar` (complete_tx).  No multicast. */
__device__ __forceinline__ void bulk_load_1d(void *dst, const void *src, uint32_t bytes,
                                             uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(static_cast<uint64_t>(__cvta_generic_to_global(src))), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

/* 2-D tiled bulk tensor load into this CTA's shared memory; completion is
 * signalled on `bar` (complete_tx).  No multicast. */
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}

/* 3-D tiled bulk tensor load (coordinates innermost first).  No multicast. */
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int32_t c0, int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

/* 2-D tiled load into this CTA's shared memory whose completion is counted
 * on the mbarrier at shared::cluster address `bar_cluster` -- the pair
 * leader's barrier (.cta_group::2 lets the barrier live in either CTA of the
 * pair).  No multicast. */
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map,
                                                 uint32_t bar_cluster, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(c0), "r"(c1)
      : "memory");
}

/* 3-D form of tma_load_2d_pair (coordinates innermost first).  No multicast. */
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map,
                                                 uint32_t bar_cluster, int32_t c0, int32_t c1,
                                                 int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

/* 2-D tiled bulk tensor store from this CTA's shared memory (coordinates
 * innermost first); out-of-range parts of the box are not written. */
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, const void *src, int32_t c0,
                                             int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(smem_u32(src)), "r"(c0), "r"(c1)
      : "memory");
}

/* 3-D tiled bulk tensor store from this CTA's shared memory (coordinates
 * innermost first); out-of-range parts of the box are not written.  The
 * writing threads issue fence_proxy_async_smem() before the store. */
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *src, int32_t c0,
                                             int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

/* Tensor maps patched on the device (problem tables built by a kernel
 * from device-resident pointer arrays): the global address of a 128-byte
 * aligned map in global memory is replaced in place, the patching thread
 * releases its generic-proxy writes to the tensor-map proxy, and a kernel
 * that then loads or stores through the map acquires it first. */
__device__ __forceinline__ void tensormap_replace_address(void *map, const void *addr) {
  asm volatile("tensormap.replace.tile.global_address.global.b1024.b64 [%0], %1;" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "l"(reinterpret_cast<uint64_t>(addr))
               : "memory");
}

/* dimension ORD's extent, and the byte stride of dimension ORD + 1 */
template <int ORD> __device__ __forceinline__ void tensormap_replace_dim(void *map, uint32_t n) {
  asm volatile("tensormap.replace.tile.global_dim.global.b1024.b32 [%0], %2, %1;" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(n), "n"(ORD)
               : "memory");
}
template <int ORD>
__device__ __forceinline__ void tensormap_replace_stride(void *map, uint64_t bytes) {
  asm volatile("tensormap.replace.tile.global_stride.global.b1024.b64 [%0], %2, %1;" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "l"(bytes), "n"(ORD)
               : "memory");
}

__device__ __forceinline__ void tensormap_release() {
  asm volatile("fence.proxy.tensormap::generic.release.gpu;" ::: "memory");
}

__device__ __forceinline__ void tensormap_acquire(const void *map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                   reinterpret_cast<uint64_t>(map))
               : "memory");
}

/* make this thread's generic-proxy shared-memory writes visible to the
 * async proxy (bulk / tensor copies) */
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

/* wait until at most N of this thread's committed bulk groups still read
 * their shared-memory source */
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

/* wait until all of this thread's committed bulk groups have completed */
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

/* ------------------------------------------------------------ tcgen05 -- */

/* TMEM allocation for a CTA pair: one warp (same warp index) in each CTA
 * of the pair issues it; both receive the same column range. */
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

/* Pair MMA (issued by one thread of the leader CTA): M = 256 rows, rows
 * 0..127 of A from the leader's shared memory and 128..255 from the peer's
 * at the same offsets; B's N columns split in halves the same way; each
 * CTA's TMEM receives its 128 rows of D. */
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

/* The pair MMA with 8-bit integer operands and an s32 accumulator. */
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

/* Arrive once on the mbarrier at this shared-memory offset in every CTA of
 * `cta_mask` when all prior pair MMAs of this thread have completed. */
__device__ __forceinline__ void mma_commit_pair(uint64_t *bar, uint16_t cta_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(smem_u32(bar)),
      "h"(cta_mask)
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
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

/* D[tmem] (+)= A[smem] * B[smem]; kind::f16 covers f16 and bf16 operands
 * with an f32 accumulator. */
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

/* D[tmem] (+)= A[smem] * B[smem]; 8-bit integer operands, s32 accumulator. */
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

/* Arrive on `bar` once all previously issued tcgen05.mma of this thread
 * have completed. */
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

/* 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives
 * lane (base + i), columns [col, col + 32). */
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
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

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

/* 32 lanes x 32 consecutive 32-bit columns written from registers: thread
 * i of the warp writes lane (base + i), columns [col, col + 32). */
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

/* ------------------------------------------------------- descriptors -- */

/* Shared-memory matrix descriptor with sm_100 version bits (46-47 = 1) and a
 * swizzle layout (bits 61-63: 2 = 128B, 4 = 64B).  Offsets in bytes.
 *   K-major:  LBO unused (16), SBO = 8 rows x row bytes (1024 for 128B,
 *             512 for 64B swizzle)
 *   MN-major (128B): LBO = byte distance between 64-element MN blocks,
 *             SBO = 1024 (8 K-rows x 128 B) */
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo,
                                              uint32_t layout) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(layout & 7u) << 61;
  return d;
}

/* SWIZZLE_128B (layout 2) form used by the 16-bit paths.  (The int8 path
 * uses SWIZZLE_64B, layout 4: K-major rows of 64 bytes, SBO = 512.) */
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return smem_desc(saddr, lbo, sbo, 2);
}

/* Instruction descriptor (kind::f16 / kind::i8, dense).
 *   c_fmt: 1 = f32, 2 = s32 accumulator;  ab_fmt: f16 = 0, bf16 = 1 (kind::f16),
 *   u8 = 0, s8 = 1 (kind::i8);  a_mn/b_mn: operand is MN-major;
 *   neg_a: negate A (f16 kinds only). */
__host__ __device__ constexpr uint32_t make_idesc(uint32_t c_fmt, uint32_t ab_fmt, bool a_mn,
                                                  bool b_mn, uint32_t M, uint32_t N,
                                                  bool neg_a = false) {
  return (c_fmt << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((neg_a ? 1u : 0u) << 13) |
         ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((N >> 3) << 17) |
         ((M >> 4) << 24);
}

/* ------------------------------------------------ split-BF16 recipes --
 * One plane pair per product: A plane pa(i) x B plane pb(i) -> accumulator
 * pacc(i); first(i) marks the first product written to its accumulator. */

/* bf16x3: lo*hi + hi*lo into accumulator 1, hi*hi into accumulator 0
 * (lo*lo dropped).  Keeping the correction terms (2^-8 smaller) apart from
 * the leading term keeps them from being truncated against it. */
struct RecipeBf16x3 {
  static constexpr int NA = 2, NB = 2, NP = 3, NACC = 2;
  static constexpr bool P3D = false;
  __host__ __device__ static constexpr int pa(int i) { return i == 0 ? 1 : 0; }
  __host__ __device__ static constexpr int pb(int i) { return i == 1 ? 1 : 0; }
  __host__ __device__ static constexpr int pacc(int i) { return i == 2 ? 0 : 1; }
  __host__ __device__ static constexpr bool first(int i) { return i == 0 || i == 2; }
};
/* bf16x6: three-way split, every product of total order <= 2; hi*hi into
 * accumulator 0, the five correction products into accumulator 1 */
struct RecipeBf16x6 {
  static constexpr int NA = 3, NB = 3, NP = 6, NACC = 2;
  static constexpr bool P3D = false;
  __host__ __device__ static constexpr int pa(int i) {
    return i == 0 ? 2 : i == 1 ? 1 : i == 2 ? 0 : i == 3 ? 1 : 0;
  }
  __host__ __device__ static constexpr int pb(int i) {
    return i == 0 ? 0 : i == 1 ? 1 : i == 2 ? 2 : i == 3 ? 0 : i == 4 ? 1 : 0;
  }
  __host__ __device__ static constexpr int pacc(int i) { return i == 5 ? 0 : 1; }
  __host__ __device__ static constexpr bool first(int i) { return i == 0 || i == 5; }
};

/* ------------------------------------- f16 C that TMA cannot address -- */

/* An f16 C whose rows or leading dimension are not whole 16-byte chunks.  The
 * kernel computes the transposed product, so that a TMEM lane is a column of C
 * and its TMEM columns are consecutive rows: two rows convert to one word in
 * one instruction, and a warp's 32 columns go through its own part of shared
 * memory, 128 rows at a time, without meeting the other warps.  (One warp per SM
 * sub-partition makes this epilogue bound by its instruction count: with a
 * TMEM lane per row, 2-byte stores of 32-row pieces took 134 us for an
 * 8191 x 8191 C at K = 33, a four-warp exchange through shared memory 224.)
 *
 * Column j of the 32 sits at pitch 272 bytes, at the same offset within 16
 * bytes as in C, so that each whole 16-byte chunk of a column moves as one
 * aligned vector between shared and global memory, two columns per warp
 * instruction; a column's ends (fewer than 8 rows each) move as 2-byte
 * elements. */
constexpr int COLS_ROWS = 128;
constexpr uint32_t COLS_PITCH = 2 * COLS_ROWS + 16; /* the rows + 16 bytes of alignment */
constexpr uint32_t COLS_WARP_BYTES = 32 * COLS_PITCH;

/* whole chunks of the 32 columns at C (ldc apart; `rows` <= COLS_ROWS rows,
 * `cols` valid columns) from shared to global memory (STORE) or back, U chunks
 * in flight per lane */
template <bool STORE, int U = 8>
__device__ __forceinline__ void cols_copy(uint8_t *buf, __half *C, long long ldc, int rows,
                                          int cols) {
  const int lane = threadIdx.x & 31;
  const int c16 = 16 * (lane & 15);
  const int j0 = lane >> 4;
  const int bytes = 2 * rows;
  uint8_t *g = reinterpret_cast<uint8_t *>(C + (long long)j0 * ldc);
  uint8_t *s = buf + j0 * COLS_PITCH + c16;
#pragma unroll 1
  for (int h = 0; h < 32; h += 2 * U) {
    uint4 v[U];
    uint8_t *at[U];
    bool on[U];
#pragma unroll
    for (int i = 0; i < U; ++i) { /* every load before the first store */
      const int mis = (int)(reinterpret_cast<uintptr_t>(g) & 15);
      on[i] = h + 2 * i + j0 < cols && c16 >= mis && c16 + 16 <= mis + bytes;
      at[i] = g - mis + c16;
      g += 4 * ldc; /* two columns */
      if (on[i])
        v[i] = STORE ? *reinterpret_cast<const uint4 *>(s + 2 * i * COLS_PITCH)
                     : *reinterpret_cast<const uint4 *>(at[i]);
    }
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (on[i]) *reinterpret_cast<uint4 *>(STORE ? at[i] : s + 2 * i * COLS_PITCH) = v[i];
    s += 2 * U * COLS_PITCH;
  }
}

/* the ends of this lane's column: the rows before its first and after its
 * last whole chunk */
template <bool STORE>
__device__ __forceinline__ void cols_ends(uint8_t *sb, __half *g, int rows) {
  const int mis = (int)(reinterpret_cast<uintptr_t>(g) & 15);
  __half *s = reinterpret_cast<__half *>(sb + mis);
  const int head = mis ? (16 - mis) >> 1 : 0;
  const int last = (((mis + 2 * rows) & ~15) - mis) >> 1;
  const int tail = last > head ? last : head;
#pragma unroll
  for (int i = 0; i < 7; ++i)
    if (i < head && i < rows) {
      if (STORE) g[i] = s[i];
      else s[i] = g[i];
    }
#pragma unroll
  for (int i = 0; i < 7; ++i)
    if (tail + i < rows) {
      if (STORE) g[tail + i] = s[tail + i];
      else s[tail + i] = g[tail + i];
    }
}

/* The three steps of a piece of C -- `nr` <= COLS_ROWS rows of the warp's 32
 * columns at C, `cols` of them valid, lane i holding column i -- with a
 * __syncwarp() between them: C into the staging (beta != 0), the sums merged
 * there, the staging to C. */
__device__ __forceinline__ void cols_fetch(uint8_t *buf, __half *C, long long ldc, int nr,
                                           int cols) {
  const int lane = threadIdx.x & 31;
  cols_copy<false>(buf, C, ldc, nr, cols);
  if (lane < cols) cols_ends<false>(buf + lane * COLS_PITCH, C + (long long)lane * ldc, nr);
}
/* the same with asynchronous copies of the whole chunks (no registers, no
 * wait): cols_fetch_wait() and a __syncwarp() before they are read */
__device__ __forceinline__ void cols_fetch_async(uint8_t *buf, __half *C, long long ldc, int nr,
                                                 int cols) {
  const int lane = threadIdx.x & 31;
  const int c16 = 16 * (lane & 15), j0 = lane >> 4;
  const uint8_t *g = reinterpret_cast<const uint8_t *>(C + (long long)j0 * ldc);
  uint32_t s = smem_u32(buf + j0 * COLS_PITCH + c16);
#pragma unroll 4
  for (int j = j0; j < 32; j += 2, g += 4 * ldc, s += 2 * COLS_PITCH) { /* two columns */
    const int mis = (int)(reinterpret_cast<uintptr_t>(g) & 15);
    if (j < cols && c16 >= mis && c16 + 16 <= mis + 2 * nr)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(g - mis + c16)
                   : "memory");
  }
  if (lane < cols) cols_ends<false>(buf + lane * COLS_PITCH, C + (long long)lane * ldc, nr);
}
__device__ __forceinline__ void cols_fetch_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}
template <int U = 8>
__device__ __forceinline__ void cols_flush(uint8_t *buf, __half *C, long long ldc, int nr,
                                           int cols) {
  const int lane = threadIdx.x & 31;
  cols_copy<true, U>(buf, C, ldc, nr, cols);
  if (lane < cols) cols_ends<true>(buf + lane * COLS_PITCH, C + (long long)lane * ldc, nr);
}
/* staging = alpha * sum (+ beta * staging); load(g, r) gives rows g .. g + 31
 * of the lane's column (f32 bit patterns).  GROUPS > 0: that many groups of
 * 32, unrolled (sums in registers). */
template <int GROUPS, class Load>
__device__ __forceinline__ void cols_merge(uint8_t *buf, const __half *C, long long ldc, int nr,
                                           float alpha, float beta, bool ld_c, Load &&load) {
  const int lane = threadIdx.x & 31;
  const int mis = (int)(reinterpret_cast<uintptr_t>(C + (long long)lane * ldc) & 15);
  uint32_t *w = reinterpret_cast<uint32_t *>(buf + lane * COLS_PITCH + (mis & ~3));
  const uint32_t sft = (mis & 2) * 8; /* 16 when the column starts in a word's upper half */
  uint32_t carry = ld_c ? w[0] : 0u, old = carry;
#pragma unroll(GROUPS > 0 ? GROUPS : 1)
  for (int g = 0; g < (GROUPS > 0 ? 32 * GROUPS : nr); g += 32) {
    if (g >= nr) continue;
    uint32_t r[32];
    load(g, r);
    uint32_t *wg = w + g / 2;
    if (ld_c) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        /* rows 2i, 2i + 1 of the group: words i and i + 1 of the column */
        const uint32_t next = wg[i + 1];
        const uint32_t c2 = __funnelshift_r(old, next, sft);
        old = next;
        const __half2 h = *reinterpret_cast<const __half2 *>(&c2);
        r[2 * i] = __float_as_uint(
            fmaf(beta, __low2float(h), alpha * __uint_as_float(r[2 * i])));
        r[2 * i + 1] = __float_as_uint(
            fmaf(beta, __high2float(h), alpha * __uint_as_float(r[2 * i + 1])));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(alpha * __uint_as_float(r[i]));
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const __half2 h =
          __floats2half2_rn(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      const uint32_t hw = *reinterpret_cast<const uint32_t *>(&h);
      wg[i] = __funnelshift_l(carry, hw, sft);
      carry = hw;
    }
    /* the last row of a shifted column; the next group rewrites the word */
    if (!ld_c || g + 32 >= nr) wg[16] = __funnelshift_l(carry, 0u, sft);
  }
}

/* One warp's 32 columns x `width` rows of C: TMEM lane i (of this warp) is
 * column i, `width` TMEM columns at tbase are consecutive rows; rows / cols
 * valid; C the first of them.  C = alpha * acc (+ beta * C). */
__device__ __forceinline__ void cols_tile(uint8_t *buf, uint32_t tbase, int width, __half *C,
                                          long long ldc, int rows, int cols, float alpha,
                                          float beta, bool ld_c) {
  if (rows > width) rows = width;
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += COLS_ROWS) {
    const int nr = rows - r0 < COLS_ROWS ? rows - r0 : COLS_ROWS;
    __syncwarp(); /* the previous rows have been copied out */
    if (ld_c) {
      cols_fetch(buf, C + r0, ldc, nr, cols);
      __syncwarp();
    }
    cols_merge<0>(buf, C + r0, ldc, nr, alpha, beta, ld_c, [&](int g, uint32_t(&r)[32]) {
      tmem_ld_32x32b_x32(tbase + r0 + g, r);
      tmem_ld_wait();
    });
    __syncwarp();
    cols_flush(buf, C + r0, ldc, nr, cols);
  }
}

}  // namespace tc
}  // namespace hcbk

#endif /* HCBLAS_B200_TC_COMMON_CUH_ */
