// tc.cuh -- PTX building blocks of the tcgen05 kernels: mbarriers with bounded
// waits, TMA loads, shared-memory and instruction descriptors, MMA issue and
// commit (one CTA and CTA pair), TMEM loads, and the tensor-map encoder.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"

namespace rimp2 {
namespace {

constexpr int TILE = 128;      // a/b tile edge (MMA M and N)
constexpr int KSTEP = 64;      // K per stage (one 128-byte swizzle row of FP16)
constexpr int PANEL_BYTES = TILE * KSTEP * 2;  // 16 KB
constexpr long long WAIT_BUDGET = 4000000000LL;  // ~2 s of SM clock per wait

// Two waits have no bound: the allocation of tensor memory and the cluster
// barriers.  A CTA of a pair allocates all 512 columns on both its SMs, where two
// pairs holding one SM each would wait for one another; but no SM has room
// for a CTA of a pair and another CTA of these kernels that allocates at all
// (228 KB of shared memory, 1 KB of each CTA's taken by the system), so
// the columns are free when such a CTA starts.  And the CTAs of a cluster start
// together, every other wait before a cluster barrier is bounded, so each arrives.
// The permit to allocate is given up after such a barrier: no CTA may allocate once
// its pair has, and blocks of other streams can hold one of the two back.
constexpr int SM_SMEM = 228 * 1024;
constexpr int TMEM_SMEM_MIN = 75008;  // least shared memory of a kernel that allocates
constexpr bool tmem_alone(int smem) { return smem + TMEM_SMEM_MIN + 2 * 1024 > SM_SMEM; }

// --------------------------------------------------------------------------
// small PTX helpers
// --------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: returns false (and raises the CTA abort flag and the global
// error word) if the phase does not complete within the clock budget or if
// another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                          int *err, int code, long long budget = WAIT_BUDGET) {
  const long long t0 = clock64();
  while (!mbar_test(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > budget) {
      *abort_flag = 1;
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}

// The kernels before this one in the stream are complete, their writes visible
// (at once for a kernel that was launched after them).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel may be set up once every block got here.
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// K-major operand tile of 128 rows x 64 FP16 (128-byte rows), 128B swizzle,
// 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);          // start address
  d |= (uint64_t)(16 >> 4) << 16;                  // leading byte offset (unused for SW128 K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset: 8-row group pitch
  d |= (uint64_t)1 << 46;                          // descriptor version (tcgen05)
  d |= (uint64_t)2 << 61;                          // swizzle: 128B
  return d;
}

// Instruction descriptor: kind::f16, A=B=F16, D=F32, K-major A and B, M=128, N=128
constexpr uint32_t IDESC = (1u << 4)            // D format F32
                           | (0u << 7)          // A format F16
                           | (0u << 10)         // B format F16
                           | ((uint32_t)(TILE >> 3) << 17)   // N >> 3
                           | ((uint32_t)(TILE >> 4) << 24);  // M >> 4

// the same with N = 256 (two stacked 128-row B panels)
constexpr uint32_t IDESC_N256 = (1u << 4) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);

// kind::f16, F16 operands, F32 accumulator, K-major, M rows, N columns
// (M = 128: N a multiple of 16 up to 256)
__host__ __device__ constexpr uint32_t idesc_mn(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(IDESC), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_f16_id(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                           uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// --------------------------------------------------------------------------
// CTA pairs
// --------------------------------------------------------------------------
// kind::f16, A = B = F16, D = F32, K-major, M = 256 (pair), N = 128 / 256
constexpr uint32_t IDESC_PAIR = (1u << 4) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
constexpr uint32_t IDESC_PAIR_N256 = (1u << 4) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// shared::cluster address of the same shared variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}

__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}

// The same without the release: it does not wait for the thread's stores to global
// memory.  For an arrival that only says that TMEM has been read (the loads are
// complete, tcgen05.fence::before_thread_sync precedes it).
__device__ __forceinline__ void mbar_arrive_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}

__device__ __forceinline__ bool mbar_test_cl(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void st_remote_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

// TMA load into this CTA's shared memory whose completion is counted on the
// pair's (rank 0) barrier
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map,
                                                 uint32_t bar_cluster, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"((uint64_t)map), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// arrive on the barrier at this shared offset in both CTAs of the pair once
// all previously issued MMAs of this thread have completed
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}

// Bounded wait that also aborts the peer CTA on a timeout.
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, bool cluster_scope,
                                          volatile int *abort_flag, uint32_t abort_peer, int *err,
                                          int code) {
  const long long t0 = clock64();
  while (!(cluster_scope ? mbar_test_cl(bar, parity) : mbar_test(bar, parity))) {
    if (*abort_flag) return false;
    if (clock64() - t0 > WAIT_BUDGET) {
      *abort_flag = 1;
      st_remote_u32(abort_peer, 1u);
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

// Launch with the device's highest scheduling priority.  The persistent
// energy kernels of a batch graph run beside the slicing of the next launch
// group on a side branch; without priority the slicer's many small blocks,
// ready at the same moment, fill the SMs first and the energy kernel's CTAs
// wait for them to drain.  (The priority is recorded into graph nodes.)
int energy_priority() {
  static int prio = 1;
  if (prio == 1) {
    int least = 0, greatest = 0;
    prio = cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess ? greatest : 0;
  }
  return prio;
}

// overlap: the kernel may be set up while the one before it in the stream still
// runs; it calls grid_wait() before it touches memory.
template <typename... KArgs, typename... Args>
cudaError_t launch_ex(bool high, bool overlap, void (*k)(KArgs...), dim3 grid, unsigned block,
                      size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (high) {
    at[n].id = cudaLaunchAttributePriority;
    at[n++].val.priority = energy_priority();
  }
  if (overlap) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_hi(void (*k)(KArgs...), unsigned grid, unsigned block, size_t smem,
                      cudaStream_t s, Args... args) {
  return launch_ex(true, false, k, grid, block, smem, s, args...);
}

}  // namespace
}  // namespace rimp2
