// Bulk asynchronous copies (global -> shared, cp.async.bulk) completed through
// an mbarrier transaction count, with bounded waits.
//
// Every copy reads this GPU's own memory into the issuing CTA's shared memory
// only (no copies into other CTAs of a cluster).  Copies need 16-byte aligned
// source and destination and a size that is a multiple of 16 bytes.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pmb {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Default poll limit of a bounded wait (pmb_set_wait_limit changes the limit
// of the first wait; the drain after a timeout always uses this one).
constexpr uint32_t kWaitPolls = 1u << 22;

// Waits for the given phase parity of the barrier; gives up after `polls`
// polls (each poll may suspend the thread for a short, hardware-defined time;
// 0 polls gives up at once) and returns false.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t polls = kWaitPolls) {
  for (uint32_t it = 0; it < polls; ++it) {
    uint32_t done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Programmatic dependent launch: a kernel launched with launch_dependent may
// start before the kernel ahead of it on the stream has ended (once that one's
// blocks have all called let_next_start or ended); from wait_for_previous on,
// all that the stream did before is complete and visible.  Every thread calls
// wait_for_previous before it touches anything but its own shared memory and
// constants of the module.  Such a kernel is resident while its inputs are still
// being written, so it reads them by ordinary loads: no __ldg and no const
// __restrict__ parameters, which would let the compiler take the non-coherent path
// or move a load above the wait.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Where a dependent launch pays: meshes of up to 2^23 cells, whose force is a
// chain of ten kernels of 4 to 14 us with everything in L2.  Force 64^3 on
// 128^3 cells 103.1 -> 85.1 us, 96^3 on 192^3 231.4 -> 216.2, a ten-step run
// of the former 1191 -> 1061; with the same launches on every mesh 256^3 on
// 512^3 went 2637 -> 3675 us and a differentiable run on 256^3 8.75 -> 9.46 ms.
// One mesh decides for a class of an ensemble too, whose passes run over all its
// members in one launch: a force early / plain, 6 members of 64^3 395 / 403 us, 24
// 1451 / 1456, 96 5639 / 5647, 24 members of 96^3 4407 / 4407.  Many particles on a
// small mesh gain little and lose nothing but in the deposit (cic.cu, launch_rows).
constexpr int64_t kDependentCells = (int64_t)1 << 23;
inline bool small_mesh(int64_t nx, int64_t ny, int64_t nz) { return nx * ny * nz <= kDependentCells; }

// early: may start before the kernel ahead has ended; false is a plain launch.
template <class... P, class... A>
inline cudaError_t launch_dependent(bool early, void (*kernel)(P...), int grid, int threads, size_t smem,
                                    cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...), last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

// After a timed-out wait on ring slot `first` of an S-stage ring whose slots
// [first, end) were issued: waits (kWaitPolls each) for every copy still in
// flight, so that none lands in shared memory after the CTA has moved on.  If
// one of these waits gives up as well, the launch's results are undefined;
// the timeout is reported either way.
__device__ __forceinline__ void mbar_drain(uint64_t* bars, int S, int first, int end) {
  for (int j = first; j < end && j < first + S; ++j) mbar_wait(&bars[j % S], (uint32_t)((j / S) & 1));
}

// Wait used by every thread of a CTA after issuing bulk copies on one
// barrier: on a timeout the counter (a device variable of the calling file,
// reported by pmb_wait_timeouts and pmb_device_status) is raised and the
// copies still in flight get the drain wait before the caller returns without
// touching the staged data.
__device__ __forceinline__ bool mbar_wait_or_flag(uint64_t* bar, uint32_t parity, unsigned int* timeouts,
                                                  uint32_t polls = kWaitPolls) {
  if (__syncthreads_or(!mbar_wait(bar, parity, polls)) == 0) return true;
  if (threadIdx.x == 0) atomicAdd(timeouts, 1u);
  mbar_wait(bar, parity);
  return false;
}

}  // namespace pmb
