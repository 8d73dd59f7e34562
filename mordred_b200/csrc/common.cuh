// common.cuh — shared device helpers for the sm_100a kernels: bulk-copy (TMA) and
// mbarrier PTX wrappers, bounded waits, the per-device status word and launch accounting.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/mordred_b200.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 900)
#error "mordred_b200 kernels target sm_100a (cp.async.bulk and mbarrier tx-counts)"
#endif

namespace mb {

static __device__ __noinline__ int slow_mod(int d, int m) { return d % m; }

// ((key - key_min) % slots) in 32-bit two's complement (crystal/join.cuh:3). Keys in
// [key_min, key_min + slots) map to themselves and the next range wraps by one
// subtraction (a dense 1-based key N lands on slot 0), both by one unsigned minimum: the
// smaller of d and d - slots (wrapping) is the slot when it lies below `slots`. Only other
// keys — and tables of more than 2^30 slots, where a negative d could look like the next
// range — divide.
__device__ __forceinline__ int pht_slot(int key, int slots, int kmin) {
  const unsigned d = static_cast<unsigned>(key) - static_cast<unsigned>(kmin), n = static_cast<unsigned>(slots);
  const unsigned h = min(d, d - n);
  if (h < n && n <= (1u << 30)) return static_cast<int>(h);
  return slow_mod(static_cast<int>(d), slots);
}

// Longest a CTA waits on one bulk-copy stage before it gives up, sets
// MB_STATUS_TIMEOUT and returns (a healthy copy lands in microseconds).
constexpr unsigned long long kWaitLimitNs = 4000000000ull;

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// Test phase `parity` of `bar`; a waiting thread is suspended until the phase completes
// or the hint (ns) elapses, so a warp waiting for a tile does not spin through issue slots.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity), "r"(1000000u)
      : "memory");
  return ok != 0;
}

// Wait for phase `parity` of `bar` to complete, for at most kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (globaltimer_ns() - t0 > kWaitLimitNs) return false;
  }
}

// L2 policy: fact-column tiles are read once, so they are marked evict-first and the
// hash tables probed alongside them keep their L2 residency.
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}

// 1-D bulk copy global -> this CTA's shared memory, completing on `bar` (no multicast).
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar,
                                         uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1], %2, [%3], %4;" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
      : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ int4 lds128(const int* p) {
  return *reinterpret_cast<const int4*>(p);
}

// Read-only 8-byte hash-table slot through the non-coherent path.
// Words that a kernel before this one in the stream may have written: hash tables, presence
// bitmaps, attribute tables, offset lists. A dependent launch (below) may begin while that kernel
// still runs, so they are plain loads — ld.global.nc and __ldg are for memory that nothing writes
// from the launch on (fact and dimension columns, cache slots).
__device__ __forceinline__ int ld_word(const int* p) {
  int v;
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned long long ld_word2(const int* p) {
  unsigned long long v;
  asm volatile("ld.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_word4(const int* p) {
  int4 v;
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// *sum += v (sign-extended), a 64-bit sum in shared memory, as two 32-bit atomics: the low
// word's old value tells whether this addition carries, and the high word takes the sign plus
// the carry — 0 for nearly every value of either sign. Every wrap of the low word is counted
// by the one addition that caused it, so the pair holds the exact sum once all have landed.
// Shared memory has no 64-bit add: a 64-bit atomicAdd is a compare-and-swap loop. 24 warps an
// SM adding to 175 sums at random: 12.3 cycles per warp operation against 46.8; to 32 sums
// 9.9 against 105; all lanes to one sum 18 against 1,989.
__device__ __forceinline__ void smem_add_i64(unsigned long long* sum, int v) {
  unsigned* w = reinterpret_cast<unsigned*>(sum);
  const unsigned lo = static_cast<unsigned>(v);
  const unsigned old = atomicAdd(w, lo);
  const unsigned hi = static_cast<unsigned>(v >> 31) + (old + lo < lo ? 1u : 0u);
  if (hi != 0u) atomicAdd(w + 1, hi);
}

// Programmatic dependent launch: a kernel launched with launch_dependent() may be set up while
// its predecessor in the stream still runs, and waits here — before it touches global memory —
// until the predecessor has completed and its writes are visible. Short kernels let their
// successor be set up from the start (allow_dependent).
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependent() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A value of a fact column read for a scattered row. The 64-byte hint keeps DRAM from fetching
// the whole 128-byte line around it, which is what a plain load does, and the value is not kept
// in L1. Query B over 24 M rows, four columns gathered at 4 % and 1.6 % of the rows: 338 MB
// from DRAM against 422 MB (367 against 414 us a call at 120 M rows).
__device__ __forceinline__ int gather_ld(const int* p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::64B.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ void set_status(unsigned int* status, unsigned int bits) {
  if (status) atomicOr(status, bits);
}

}  // namespace mb

// ---- host side -----------------------------------------------------------------
namespace mb {

// Per-device runtime state: the status word kernels report into, SM count and smem
// limits. Created once per device by mb_init (or the first launch).
struct DeviceState {
  int device = -1;
  int num_sms = 0;
  int max_smem_optin = 0;
  unsigned int* status = nullptr;  // device word, cudaMalloc'd at init
};

// Returns nullptr (and sets *err) if the current device cannot be initialised.
DeviceState* current_device_state(int* err);
void note_launches(unsigned long long n);

// Launch `fn` on `stream` so that its set-up overlaps the end of the kernel before it; `fn`
// begins with wait_for_predecessor().
template <class... Params, class... Args>
inline cudaError_t launch_dependent(void (*fn)(Params...), int grid, int block, size_t smem, cudaStream_t stream,
                                    Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, static_cast<Params>(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // reported by the caller: not for a later call to find
  return e;
}

inline int cuda_status(cudaError_t e) { return e == cudaSuccess ? MB_OK : MB_ERR_CUDA; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool aligned8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; }

}  // namespace mb
