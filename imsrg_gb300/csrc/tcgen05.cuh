// mbarrier, TMA and tcgen05 primitives of the tensor-core products
// (kernels_split.cu, kernels_dgemm.cu), as inline PTX for sm_103a.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <stdexcept>

namespace imsrg {

// bounded spin: every mbarrier wait gives up after WAIT_LIMIT try_wait rounds.
// One round (try_wait's own suspend plus the nanosleep backoff) measured
// about 8000 SM cycles on GB300 (imsrg_space_wait_selftest), so the bound is
// about 2 s at 2 GHz; the longest wait of a healthy launch (one tile's MMAs)
// is microseconds
constexpr unsigned WAIT_LIMIT = 1u << 19;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned a, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned a, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned a)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}

__device__ __forceinline__ bool mbar_try(unsigned a, unsigned parity)
{
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait: false on timeout
__device__ __forceinline__ bool mbar_wait(unsigned a, unsigned parity, unsigned limit)
{
  for (unsigned it = 0; it < limit; ++it) {
    if (mbar_try(a, parity)) return true;
    if (it > 64) __nanosleep(it > 4096 ? 256 : 32);
  }
  return false;
}

// one box of all S digit planes: coordinates (K element, plane row, digit 0)
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(dst),
      "l"((unsigned long long)map), "r"(x), "r"(y), "r"(0), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_mma(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc,
                                       unsigned idesc, unsigned accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tc_commit(unsigned bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// UMMA shared-memory descriptor: K-major operand, 64-byte swizzle
// (8 rows x 64 bytes per swizzle atom, 512 bytes between 8-row groups).
__device__ __forceinline__ unsigned long long sdesc_sw64(unsigned addr)
{
  unsigned long long d = 0;
  d |= (unsigned long long)((addr >> 4) & 0x3FFF);
  d |= (unsigned long long)1 << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (unsigned long long)(512 >> 4) << 32;    // stride byte offset
  d |= (unsigned long long)1 << 46;             // descriptor version (sm_100 family)
  d |= (unsigned long long)4 << 61;             // layout: 64-byte swizzle
  return d;
}

// instruction descriptor, kind::f16: BF16 x BF16 -> F32, both K-major
// (bit 13, set by the caller where needed, negates the A operand)
__host__ __device__ constexpr unsigned idesc_bf16(int M, int N)
{
  return (1u << 4)                   // D format F32
         | (1u << 7)                 // A format BF16
         | (1u << 10)                // B format BF16
         | ((unsigned)(N >> 3) << 17)  // N / 8
         | ((unsigned)(M >> 4) << 24); // M / 16
}

__device__ __forceinline__ void tmem_ld8(unsigned taddr, unsigned (&r)[8])
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void set_status(int* st, int code)
{
  if (st) atomicCAS(st, 0, code);
}

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline PFN_encodeTiled get_encode()
{
  static PFN_encodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
      throw std::runtime_error("cuTensorMapEncodeTiled unavailable");
    fn = (PFN_encodeTiled)p;
  }
  return fn;
}

// Named barrier `id` over `n` threads that tells all of them whether any arrived
// with bad set.  (A shared flag read after a plain barrier can be set by a
// thread that is past it already: some would leave, others wait for them.)
__device__ __forceinline__ bool barrier_any(int id, int n, bool bad)
{
  unsigned any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n}"
               : "=r"(any)
               : "r"(bad ? 1u : 0u), "r"(id), "r"(n)
               : "memory");
  return any != 0;
}

// After a wait that ran out, before the CTA frees its tensor memory and exits:
// waits (again with a limit) for the TMA loads still on their way into its
// shared memory and for the MMAs it issued.  Called by every thread once all
// roles have left their loops; issued: loads issued so far, stage k % nstage each;
// drain: a barrier (count 1) that nothing else uses; the MMAs are those of thread 32.
template <class Bar>
__device__ __forceinline__ void drain_products(int issued, int nstage, const Bar& full_bar, unsigned drain)
{
  if (threadIdx.x == 0) {
    for (int k = issued > nstage ? issued - nstage : 0; k < issued; ++k)
      mbar_wait(full_bar(k % nstage), (unsigned)((k / nstage) & 1), WAIT_LIMIT);
  } else if (threadIdx.x == 32) {
    tc_commit(drain);
    mbar_wait(drain, 0, WAIT_LIMIT);
  }
  __syncthreads();
}

}  // namespace imsrg
