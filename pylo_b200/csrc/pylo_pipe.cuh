// A ring of shared-memory stages that the first warp of a CTA fills with bulk copies, PIPE_STAGES - 1 ahead of what all
// eight warps consume (included by pylo_kernels.cu).
//
// The sweeps over a tensor read six streams (gradient, parameter, three momenta, second moment).  Loaded into registers, a
// thread can have one or two float4 of each in flight, which with two CTAs of 256 threads per SM is 50 KB; the ring has
// 72 KB per CTA on the way whatever the warps are doing, and their registers are free for the arithmetic.  (A ninth warp for
// the copies alone costs every other one a fifth of its registers.)
#pragma once

#define PIPE_STAGES 4
#define PIPE_STREAMS 6
#define PIPE_ELEMS 1024                  // elements of a stream per stage: one float4 per thread
#define PIPE_SPIN_LIMIT (1 << 22)

struct PipeSmem {
  float st[PIPE_STAGES][PIPE_STREAMS][PIPE_ELEMS];
  uint64_t full[PIPE_STAGES], empty[PIPE_STAGES];
};

__device__ __forceinline__ void pipe_init(PipeSmem& p) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < PIPE_STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&p.full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&p.empty[s])), "r"(NWARP) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}
// bounded wait of a whole warp for the phase with the given parity; false, in all of its lanes, if it ran out
__device__ __forceinline__ bool pipe_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  uint32_t ok = 0;
  for (int it = 0; it < PIPE_SPIN_LIMIT && !ok; ++it)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ bool pipe_wait_full(PipeSmem& p, uint32_t k) { return pipe_wait(&p.full[k % PIPE_STAGES], (k / PIPE_STAGES) & 1); }
// the calling warp has read stage k
__device__ __forceinline__ void pipe_release(PipeSmem& p, uint32_t k) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&p.empty[k % PIPE_STAGES])) : "memory");
}
// first warp: wait until stage k is free and announce `bytes` for it
__device__ __forceinline__ bool pipe_begin(PipeSmem& p, uint32_t k, uint32_t bytes) {
  if (k >= PIPE_STAGES && !pipe_wait(&p.empty[k % PIPE_STAGES], (k / PIPE_STAGES - 1) & 1)) return false;
  if ((threadIdx.x & 31) == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&p.full[k % PIPE_STAGES])), "r"(bytes) : "memory");
  __syncwarp();
  return true;
}
// one copy; both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void pipe_copy(PipeSmem& p, uint32_t k, int stream, int at, const float* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_addr(&p.st[k % PIPE_STAGES][stream][at])), "l"(src), "r"(bytes), "r"(smem_addr(&p.full[k % PIPE_STAGES])) : "memory");
}
// first warp, after a failed wait: nothing may be on its way into shared memory when the CTA ends
__device__ __forceinline__ void pipe_drain(PipeSmem& p, uint32_t k) {
  for (uint32_t q = k > PIPE_STAGES ? k - PIPE_STAGES : 0; q < k; ++q) pipe_wait_full(p, q);
}
__device__ __forceinline__ void pipe_failed(const pylo_step_params& prm) {
  if (prm.status) atomicOr(prm.status, 8);
  if (prm.host_status) *reinterpret_cast<volatile int*>(prm.host_status) = 8;
}
