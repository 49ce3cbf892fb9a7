// Phase C for AdafacLO / ELO on the tensor cores (included by pylo_kernels.cu).
//
// The per-element network is a pair of small dense products, [elements x 29] x [29 x 32] and
// [elements x 32] x [32 x 32]; on the CUDA cores they cost ~1600 fp32 FMAs per element and bound the whole
// step.  Here a warpgroup (128 threads) treats 128 consecutive elements of one tensor row as the M = 128 rows
// of tcgen05 products:
//   * each thread builds its element's 16 element-wise features in registers and writes them with tcgen05.st
//     into tensor memory, where they are operand A (lane = element, column = two features);
//   * the six features that depend only on the element's column join operand A from registers, where they stay for
//     all rows of a work item; the six that depend only on its row come from shared memory, where a warpgroup makes
//     them for up to 64 rows at a time (of convolution weights, KERNEL, the row's features differ from one position to the
//     next: 14 rows of 9 positions).  First layer: K = 28 of 32;
//   * fp32 accuracy is kept by splitting every operand into two fp16 planes (11 + 11 significant bits) and running
//     three products per layer and K step (hi x hi, hi x lo, lo x hi) into one accumulator of 32 columns.  The features
//     are normalised before they are split: over its root mean square no feature exceeds sqrt(n), so that powers of two
//     can be found, for every hidden unit, that keep both layers' operands in fp16's range for any gradient (tc_network).  Operand
//     B holds the high planes in rows 0..31 and the low planes in rows 32..63 of one block; a product addresses
//     either half through its descriptor's start address;
//   * a layer's last product is of a constant operand A (in shared memory) with a block that holds the bias; the tensor
//     core scales the sums before it by 2^-TC_SHIFT.  A tile takes 7 + 7 products of width 32 (K = 16).  TF32 planes took 22
//     (K = 8), twice the operand stores, and the row's features through operand B: 8192 x 4096 elements 714 -> 678 us, step over ViT-B/16
//     2647 -> 2287, two Llama blocks 12770 -> 11480 (one GPU, in turn); the movement's error against fp64 is half of what it was
//     (4096 x 4096, normal gradients: 1.6e-7 -> 0.9e-7 rms);
//   * other tensors (ragged rows, vectors, odd convolutions) are taken as 128 consecutive elements that
//     may lie in several rows (GEN items): their twelve vector features are made per element (the scalar kernel that took them before needed 752
//     us for the 5 M parameters of a small convolutional network, FMA-bound);
//   * relu, the split of the hidden activations (whose conversions to fp16 clamp at zero by themselves), the two output heads and
//     the parameter update stay on the CUDA
//     cores, which work on one warpgroup's tile while the tensor core works on another's: four warpgroups per
//     CTA, one CTA per SM; every warpgroup is an independent worker with its own work items, its own
//     copy of the weights in shared memory, its own 64 tensor-memory columns (16 operand A high planes, 16 low
//     planes, 32 accumulator) and its own barriers, so the warpgroups drift apart instead of marching in step;
//   * the products are issued by one elected lane inside a warp-uniform branch (the warp index is a broadcast
//     from lane 0), so that their descriptors and tensor-memory addresses live in uniform registers: issued from
//     a branch on the thread index, each product cost its thread ~52 cycles; this way ~24.
//   * the output layer, one network's for all units, is an argument of the launch: read from shared memory, with no registers
//     to ask ahead, each pair of units waited for its weights (the heads took 700 of a tile's 2970 cycles, as an argument 500).
// What bounds it: issue slots (386 instructions per element, 66 % of the slots) and the latency of a tile's stages, one serial chain of
// 2500 cycles with four tiles per SM in flight, one per warpgroup (features 292, operand stores and next row's requests 169, first products
// 403, relu and split 424, second products 407, heads and store 523, waits and barriers 85, loop 110); on large models the GPU's power
// limit.  Tensor pipe 38 %, ALU pipe 38 %, fma pipe 41 %, DRAM 19 %.
// Every wait on the tensor core is bounded.  A thread whose wait ran out records it in *status (and in *host_status, a word
// of pinned host memory that the host looks at without asking the device), stops waiting
// and stops storing (its parameters, and their copies on the peers, keep their old values), and goes on to
// the end, where the kernel frees its tensor memory.  A launch that finds *status already set stores nothing.
#pragma once

#ifndef TC_WGS
// Warpgroups per CTA.  More hide more of a tile's chain, but have fewer registers each (six: 80), and at the power limit instructions
// per element count: us per step with 3, 4, 5, 6 (the first version on fp16 planes): ViT-B/16 2643, 2533, 2757, 2668, two Llama blocks
// 12530, 11926, 12740, 12625.
#define TC_WGS 4
#endif
#define TC_NT (TC_WGS * 128)
#ifndef TC_BOUND_THREADS
#define TC_BOUND_THREADS TC_NT   // a larger bound lowers the register cap (65536 / bound): room for a co-resident kernel
#endif
#define TC_COLS 128              // tensor columns per work item: one per lane of the accumulator tile
#define TC_WG_TMEM 64            // tensor-memory columns per warpgroup: [0,16) operand A high planes, [16,32) low planes, [32,64) accumulator
#define TC_ROWS 64               // FAST2D: tensor rows whose factors and features a warpgroup makes at once
#define TC_RECORDS 128           // KERNEL: the same of rows and positions
#define TC_GEN_ITEM (1 << 16)    // set in an item's tag: `strip` counts items of `rows` x 128 consecutive elements
#define TC_SPIN_LIMIT (1 << 20)
#ifndef TC_POLL_SLEEP_NS
#define TC_POLL_SLEEP_NS 40
#endif
#define TC_LBO 512               // bytes between 16-byte K chunks of a 32-row operand B (32 rows x 16 bytes)
#define TC_LBO64 1024            // the same for a 64-row operand B (high planes in rows 0..31, low planes in rows 32..63)
#define TC_SBO 128               // bytes between groups of eight rows
#define TC_LOW_HALF ((4 * TC_SBO) >> 4)   // descriptor start-address offset (16-byte units) of rows 32..63
#define TC_ONES_BYTES 2304       // constant operand A: every 16-byte chunk is (1, 2^-11, 0, ...)

__device__ __forceinline__ void tc_alloc(uint32_t* dst_smem, int ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, int ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// one lane of the (converged) warp: true in exactly one thread
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void wg_barrier(int wg) { asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory"); }

// D[128 x N] (+)= A[128 x 16] * B[N x 16]^T, A in tensor memory (two fp16 per column), B through a shared-memory descriptor
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// D = A * B^T + D * 2^-TC_SHIFT, A through a shared-memory descriptor
__device__ __forceinline__ void tc_mma_bias(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %4;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(TC_SHIFT) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok;
}
// bounded wait for the phase with the given parity to complete; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
#pragma unroll 1
  for (int it = 0; it < TC_SPIN_LIMIT; ++it) {
    if (mbar_try(a, parity)) return true;
    __nanosleep(TC_POLL_SLEEP_NS);  // back off: a waiting warp should not spend the issue slots of the working ones
  }
  return false;
}

// 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

// shared-memory matrix descriptor: start address, leading (K) and stride (row-group) byte offsets in 16-byte
// units, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, int lbo = TC_LBO, int sbo = TC_SBO) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor: fp32 accumulate, fp16 x fp16, both operands K-major, M = 128, N = 32
constexpr uint32_t TC_IDESC = (1u << 4) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

// Stage clocks (debug builds with -DTC_STAGE_CLOCKS only): lane 0 of every warpgroup's first warp adds the cycles it
// spends in each stage of a tile to status[8 + 12 * wg + stage].
#ifdef TC_STAGE_CLOCKS
#define TC_CLK_DECL long long clk_acc[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}; long long clk_t = clock64();
#define TC_CLK(stage) { const long long now_ = clock64(); clk_acc[stage] += now_ - clk_t; clk_t = now_; }
#define TC_CLK_FLUSH if (col == 0 && status) { for (int q_ = 0; q_ < 12; ++q_) atomicAdd(status + 8 + 12 * wg + q_, (int)(clk_acc[q_] >> 10)); }
#else
#define TC_CLK_DECL
#define TC_CLK(stage)
#define TC_CLK_FLUSH
#endif

// Two values as fp16 planes: hi the values cut to fp16, lo what that leaves, rounded; packed, the first value in the
// lower half.  RELU: of the values' positive parts: the high plane of a negative value is zero and what it leaves negative, so both
// conversions clamp at zero by themselves.
template <bool RELU>
__device__ __forceinline__ void tc_split2(uint64_t x, uint32_t& hi, uint32_t& lo) {
  float a, b;
  unpack2(x, a, b);
  if constexpr (RELU) asm("cvt.rz.relu.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
  else asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
  const float2 cut = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  float ra, rb;
  unpack2(fma2(pack2(cut.x, cut.y), pack2(-1.f, -1.f), x), ra, rb);   // exact
  if constexpr (RELU) asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(rb), "f"(ra));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(rb), "f"(ra));
}

// One warpgroup's private shared memory: its copy of the weights and its tensor-core barrier.  Warpgroups never
// wait on one another.
struct __align__(128) TcWgSmem {
  TcImage img;               // of the unit of the present item
  float row[TC_RECORDS][12]; // FAST2D, KERNEL, per tensor row (and position): three factors, then its six features as three words of high and three of low planes
  float w3[64 + 4];          // output layer, pair-major (Fold::W3P), then its two biases
  uint64_t bar;
};
struct TcSmem {
  TcWgSmem wg[TC_WGS];
  __align__(128) uint32_t ones[TC_ONES_BYTES / 4];
  uint32_t tmem_base;
  int poisoned;  // the status word at launch: non-zero means an earlier launch reported a timed-out wait
};

// The output layer as an argument of the launch, where one network serves all units: pairs of units' direction and magnitude weights
// (Fold::W3P), then the two biases.
struct TcHeads { float w[64], b[2]; };

// GENERIC: the launch may hold items on tensors that are not FAST2D.  The variant without them is the faster one on large
// models (their body costs the other one registers: 2 % of the step over two Llama blocks).
template <bool GENERIC, bool ARG>
__global__ void __launch_bounds__(TC_BOUND_THREADS, 1) k_apply_adafac_tc(const pylo_tensor_desc* __restrict__ descs,
                                                              const pylo_atile* __restrict__ ttiles, int n_ttiles,
                                                              const pylo_step_params prm, int* __restrict__ status,
                                                              int* __restrict__ host_status, const __grid_constant__ TcHeads heads_arg) {
  using F = Fam<PYLO_FAM_ADAFAC>;
  using L = Fold<PYLO_FAM_ADAFAC>;
  extern __shared__ __align__(128) unsigned char tc_raw[];
  TcSmem& smem = *reinterpret_cast<TcSmem*>(tc_raw);
  const int tid = threadIdx.x, col = tid & 127;
  // The warp index as a value the compiler knows to be the same in all lanes (a broadcast from lane 0): the branch
  // that issues the products is then warp-uniform and its operands (descriptors, tensor-memory addresses) live in
  // uniform registers.  Issued from a branch on the thread index instead, a product cost its thread ~52 cycles on
  // top of the ~270 of the first; this way ~24 (6 products: 240 cycles instead of 522).
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), wg = warp >> 2;
  TcWgSmem& sm = smem.wg[wg];
  if (col == 0) mbar_init(&sm.bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int e = tid; e < TC_ONES_BYTES / 4; e += TC_NT) smem.ones[e] = e & 3 ? 0u : 0x10003c00u;
  pdl_begin();  // the set-up so far overlaps the previous kernel's end
  if (tid == 32) smem.poisoned = status ? *reinterpret_cast<volatile int*>(status) : 0;
  if (warp == 0) { tc_alloc(&smem.tmem_base, 512); tc_relinquish(); }
  fence_async_smem();  // the constant operand is read by the tensor core through the async proxy
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // A launch that finds the status word already set writes nothing (no parameter, no peer store): the
  // parameters stay as the last good step left them until the host has looked at the error and cleared it.
  const int n_items = smem.poisoned ? 0 : n_ttiles;
  if (smem.poisoned && host_status && blockIdx.x == 0 && tid == 0) *reinterpret_cast<volatile int*>(host_status) = smem.poisoned;
  const uint32_t t_wg = __shfl_sync(0xffffffffu, smem.tmem_base, 0) + wg * TC_WG_TMEM;   // lane 0 of this warpgroup's columns
  const uint32_t t_lane = t_wg + ((uint32_t)((warp & 3) * 32) << 16);   // this warp's 32 lanes
  const uint32_t tA = t_lane, tD = t_lane + 32;
  constexpr uint64_t KSTEP64 = (2 * TC_LBO64) >> 4;  // one product consumes two K chunks of operand B
  // every chunk of the constant operand is (1, 2^-11, 0, ...): any in-range chunk of the buffer holds that pattern
  const uint64_t desc_ones = tc_desc(smem_addr(smem.ones), 128, 128);
  uint32_t parity = 0;
  bool timed_out = false;
  int loaded = -1;
  TC_CLK_DECL
  // every warpgroup is a worker of its own: it takes every (gridDim.x * TC_WGS)-th work item
  for (int t = blockIdx.x * TC_WGS + wg; t < n_items; t += gridDim.x * TC_WGS) {
    const pylo_atile ct = ttiles[t];
    const pylo_tensor_desc& d = descs[ct.tensor];
    const int rows_item = ct.pad_ & (TC_GEN_ITEM - 1);  // rows (tiles of 128 elements) per work item
    // One item: on a FAST2D tensor, a KERNEL one, or (GEN) any other.  A body for each, so that none holds another's registers.
    auto item = [&](auto mode_tag) {
    constexpr bool GEN = decltype(mode_tag)::value == PYLO_MODE_GENERIC, KERNEL = decltype(mode_tag)::value == PYLO_MODE_KERNEL;
    const int I = KERNEL ? d.I : 1;   // positions; a matrix of Y * I columns
    const int X = d.X, Y = d.Y * I;
    const int64_t n = d.n;
    const int y = ct.cb * TC_COLS + col;
    const int x0 = ct.strip * rows_item;
    const int x_end = x0 + (int)min((int64_t)rows_item, (GEN ? (n + TC_COLS - 1) / TC_COLS : (int64_t)X) - x0);
    const int64_t e0 = (int64_t)x0 * TC_COLS + col;      // GEN: this thread's first element
    const bool colok = y < Y;
    const int yc = colok ? y : 0;
    const float* __restrict__ gp = d.g;
    float* __restrict__ pp = d.p;
    const float* __restrict__ mp = d.m;
    const float* __restrict__ vp = d.v;
    const float *m1p = mp + n, *m2p = m1p + n;
    uint32_t at_next = (uint32_t)x0 * (uint32_t)Y + yc, at = 0;   // FAST2D: the elements whose operands are asked for next, and of this row
    // GEN: the accumulators of the "r" and "c" vectors and the "r" factor (the "c" factor is a function of its accumulator)
    const bool vec1d = d.mode == PYLO_MODE_VEC1D, r_is_a = d.r_is_a != 0;
    const float* __restrict__ facr = GEN ? (r_is_a ? d.fac_a : d.fac_b) : nullptr;
    const float* __restrict__ facc = GEN ? (vec1d ? (d.fac_b ? d.fac_b : d.fac_a) : (r_is_a ? d.fac_b : d.fac_a)) : nullptr;
    const float* __restrict__ frp = GEN && !vec1d ? (r_is_a ? d.f_a : d.f_b) : nullptr;
    const int64_t Lr = vec1d ? n : (r_is_a ? d.La : d.Lb), Lc = vec1d ? n : (r_is_a ? d.Lb : d.La);
    GenPos pos(d, GEN && !vec1d ? e0 : 0, TC_COLS);
    float cg, cp, cm0, cm1, cm2, cv;
    float4 cfa;          // GEN: the element's "r" factors (vectors: unused)
    float cr[3], cc[3];  // GEN: the element's accumulators
    auto load_row = [&](int x, float& g, float& p, float& m0, float& m1, float& m2, float& v) {
      if constexpr (GEN) {
        const int64_t e = (int64_t)x * TC_COLS + col;
        const int64_t idx = e < n ? e : 0;
        g = ldg_early(gp + idx); p = ldg_early(pp + idx); m0 = ldg_early(mp + idx);
        m1 = ldg_early(mp + n + idx); m2 = ldg_early(mp + 2 * n + idx); v = ldg_early(vp + idx);
        int64_t ir = idx, ic = idx;
        if (!vec1d) {
          const int64_t a = e < n ? pos.a() : 0, b = e < n ? pos.b() : 0;
          pos.next();
          ir = r_is_a ? a : b; ic = r_is_a ? b : a;
          cfa.x = ldg_early(frp + ir); cfa.y = ldg_early(frp + Lr + ir); cfa.z = ldg_early(frp + 2 * Lr + ir);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) { cr[k] = ldg_early(facr + k * Lr + ir); cc[k] = ldg_early(facc + k * Lc + ic); }
      } else {
        const uint32_t idx = at_next;   // n < 2^31 here
        g = ldg_early(gp + idx); p = ldg_early(pp + idx); m0 = ldg_early(mp + idx);
        m1 = ldg_early(m1p + idx); m2 = ldg_early(m2p + idx); v = ldg_early(vp + idx);
      }
    };
    load_row(x0, cg, cp, cm0, cm1, cm2, cv);   // in flight during the set-up
    // per-item constants: in registers for all rows of the item
    float fb0 = 0.f, fb1 = 0.f, fb2 = 0.f, fc[3];   // FAST2D: the column's factors and accumulators
    if constexpr (!GEN) {
      fb0 = __ldg(d.f_b + yc); fb1 = __ldg(d.f_b + Y + yc); fb2 = __ldg(d.f_b + 2 * (int64_t)Y + yc);
#pragma unroll
      for (int k = 0; k < 3; ++k) fc[k] = colok ? __ldg(d.fac_b + (int64_t)k * Y + yc) : 0.f;
    }
    const Peers peers = load_peers(d);
    const float gs = grad_scale_of(d, prm);
    const Fin fin{d.exp_mult, d.step_mult, d.wd, d.lr, __ldg(d.wfold + L::SC + 1), 1.0f, prm.wd_mode};
    const bool plain = plain_grad(gs, prm);
    wg_barrier(wg);  // the four warps are done with the previous item's weights
    if (loaded != ct.tensor) {
      const float4* __restrict__ src = reinterpret_cast<const float4*>(d.wfold + TC_IMAGE);
      float4* dst = reinterpret_cast<float4*>(&sm.img);
#pragma unroll
      for (int e = 0; e < (int)sizeof(TcImage) / 16; e += 128)
        if (e + col < (int)sizeof(TcImage) / 16) dst[e + col] = __ldg(src + e + col);
      if (!ARG && col < 64) sm.w3[col] = __ldg(d.wfold + L::W3P + col);
      if (!ARG && col < 2) sm.w3[64 + col] = __ldg(d.wfold + L::B3 + col);
      loaded = ct.tensor;
      // small models: k_small_front has left the network and the partial sums of squares; the features' scales are made here, the
      // partials added up as unit_sum does
      if (GENERIC && prm.no_tables == 4) {
        double(*const part)[32] = reinterpret_cast<double(*)[32]>(sm.row);
        static_assert(TC_SUM_ROWS == 4, "a warp per row");
        const int q = warp & 3, j = col & 31, f = tc_slot_feature(j < F::NF ? j : 0, tc_swap(d));
        const float closed = d.closed[f];
        double acc = 0.0;
        for (int t = q; t < d.n_tiles; t += TC_SUM_ROWS) acc += (double)d.tile_part[(int64_t)t * PYLO_STAT_STRIDE + f];
        part[q][j] = acc;
        wg_barrier(wg);
        if (col < F::NF) {
          const float tot = (float)(part[0][col] + part[1][col] + part[2][col] + part[3][col] + (double)closed);
          sm.img.sn[col] = rsqrtf(tot / (float)n + prm.eps_norm) * sm.img.sn[F::NF + 1];
          if (ct.strip == 0 && ct.cb == 0) d.sums[f] = tot;
        }
      }
      fence_async_smem();  // the tensor core reads the weights through the async proxy
      wg_barrier(wg);
    }
    const float* __restrict__ sn = sm.img.sn;
    const float out_scale = sn[F::NF];
    // six features of one vector (a row's, a column's): its accumulators and their inverse roots, from slot k on
    auto planes6 = [&](int k, float v0, float v1, float v2, uint32_t (&hi)[3], uint32_t (&lo)[3]) {
      tc_split2<false>(pack2(v0 * sn[k], v1 * sn[k + 1]), hi[0], lo[0]);
      tc_split2<false>(pack2(v2 * sn[k + 2], rsqrtf(v0 + 1e-8f) * sn[k + 3]), hi[1], lo[1]);
      tc_split2<false>(pack2(rsqrtf(v1 + 1e-8f) * sn[k + 4], rsqrtf(v2 + 1e-8f) * sn[k + 5]), hi[2], lo[2]);
    };
    uint32_t chi[3] = {0u, 0u, 0u}, clo[3] = {0u, 0u, 0u};
    if constexpr (!GEN)
      if (colok) planes6(16, fc[0], fc[1], fc[2], chi, clo);
    TC_CLK(7)  // item set-up
    const float* rec = nullptr;   // KERNEL: of this row and this thread's position
    int ready = 0;                // rows ahead whose factors and features are there
#pragma unroll 1
    for (int x = x0; x < x_end; ++x) {   // the same for the whole warpgroup
      const int i = x - x0;
      if (KERNEL ? ready == 0 : !GEN && (i & (TC_ROWS - 1)) == 0) {   // the next rows' factors and features (the previous ones were read before a barrier)
        ready = min(KERNEL ? TC_RECORDS / I : TC_ROWS, x_end - x);
        if (col < ready * I) {
          const int64_t a = (int64_t)x * I + col, La = (int64_t)X * I;
          const float4 f = ld4(d.fx + 4 * a);
          uint32_t hi[3], lo[3];
          planes6(22, d.fac_a[a], d.fac_a[La + a], d.fac_a[2 * La + a], hi, lo);
          float* q = sm.row[col];
          st4(q, make_float4(f.x, f.y, f.z, __uint_as_float(hi[0])));
          st4(q + 4, make_float4(__uint_as_float(hi[1]), __uint_as_float(hi[2]), __uint_as_float(lo[0]), __uint_as_float(lo[1])));
          q[8] = __uint_as_float(lo[2]);
        }
        if (KERNEL) rec = sm.row[yc % I];
        wg_barrier(wg);
      }
      TC_CLK(8)  // loop overhead, rows' features
      // ---- operand A of the first layer, high and low planes
      {
        const float g = plain ? cg : xform_grad(cg, gs, prm.clip_val, prm.nan_to_num);
        const float rs = rsqrt_pos(cv + prm.eps_feat);
        float k0, k1, k2;
        uint32_t hi[16], lo[16];
        if constexpr (GEN) {
          k0 = vec1d ? safe_rsqrt(cr[0] + 1e-9f) : cfa.x * safe_rsqrt(cc[0]);
          k1 = vec1d ? safe_rsqrt(cr[1] + 1e-9f) : cfa.y * safe_rsqrt(cc[1]);
          k2 = vec1d ? safe_rsqrt(cr[2] + 1e-9f) : cfa.z * safe_rsqrt(cc[2]);
          uint32_t h[3], l[3];
          planes6(16, cr[0], cr[1], cr[2], h, l);
#pragma unroll
          for (int j = 0; j < 3; ++j) { hi[8 + j] = h[j]; lo[8 + j] = l[j]; }
          planes6(22, cc[0], cc[1], cc[2], h, l);
#pragma unroll
          for (int j = 0; j < 3; ++j) { hi[11 + j] = h[j]; lo[11 + j] = l[j]; }
        } else {
          const float* q = KERNEL ? rec : sm.row[i & (TC_ROWS - 1)];
          const float4 r0 = ld4(q), r1 = ld4(q + 4);
          k0 = r0.x * fb0; k1 = r0.y * fb1; k2 = r0.z * fb2;
#pragma unroll
          for (int j = 0; j < 3; ++j) { hi[8 + j] = chi[j]; lo[8 + j] = clo[j]; }
          hi[11] = __float_as_uint(r0.w); hi[12] = __float_as_uint(r1.x); hi[13] = __float_as_uint(r1.y);
          lo[11] = __float_as_uint(r1.z); lo[12] = __float_as_uint(r1.w); lo[13] = __float_as_uint(q[8]);
          if (KERNEL) { rec += 12 * I; --ready; }
        }
        hi[14] = hi[15] = lo[14] = lo[15] = 0u;
        const uint64_t fe[8] = {pack2(g, cp), pack2(cm0, cm1), pack2(cm2, cv), pack2(cm0 * rs, cm1 * rs), pack2(cm2 * rs, rs),
                                pack2(k0 * g, k1 * g), pack2(k2 * g, k0 * cm0), pack2(k1 * cm1, k2 * cm2)};
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(sn + 2 * j);
          tc_split2<false>(mul2(fe[j], s.x), hi[j], lo[j]);
          tc_split2<false>(mul2(fe[j + 1], s.y), hi[j + 1], lo[j + 1]);
        }
        TC_CLK(10)  // features and split
        tc_st16(tA, hi);
        tc_st16(tA + 16, lo);
      }
      // the next row's operands: requested now that this row's are consumed (only p is still needed, for the
      // update), so the two sets never share the register file; they land during the two products.  (Requesting
      // them at the top of the iteration instead, into registers of their own, measured 12 % slower.)
      float np_;
      at = at_next;
      if (x + 1 < x_end) at_next += Y;   // behind the last row, that row again
      load_row(x + 1, cg, np_, cm0, cm1, cm2, cv);
      TC_CLK(0)  // stores issued, next row requested
      tc_wait_st();
      tc_fence_before();
      wg_barrier(wg);
      TC_CLK(1)  // wait for the stores + warpgroup barrier
      auto products = [&](const uint16_t* b, const uint16_t* bias) {
        if ((warp & 3) == 0) {
          if (elect_one()) {
            tc_fence_after();
            const uint64_t desc = tc_desc(smem_addr(b), TC_LBO64);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              tc_mma(t_wg + 32, t_wg + 16 + 8 * s, desc + s * KSTEP64, TC_IDESC, s > 0);          // lo x hi
              tc_mma(t_wg + 32, t_wg + 8 * s, desc + TC_LOW_HALF + s * KSTEP64, TC_IDESC, 1);     // hi x lo
            }
#pragma unroll
            for (int s = 0; s < 2; ++s) tc_mma(t_wg + 32, t_wg + 8 * s, desc + s * KSTEP64, TC_IDESC, 1);   // hi x hi
            tc_mma_bias(t_wg + 32, desc_ones, tc_desc(smem_addr(bias)), TC_IDESC);
            tc_commit(&sm.bar);
          }
          __syncwarp();
        }
        if (!timed_out && !mbar_wait(&sm.bar, parity)) timed_out = true;
        parity ^= 1;
        tc_fence_after();
      };
      products(sm.img.b1, sm.img.bias1);
      TC_CLK(2)  // first-layer products: issue + wait
      // ---- hidden layer 1: relu, split, back into tensor memory as operand A
      {
        uint32_t d0[16], d1[16], hi[16], lo[16];
        tc_ld16(tD, d0);        // everything is requested before anything is touched: one load latency
        tc_ld16(tD + 16, d1);
        tc_wait_ld();
        TC_CLK(3)  // accumulator read-back
        // A feature that is not a number makes all 32 sums that: as fmaxf does, it counts as zero.
        if (__any_sync(0xffffffffu, isnan(__uint_as_float(d0[0])))) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            d0[k] = __float_as_uint(fmaxf(__uint_as_float(d0[k]), 0.f));
            d1[k] = __float_as_uint(fmaxf(__uint_as_float(d1[k]), 0.f));
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          tc_split2<true>(pack2(__uint_as_float(d0[2 * k]), __uint_as_float(d0[2 * k + 1])), hi[k], lo[k]);
          tc_split2<true>(pack2(__uint_as_float(d1[2 * k]), __uint_as_float(d1[2 * k + 1])), hi[8 + k], lo[8 + k]);
        }
        tc_st16(tA, hi);
        tc_st16(tA + 16, lo);
      }
      TC_CLK(4)  // relu, split, stores issued
      tc_wait_st();
      tc_fence_before();
      wg_barrier(wg);
      TC_CLK(1)
      products(sm.img.b2, sm.img.bias2);
      TC_CLK(5)  // second-layer products: issue + wait
      // ---- hidden layer 2 (relu) and the two output heads as packed dot products over unit pairs
      uint64_t od[2] = {0ull, 0ull}, om[2] = {0ull, 0ull};
      {
        uint32_t d0[16], d1[16];
        tc_ld16(tD, d0);
        tc_ld16(tD + 16, d1);
        tc_wait_ld();
        TC_CLK(3)
        auto heads = [&](const uint32_t (&a)[16], int half) {
#pragma unroll
          for (int jp = 0; jp < 8; ++jp) {
            ulonglong2 w;   // (dir pair, mag pair)
            if constexpr (ARG) {
              const float* q = &heads_arg.w[4 * (half * 8 + jp)];
              w = make_ulonglong2(pack2(q[0], q[1]), pack2(q[2], q[3]));
            } else {
              w = *reinterpret_cast<const ulonglong2*>(&sm.w3[4 * (half * 8 + jp)]);
            }
            const uint64_t r = pack2(fmaxf(__uint_as_float(a[2 * jp]), 0.f), fmaxf(__uint_as_float(a[2 * jp + 1]), 0.f));
            od[jp & 1] = fma2(w.x, r, od[jp & 1]);
            om[jp & 1] = fma2(w.y, r, om[jp & 1]);
          }
        };
        heads(d0, 0);
        heads(d1, 1);
      }
      {
        float a, b, c, dd;
        unpack2(add2(od[0], od[1]), a, b);
        unpack2(add2(om[0], om[1]), c, dd);
        const float o0 = fmaf(a + b, out_scale, ARG ? heads_arg.b[0] : sm.w3[64]), o1 = fmaf(c + dd, out_scale, ARG ? heads_arg.b[1] : sm.w3[65]);
        const int64_t idx = GEN ? (int64_t)x * TC_COLS + col : at;
        if ((GEN ? idx < n : colok) && !timed_out) {  // after a wait that ran out the accumulators are not to be trusted: keep the old value
          const float pn = finish<PYLO_FAM_ADAFAC>(cp, o0, o1, fin);
          pp[idx] = pn;
          peer_store(peers, idx, pn);
        }
      }
      cp = np_;
      TC_CLK(6)  // heads, update, store
    }
    };
    if constexpr (GENERIC) {
      if (ct.pad_ & TC_GEN_ITEM) item(std::integral_constant<int, PYLO_MODE_GENERIC>{});
      else if (d.mode == PYLO_MODE_KERNEL) item(std::integral_constant<int, PYLO_MODE_KERNEL>{});
      else item(std::integral_constant<int, PYLO_MODE_FAST2D>{});
    } else {
      item(std::integral_constant<int, PYLO_MODE_FAST2D>{});
    }
  }
  TC_CLK_FLUSH
  if (timed_out && status) atomicOr(status, 1);
  if (timed_out && host_status) *reinterpret_cast<volatile int*>(host_status) = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tc_dealloc(smem.tmem_base, 512);
}
