// Shared device helpers for the pylo_b200 kernels (sm_100a).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <type_traits>

#include "pylo_b200.h"

#define NT 256                 // threads per CTA in the streaming kernels
#define NWARP (NT / 32)
#define SUMS_LO 38             // desc.sums: [0,30) feature sums, [30,38) VeLO statistics, [38,46) their low parts
#define SUMS_STRIDE 48
#define PYLO_A_ROWS_MAX 128    // rows of a row/column-sum strip

// ----------------------------------------------------------------------------------------------
// family traits: feature counts and where the twelve vector-only features sit in reference order
// (learned_optimizer.cu:59-96, celo2_kernel.cu:87-124, velo_kernel.cu:123-162)
// ----------------------------------------------------------------------------------------------
template <int FAM>
struct Fam;
template <>
struct Fam<PYLO_FAM_ADAFAC> {
  static constexpr int NF = 28, NIN = 39, H = 32, NOUT = 2;
  static constexpr int R = 13, C = 16, RR = 19, RC = 22;  // fac_r, fac_c, rsqrt(fac_r), rsqrt(fac_c)
};
template <>
struct Fam<PYLO_FAM_CELO2> {
  static constexpr int NF = 30, NIN = 30, H = 8, NOUT = 3;
  static constexpr int R = 15, C = 18, RR = 21, RC = 24;
};
template <>
struct Fam<PYLO_FAM_VELO> {
  static constexpr int NF = 30, NIN = 30, H = 4, NOUT = 3;
  static constexpr int R = 15, C = 18, RR = 21, RC = 24;
};

template <int FAM>
__host__ __device__ constexpr bool is_vec_feature(int j) {
  return j >= Fam<FAM>::R && j < Fam<FAM>::R + 12;
}

// folded-network layout inside desc.wfold (floats)
template <int FAM>
struct Fold {
  using F = Fam<FAM>;
  static constexpr int W1 = 0;                    // [NF][H], k-major
  static constexpr int B1 = W1 + F::NF * F::H;    // [H]
  static constexpr int W2 = B1 + F::H;            // [H][H], k-major
  static constexpr int B2 = W2 + F::H * F::H;     // [H]
  static constexpr int W3 = B2 + F::H;            // [H][2], k-major (only direction and magnitude)
  static constexpr int B3 = W3 + F::H * 2;        // [2]
  static constexpr int SC = B3 + 2;               // [0] param_scale (VeLO), [1] lr_eff
  static constexpr int W3P = SC + 2;              // [H/2][4]: (dir[2j], dir[2j+1], mag[2j], mag[2j+1]) for packed dot products
  static constexpr int SN = W3P + 2 * F::H;       // [NF]: the features' normalisers
  static constexpr int SIZE = SN;                 // of what a kernel with the folded network needs
};

// What the tensor-core sweep reads of a unit, behind the folded network in desc.wfold: the operands B of its products as they lie
// in shared memory (fp16 planes in the K-major no-swizzle layout: 8-row x 16-byte core matrices), then the features' scales.
struct __align__(128) TcImage {
  uint16_t b1[64 * 32];     // first layer, rows 0..31 the high planes, 32..63 the low planes; K = 32 slots (see tc_slot_feature)
  uint16_t b2[64 * 32];     // second layer
  uint16_t bias1[32 * 16];  // K = 16: column 0 the bias's high plane, column 1 what that leaves, times 2^11
  uint16_t bias2[32 * 16];
  float sn[32];             // [slot] normaliser times the features' power of two; [28] the scale of the second layer's sums
};
constexpr int TC_IMAGE = (Fold<PYLO_FAM_ADAFAC>::SN + Fam<PYLO_FAM_ADAFAC>::NF + 31) / 32 * 32;   // floats
static_assert(TC_IMAGE + (int)sizeof(TcImage) / 4 <= PYLO_WFOLD_STRIDE, "wfold too small");
// Which feature the first layer's operand A holds in slot k < 28: 0..12 and 25..27, then the six of one vector and the six of the
// other ("r" first, or "c" first where swap is set)
__host__ __device__ constexpr int tc_slot_feature(int k, bool swap) {
  using F = Fam<PYLO_FAM_ADAFAC>;
  return k < 13 ? k : k < 16 ? k + 12 : k < 19 ? (swap ? F::C : F::R) + k - 16 : k < 22 ? (swap ? F::RC : F::RR) + k - 19
         : k < 25 ? (swap ? F::R : F::C) + k - 22 : (swap ? F::RR : F::RC) + k - 25;
}

// compile-time loop: guarantees static register indexing however large the unrolled body gets
template <int I, int N, class Fn>
__device__ __forceinline__ void static_for(Fn&& fn) {
  if constexpr (I < N) {
    fn(std::integral_constant<int, I>{});
    static_for<I + 1, N>(fn);
  }
}

// First statement of every kernel: let the next kernel of the stream be set up, then wait until the previous one is
// complete and its writes are visible.  Nothing that a predecessor may write is read before.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The status word of a step: set by a kernel whose bounded wait ran out.  A kernel that writes parameters (or the LSTM's state)
// and finds it set leaves them as they are, since its inputs are incomplete, and passes the word on to the host.  It is asked
// for at the kernel's start and looked at behind the first barrier, where it has arrived with everything else.
__device__ __forceinline__ int reported(const int* status) { return status ? *reinterpret_cast<const volatile int*>(status) : 0; }
__device__ __forceinline__ void pass_on(int word, int* host_status) {
  if (word && host_status && blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<volatile int*>(host_status) = word;
}

// ----------------------------------------------------------------------------------------------
// scalar helpers
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ float lerp_torch(float a, float b, float w) {
  // torch.lerp: a + w*(b-a) for |w| < 0.5, else b - (b-a)*(1-w)
  const float d = b - a;
  return (fabsf(w) < 0.5f) ? fmaf(w, d, a) : b - d * (1.0f - w);
}

__device__ __forceinline__ float safe_rsqrt(float x) { return rsqrtf(fmaxf(x, 1e-9f)); }

// rsqrt of a value known to be a positive normal number (v + eps with eps >= 1e-8): the bare
// hardware approximation (about 1.5 ulp), without the range fix-ups rsqrtf() carries
__device__ __forceinline__ float rsqrt_pos(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float grad_scale_of(const pylo_tensor_desc& d, const pylo_step_params& prm) {
  if (d.clip_norm <= 0.0f || prm.gnorm_sq == nullptr) return 1.0f;
  const float norm = sqrtf(*prm.gnorm_sq);
  const float denom = fmaxf(norm, d.clip_norm);
  return denom > 0.0f ? d.clip_norm / denom : 1.0f;
}

// g' = clamp(nan_to_num?(g * scale), +-clip); NaN passes through the clamp like torch.clamp
__device__ __forceinline__ float xform_grad(float g, float gs, float clip, int nan2num) {
  g *= gs;
  if (nan2num) {
    if (g != g) g = 0.0f;
    else if (isinf(g)) g = g > 0 ? 3.4028234663852886e38f : -3.4028234663852886e38f;
  }
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(g) : "f"(-clip));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(g) : "f"(clip));
  return g;
}

// whether xform_grad changes nothing: no global-norm scale, no nan_to_num, no clamp (AdafacLO's defaults)
__device__ __forceinline__ bool plain_grad(float gs, const pylo_step_params& prm) {
  return !prm.nan_to_num && prm.clip_val == CUDART_INF_F && gs == 1.0f;
}

// elements of a tile of a tensor (or item) of n elements
__device__ __forceinline__ int tile_count(const pylo_tile& t, int64_t n) {
  const int64_t most = t.elems > 0 ? t.elems : PYLO_TILE_ELEMS, left = n - t.start;
  return (int)(left < most ? left : most);
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Shared-memory loads of the network weights.  They are issued as volatile PTX so that the
// compiler neither hoists thousands of loop-invariant weight loads out of the element loop
// (which would spill them to local memory) nor merges them across elements.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int OFF_FLOATS>
__device__ __forceinline__ float4 lds4(uint32_t base) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(base), "n"(OFF_FLOATS * 4));
  return v;
}
template <int OFF_FLOATS>
__device__ __forceinline__ float2 lds2(uint32_t base) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(base), "n"(OFF_FLOATS * 4));
  return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block sum of one float; result valid in every thread.  s_red: >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* s_red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < nw; ++w) t += s_red[w];
    s_red[32] = t;
  }
  __syncthreads();
  return s_red[32];
}

// Sums of accumulators FIRST .. FIRST + WIDTH - 1 over the lanes of a warp, lane l (and l + WIDTH, ...) ending with that of
// accumulator FIRST + l % WIDTH: after the step of offset o a lane holds the o of them whose index agrees with its own in that
// bit.  WIDTH - 1 shuffles (and one per halving of the lanes left), where one sum after the other takes five each.
template <int FIRST, int WIDTH, int N>
__device__ __forceinline__ float warp_fold(const float (&acc)[N]) {
  const int lane = threadIdx.x & 31;
  float a[WIDTH];
#pragma unroll
  for (int j = 0; j < WIDTH; ++j) a[j] = FIRST + j < N ? acc[FIRST + j < N ? FIRST + j : 0] : 0.f;
#pragma unroll
  for (int o = WIDTH / 2; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float keep = up ? a[j + o] : a[j], give = up ? a[j] : a[j + o];
      a[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (int o = WIDTH; o < 32; o <<= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
  return a[0];
}

// Deterministic block reduction of N per-thread accumulators; thread j < N writes out[j].
// s_red: WARPS * N floats.
template <int N, int WARPS = NWARP>
__device__ __forceinline__ void block_reduce_store(float (&acc)[N], float* s_red, float* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  static_assert(N > 16 && N <= 40, "one fold of 32, and one of 8");
  const float v = warp_fold<0, 32>(acc);
  if (lane < N) s_red[warp * N + lane] = v;
  if constexpr (N > 32) {
    const float w = warp_fold<32, 8>(acc);
    if (lane < N - 32) s_red[warp * N + 32 + lane] = w;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) t += s_red[w * N + threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// Where an element of a [O,X,M,Y,I] tensor sits: R = o*X + x and c = (m*Y + y)*I + i, the tensor being a matrix of O*X rows
// of C = M*Y*I.  A thread that walks through a tensor in equal strides moves its position by additions; one division pair
// finds the first.  R and C fit 32 bits: X and Y are the two largest sides, so either would need a tensor of over 2^33
// elements to overflow.
struct GenPos {
  uint32_t R, c, C, dR, dc, YI, Y, X, M, I;
  bool plain;     // M == I == 1: a matrix
  bool one;       // O == 1
  __device__ __forceinline__ GenPos(const pylo_tensor_desc& d, int64_t first, uint32_t stride) {
    X = d.X; Y = d.Y; M = d.M; I = d.I;
    YI = Y * I; C = M * YI;
    plain = M == 1 && I == 1;
    one = d.O == 1;
    if ((uint64_t)first < (1ull << 32)) { R = (uint32_t)first / C; c = (uint32_t)first - R * C; }
    else { R = (uint32_t)((uint64_t)first / C); c = (uint32_t)((uint64_t)first - (uint64_t)R * C); }
    dR = stride / C;
    dc = stride - dR * C;
  }
  __device__ __forceinline__ void next() {
    R += dR;
    c += dc;
    if (c >= C) { c -= C; ++R; }
  }
  // index into the "a" vectors (which drop Y) and the "b" vectors (which drop X)
  __device__ __forceinline__ int64_t a() const { return plain ? (int64_t)R : ((int64_t)R * M + c / YI) * I + c % I; }
  __device__ __forceinline__ int64_t b() const { return one ? (int64_t)c : (int64_t)(R / X) * C + c; }
};
