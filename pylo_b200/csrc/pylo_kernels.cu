// pylo_b200: learned-optimizer step kernels for B200 (sm_100a) and their C ABI.
//
// One optimizer step is a fixed sequence of launches over a device-resident
// table of tensor descriptors and tile lists (see include/pylo_b200.h):
//   [grad_sumsq] -> rowcol_sums (A) -> factor_update (A2) -> state_moments (B)
//   -> finalize_moments (B2) -> [velo front end] -> prep_apply (P) -> apply (C)
//   -> [celo2 post] / [adamw]
// All reductions go through fixed-slot partials and fixed-order final sums, so
// results are bit-reproducible from run to run (no floating-point atomics).

#include <stddef.h>
#include <string.h>

#include <mutex>

#include "pylo_common.cuh"
#include "pylo_pipe.cuh"

// ================================================================================================
// feature construction (reference order; learned_optimizer.cu:59-96, celo2_kernel.cu:87-124)
// ================================================================================================
template <int FAM>
__device__ __forceinline__ void elem_features(float* f, float g, float p, float m0, float m1, float m2, float v,
                                              float rs, float k0, float k1, float k2) {
  if (FAM == PYLO_FAM_ADAFAC) {
    f[0] = g; f[1] = p; f[2] = m0; f[3] = m1; f[4] = m2; f[5] = v;
    f[6] = m0 * rs; f[7] = m1 * rs; f[8] = m2 * rs; f[9] = rs;
    f[10] = k0 * g; f[11] = k1 * g; f[12] = k2 * g;
    f[25] = k0 * m0; f[26] = k1 * m1; f[27] = k2 * m2;
  } else {
    f[0] = g; f[1] = fminf(fmaxf(g, -0.1f), 0.1f); f[2] = p; f[3] = m0; f[4] = m1; f[5] = m2; f[6] = v;
    f[7] = m0 * rs; f[8] = m1 * rs; f[9] = m2 * rs; f[10] = rs;
    f[11] = k0 * g; f[12] = k1 * g; f[13] = k2 * g; f[14] = g * rs;
    f[27] = k0 * m0; f[28] = k1 * m1; f[29] = k2 * m2;
  }
}

template <int FAM>
__device__ __forceinline__ void vec_features(float* f, float r0, float r1, float r2, float c0, float c1, float c2) {
  using F = Fam<FAM>;
  f[F::R] = r0; f[F::R + 1] = r1; f[F::R + 2] = r2;
  f[F::C] = c0; f[F::C + 1] = c1; f[F::C + 2] = c2;
  f[F::RR] = rsqrtf(r0 + 1e-8f); f[F::RR + 1] = rsqrtf(r1 + 1e-8f); f[F::RR + 2] = rsqrtf(r2 + 1e-8f);
  f[F::RC] = rsqrtf(c0 + 1e-8f); f[F::RC + 1] = rsqrtf(c1 + 1e-8f); f[F::RC + 2] = rsqrtf(c2 + 1e-8f);
}

// ================================================================================================
// global gradient norm
// ================================================================================================
__global__ void __launch_bounds__(NT) k_grad_sumsq(const pylo_gvec* __restrict__ descs,
                                                   const pylo_tile* __restrict__ tiles, int n_tiles,
                                                   float* __restrict__ scratch) {
  pdl_begin();
  __shared__ float s_red[40];
  for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const pylo_tile tl = tiles[t];
    const float* g = descs[tl.tensor].g + tl.start;
    const int cnt = tile_count(tl, descs[tl.tensor].n);
    float acc = 0.f;
    if ((((uintptr_t)g) & 15) == 0) {
      const int c4 = cnt & ~3;
      for (int i = threadIdx.x * 4; i < c4; i += NT * 4) {
        const float4 q = ldg4(g + i);
        acc += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
      }
      for (int i = c4 + threadIdx.x; i < cnt; i += NT) acc += g[i] * g[i];
    } else {
      for (int i = threadIdx.x; i < cnt; i += NT) acc += g[i] * g[i];
    }
    const float tot = block_sum(acc, s_red);
    if (threadIdx.x == 0) scratch[t] = tot;
  }
}

__global__ void __launch_bounds__(1024) k_sum_final(const float* __restrict__ scratch, int n, float* __restrict__ out) {
  pdl_begin();
  __shared__ double s_d[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += (double)scratch[i];
  acc = warp_sum_d(acc);
  if ((threadIdx.x & 31) == 0) s_d[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_d[w];
    out[0] = (float)t;
  }
}

// ================================================================================================
// Phase A: row / column sums of g'^2 + 1e-30
// ================================================================================================
// GENERIC tensors, seen as a matrix of O*X rows of C = M*Y*I (see GenPos).  Two kinds of work item, told apart by pad_:
//   1: column sums: 256 of the Lb columns, one per thread, over the rows of a strip (partials as on the float4 path);
//   0: row sums: a row is M blocks of Y*I consecutive elements, every block has I sums over y.  A group of lanes takes a
//      block and reads it front to back; with I > 1 a lane stays on one i because the group's stride is a multiple of I.
// Both read whole lines.  (One warp per output with lanes along the reduced axis, as it was, read one element per line
// wherever that axis is not the last: 211 us for 5 M parameters of 3x3 convolutions, 302 us for a ViT patch embedding.)
#define GA_LONG 1024      // from this block length on (I <= 32) a CTA, not a warp, takes a block: the loads of a block are a serial chain
__device__ __forceinline__ void rowcol_generic(const pylo_tensor_desc* __restrict__ descs, const pylo_atile it, const pylo_step_params& prm,
                                               float* s_red) {   // s_red: NT floats
  const pylo_tensor_desc& d = descs[it.tensor];
  const float gs = grad_scale_of(d, prm);
  const bool plain = plain_grad(gs, prm);
  auto square = [&](float e) {
    const float g = plain ? e : xform_grad(e, gs, prm.clip_val, prm.nan_to_num);
    return g * g + 1e-30f;
  };
  const int64_t L = (int64_t)d.Y * d.I;
  if (it.pad_ == 1) {
    const int64_t C = d.M * L, b = (int64_t)it.cb * NT + threadIdx.x;
    if (b >= d.Lb) return;
    const int64_t o = d.O == 1 ? 0 : b / C;
    const int x0 = it.strip * d.rb, x1 = min(x0 + d.rb, d.X);
    const float* __restrict__ g = d.g + (o * d.X + x0) * C + (b - o * C);
    float acc = 0.f;
#pragma unroll 8
    for (int x = x0; x < x1; ++x, g += C) acc += square(__ldg(g));
    d.part_b[(int64_t)it.strip * d.Lb + b] = acc;
    return;
  }
  const int64_t blocks = d.La / d.I, b0 = (int64_t)it.strip * it.cb, b1 = min(b0 + it.cb, blocks);
  const int I = d.I;
  const int lane = threadIdx.x & 31;
  if (I <= 32 && L >= GA_LONG) {
    const int S = NT / I * I;   // active threads: a thread stays on one i
    for (int64_t k = b0; k < b1; ++k) {
      const float* __restrict__ g = d.g + k * L;
      float acc = 0.f;
      if (threadIdx.x < S)
#pragma unroll 8
        for (int64_t e = threadIdx.x; e < L; e += S) acc += square(__ldg(g + e));
      if (I == 1) {
        acc = block_sum(acc, s_red);
        if (threadIdx.x == 0) d.sum_a[k] = acc;
      } else {
        __syncthreads();   // the previous block's sums have been read
        s_red[threadIdx.x] = acc;
        __syncthreads();
        if (threadIdx.x < I) {
          for (int q = threadIdx.x + I; q < S; q += I) acc += s_red[q];
          d.sum_a[k * I + threadIdx.x] = acc;
        }
      }
    }
  } else if (I == 1) {
    const int w = L > 16 ? 32 : (L > 8 ? 16 : (L > 4 ? 8 : 4));   // lanes per block
    for (int64_t k = b0 + threadIdx.x / w; k < b1 + NT / w; k += NT / w) {   // whole warps stay in the loop for the shuffles
      float acc = 0.f;
      if (k < b1) {
        const float* __restrict__ g = d.g + k * L;
#pragma unroll 8
        for (int64_t e = lane & (w - 1); e < L; e += w) acc += square(__ldg(g + e));
      }
      for (int o = w >> 1; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, w);
      if ((lane & (w - 1)) == 0 && k < b1) d.sum_a[k] = acc;
      if (k - threadIdx.x / w + NT / w >= b1) break;   // the same for all threads
    }
  } else if (I <= 32) {
    const int S = 32 / I * I;   // active lanes
    for (int64_t k = b0 + (threadIdx.x >> 5); k < b1; k += NWARP) {
      const float* __restrict__ g = d.g + k * L;
      float acc = 0.f;
      if (lane < S)
#pragma unroll 8
        for (int64_t e = lane; e < L; e += S) acc += square(__ldg(g + e));
      float tot = acc;
      for (int q = I; q < S; q += I) tot += __shfl_sync(0xffffffffu, acc, (lane + q) & 31);   // read by lanes < I only
      if (lane < I) d.sum_a[k * I + lane] = tot;
    }
  } else {
    for (int64_t k = b0 + (threadIdx.x >> 5); k < b1; k += NWARP) {
      const float* __restrict__ g = d.g + k * L;
      for (int i = lane; i < I; i += 32) {
        float acc = 0.f;
#pragma unroll 4
        for (int y = 0; y < d.Y; ++y) acc += square(__ldg(g + (int64_t)y * I + i));
        d.sum_a[k * I + i] = acc;
      }
    }
  }
}

// Bound by HBM.  Of the CTA's eight warps, four pairs take every fourth row of the strip and the warps of a pair one half
// (512 columns) of the block each, so that a lane keeps 16 column accumulators (not 32) and has room to request its next
// row before it adds up the present one: the loads of the next row fly during the shuffles of this one's row sum.
// 355 M elements (GPT-2-medium shapes): 417 us before (a warp per row, 32 accumulators, no row ahead).
// Matrices whose rows are not aligned (GENERIC, with part_a) go the same way with single loads (not VEC), a piece's columns 32 apart.
#define RC_GROUPS 4
// MIX: the list may hold convolution weights, and the first n_gitems CTAs take the GENERIC tensors' items, one each: a launch of their own
// took 13 us for the one 64 x 3 x 7 x 7 tensor of a convolutional network, a chain of latencies.  Both cost registers, so this
// variant has three CTAs per SM and large models do without it (with it, spilling, 355 M elements 277 -> 340 us).
template <bool VEC, bool MIX>
__global__ void __launch_bounds__(NT, VEC && !MIX ? 4 : 3) k_rowcol_fast(const pylo_tensor_desc* __restrict__ descs,
                                                       const pylo_atile* __restrict__ atiles, int n_atiles,
                                                       const pylo_atile* __restrict__ gitems, int n_gitems,
                                                       const pylo_step_params prm) {
  pdl_begin();
  __shared__ float s_col[RC_GROUPS][PYLO_A_COLS];
  if (MIX && (int)blockIdx.x < n_gitems) {
    rowcol_generic(descs, gitems[blockIdx.x], prm, s_col[0]);
    return;
  }
  const int cta = MIX ? blockIdx.x - n_gitems : blockIdx.x, ctas = MIX ? gridDim.x - n_gitems : gridDim.x;
  __shared__ float s_row[PYLO_A_ROWS_MAX][2];
  const int lane = threadIdx.x & 31, half = (threadIdx.x >> 5) & 1, grp = threadIdx.x >> 6;
  for (int t = cta; t < n_atiles; t += ctas) {
    const pylo_atile at = atiles[t];
    const pylo_tensor_desc& d = descs[at.tensor];
    const int I = MIX ? d.I : 1;   // a row has a sum per position
    const int X = d.X, Y = d.Y * I, rb = d.rb;
    const int row0 = at.strip * rb;
    const int rows = min(rb, X - row0);
    const int col0 = at.cb * PYLO_A_COLS;
    const float gs = grad_scale_of(d, prm);
    const bool plain = plain_grad(gs, prm);
    const int c0 = half * 512 + (VEC ? lane * 4 : lane);
    const float* base = d.g + (int64_t)row0 * Y + col0 + c0;
    const int left = Y - col0 - c0;   // columns of this lane's pieces that exist: VEC: piece j is there if j * 128 < left, else column k if k * 32 is
    float colacc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) colacc[j] = 0.f;
    const int lanes = 32 / I * I, first = (col0 + half * 512) % I;   // lanes that add up, and the position of the half's first column
    float* const own = &s_col[grp][half * 512];
    float4 cur[4], nxt[4];
    auto load = [&](int r, float4 (&q)[4]) {
      const float* p = base + (int64_t)r * Y;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (VEC) {
          if (j * 128 < left) q[j] = ldg4(p + j * 128);
        } else {
          if (j * 128 < left) q[j].x = __ldg(p + j * 128);
          if (j * 128 + 32 < left) q[j].y = __ldg(p + j * 128 + 32);
          if (j * 128 + 64 < left) q[j].z = __ldg(p + j * 128 + 64);
          if (j * 128 + 96 < left) q[j].w = __ldg(p + j * 128 + 96);
        }
      }
    };
    if (grp < rows) load(grp, cur);
    for (int r = grp; r < rows; r += RC_GROUPS) {
      if (r + RC_GROUPS < rows) load(r + RC_GROUPS, nxt);
      float rowsum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float sq[4] = {0.f, 0.f, 0.f, 0.f};
        if (j * 128 < left) {
          const float e[4] = {cur[j].x, cur[j].y, cur[j].z, cur[j].w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (!VEC && j * 128 + u * 32 >= left) continue;
            const float g = plain ? e[u] : xform_grad(e[u], gs, prm.clip_val, prm.nan_to_num);
            const float q = g * g + 1e-30f;
            colacc[j * 4 + u] += q;
            rowsum += q;
            sq[u] = q;
          }
        }
        if (I > 1) st4(own + lane * 4 + j * 128, make_float4(sq[0], sq[1], sq[2], sq[3]));
      }
      if (I == 1) {
        rowsum = warp_sum(rowsum);
        if (lane == 0) s_row[r][half] = rowsum;
      } else {   // through shared memory, where a lane stays on one position because the lanes' stride is a multiple of I
        __syncwarp();
        float acc = 0.f;
        if (lane < lanes)
#pragma unroll 8
          for (int e = lane; e < 512; e += lanes) acc += own[e];
        float tot = acc;
        for (int q = I; q < lanes; q += I) tot += __shfl_sync(0xffffffffu, acc, (lane + q) & 31);   // read by lanes < I only
        const int i = first + lane < I ? first + lane : first + lane - I;
        if (lane < I) d.part_a[((int64_t)(row0 + r) * I + i) * (2 * d.n_cb) + 2 * at.cb + half] = tot;
        __syncwarp();
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) cur[j] = nxt[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (VEC) st4(&s_col[grp][c0 + j * 128], make_float4(colacc[j * 4], colacc[j * 4 + 1], colacc[j * 4 + 2], colacc[j * 4 + 3]));
      else
#pragma unroll
        for (int u = 0; u < 4; ++u) s_col[grp][c0 + j * 128 + u * 32] = colacc[j * 4 + u];
    }
    __syncthreads();
    if constexpr (VEC) {
      const int c = threadIdx.x * 4;
      if (col0 + c < Y) {
        float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < RC_GROUPS; ++w) {
          const float4 q = ld4(&s_col[w][c]);
          tot.x += q.x; tot.y += q.y; tot.z += q.z; tot.w += q.w;
        }
        st4(d.part_b + (int64_t)at.strip * Y + col0 + c, tot);
      }
    } else {
      for (int c = threadIdx.x; c < PYLO_A_COLS && col0 + c < Y; c += NT) {
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < RC_GROUPS; ++w) tot += s_col[w][c];
        d.part_b[(int64_t)at.strip * Y + col0 + c] = tot;
      }
    }
    if (I == 1 && threadIdx.x < rows) d.part_a[(int64_t)(row0 + threadIdx.x) * d.n_cb + at.cb] = s_row[threadIdx.x][0] + s_row[threadIdx.x][1];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(NT) k_rowcol_generic(const pylo_tensor_desc* __restrict__ descs, const pylo_atile* __restrict__ items,
                                                       const pylo_step_params prm) {
  pdl_begin();
  __shared__ float s_red[NT];
  rowcol_generic(descs, items[blockIdx.x], prm, s_red);
}

// ================================================================================================
// Phase A2: factored accumulators, factors, closed-form vector-feature moments.  One cluster of eight CTAs per tensor.
//
// Latency-bound: a tensor's vectors are a few ten thousand entries, but every column's sum runs over all strips of phase
// A and the factors need the mean of the whole vector.  Eight CTAs share the tensor (one CTA took 185 us for the 50257
// rows of a GPT-2 embedding) and exchange their partial sums through distributed shared memory; every CTA adds the eight
// in rank order, so the result does not depend on timing.  The sum over the strips is part of this kernel: 128 columns
// per pass (512 where there are enough), the strips dealt to eight groups of 128 threads, or to four: a CTA has A2_NT threads, or half
// of them where the model has more clusters than run at once, which then share the SMs two and two, so that one's barriers and
// latencies are another's time.  The number of threads decides the order of the sums; the host takes it from the whole model (sum_order).
// ================================================================================================
#define A2_NT 1024
#define A2_CL 8
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  return n;
}
// all threads of all CTAs of the cluster; orders shared, distributed shared and global memory accesses
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same in two parts that order nothing: after cluster_wait() every CTA of the cluster is known to be running.  Until then
// none may reach into another's shared memory.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_store(float* p, uint32_t rank, float v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(int* p, uint32_t rank, int v) { cluster_store(reinterpret_cast<float*>(p), rank, __int_as_float(v)); }

__device__ __forceinline__ float cluster_load(const float* p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// mats: which tensors (those with fewer than two dims have no factors, and their closed forms stay zero), or NULL for all.
template <int FAM, int THREADS>
__global__ void __cluster_dims__(A2_CL, 1, 1) __launch_bounds__(THREADS, A2_NT / THREADS) k_factor_update(const pylo_tensor_desc* __restrict__ descs,
                                                                                          const int* __restrict__ mats, const pylo_step_params prm) {
  pdl_begin();
  using F = Fam<FAM>;
  constexpr int NS = 15;  // sums per CTA: row accumulator (its mean), then the four closed forms, three decays each
  __shared__ __align__(16) float s_part[THREADS / 128][512];
  __shared__ float s_warp[THREADS / 32][NS];
  __shared__ float s_cta[A2_CL][NS + 1];
  __shared__ float s_tot[NS + 1];
  const pylo_tensor_desc& d = descs[mats ? mats[blockIdx.x / A2_CL] : blockIdx.x / A2_CL];
  const int tid = threadIdx.x, rank = (int)cluster_rank();
  if (d.mode == PYLO_MODE_VEC1D) {  // the same for all CTAs of the cluster
    if (rank == 0 && tid < PYLO_STAT_STRIDE) d.closed[tid] = 0.f;
    return;
  }
  cluster_arrive();   // waited for below, before the first store into another CTA
  const bool blocks = d.part_a != nullptr, r_is_a = d.r_is_a != 0;   // blocks: phase A has left row sums per block of columns
  const int64_t La = d.La, Lb = d.Lb;
  const int parts = d.mode == PYLO_MODE_KERNEL ? 2 * d.n_cb : d.n_cb;
  const float inv_n_a = (float)d.Y, inv_n_b = (float)d.X;
  float acc[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) acc[j] = 0.f;
  auto add = [&](bool is_r, int k, float v) {
    const float q = rsqrtf(v + 1e-8f);
    if (is_r) { acc[k] += v; acc[3 + k] = fmaf(v, v, acc[3 + k]); acc[6 + k] = fmaf(q, q, acc[6 + k]); }
    else { acc[9 + k] = fmaf(v, v, acc[9 + k]); acc[12 + k] = fmaf(q, q, acc[12 + k]); }
  };

  // 1. "a" vectors: finish the row sums, EMA of the accumulator lerp(acc, mean, 1 - beta_fac[k])
  const int gtid = rank * THREADS + tid;
  for (int64_t i = gtid; i < La; i += A2_CL * THREADS) {
    float old[3];  // requested before the partials are added up
#pragma unroll
    for (int k = 0; k < 3; ++k) old[k] = d.fac_a[k * La + i];
    float s;
    if (blocks) {
      s = 0.f;
#pragma unroll 4
      for (int c = 0; c < parts; ++c) s += d.part_a[i * parts + c];
      d.sum_a[i] = s;
    } else {
      s = d.sum_a[i];
    }
    const float mean = s / inv_n_a;
    float f[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = lerp_torch(old[k], mean, prm.w_f[k]);
      d.fac_a[k * La + i] = v;
      add(r_is_a, k, v);
      f[k] = safe_rsqrt(v);
    }
    if (!r_is_a) {  // col_factor = safe_rsqrt(fac_c)
#pragma unroll
      for (int k = 0; k < 3; ++k) d.f_a[k * La + i] = f[k];
      if (d.fx) st4(d.fx + 4 * i, make_float4(f[0], f[1], f[2], 0.f));
    }
  }
  // 2. "b" vectors: sum over the strips (in a fixed order), EMA.  A pass takes 128 columns, or 512 where there are enough of them, its
  // strips dealt to the groups of 128 threads.
  auto columns = [&](auto width) {
    constexpr int V = decltype(width)::value, W = 128 * V;
    for (int64_t c0 = (int64_t)rank * W; c0 < Lb; c0 += A2_CL * W) {
      const int64_t i = c0 + V * (tid & 127);
      float s[V], old[3] = {0.f, 0.f, 0.f};
      if (tid < W && c0 + tid < Lb) {
#pragma unroll
        for (int k = 0; k < 3; ++k) old[k] = d.fac_b[k * Lb + c0 + tid];
      }
#pragma unroll
      for (int u = 0; u < V; ++u) s[u] = 0.f;
      if (i < Lb) {
        const float* __restrict__ src = d.part_b + i;
#pragma unroll 8
        for (int r = tid >> 7; r < d.n_strips; r += THREADS / 128) {
          if constexpr (V == 4) {
            const float4 q = ld4(src + (int64_t)r * Lb);
            s[0] += q.x; s[1] += q.y; s[2] += q.z; s[3] += q.w;
          } else {
            s[0] += src[(int64_t)r * Lb];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < V; ++u) s_part[tid >> 7][V * (tid & 127) + u] = s[u];
      __syncthreads();
      if (tid < W && c0 + tid < Lb) {
        const int64_t j = c0 + tid;
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < THREADS / 128; ++w) tot += s_part[w][tid];
        d.sum_b[j] = tot;
        const float mean = tot / inv_n_b;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float v = lerp_torch(old[k], mean, prm.w_f[k]);
          d.fac_b[k * Lb + j] = v;
          add(!r_is_a, k, v);
          if (r_is_a) d.f_b[k * Lb + j] = safe_rsqrt(v);
        }
      }
      __syncthreads();
    }
  };
  static_assert(THREADS >= 512, "a pass of 512 columns is finished by a thread per column");
  if (Lb % 4 == 0 && Lb > A2_CL * 128) columns(std::integral_constant<int, 4>{});
  else columns(std::integral_constant<int, 1>{});
  // 3. the fifteen sums over the tensor, in every CTA
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const float v = warp_sum(acc[j]);
    if ((tid & 31) == 0) s_warp[tid >> 5][j] = v;
  }
  __syncthreads();
  cluster_wait();
  if (tid < NS) {
    float v = 0.f;
    for (int w = 0; w < THREADS / 32; ++w) v += s_warp[w][tid];
    for (uint32_t q = 0; q < A2_CL; ++q) cluster_store(&s_cta[rank][tid], q, v);
  }
  cluster_sync();  // also: every CTA's accumulators are visible to the others
  if (tid < NS) {
    float v = 0.f;
    for (int q = 0; q < A2_CL; ++q) v += s_cta[q][tid];
    s_tot[tid] = v;
  }
  __syncthreads();

  // 4. row_factor = safe_rsqrt(fac_r / (mean over the reduce axis + 1e-9))
  const float* fac_r = r_is_a ? d.fac_a : d.fac_b;
  float* f_r = r_is_a ? d.f_a : d.f_b;
  const int64_t Lr = r_is_a ? La : Lb;
  const int64_t pre = d.rcm_pre, A = d.rcm_A, post = d.rcm_post;
  auto put = [&](int64_t e, float v) {   // entry e of [3][Lr]
    f_r[e] = v;
    if (d.fx && r_is_a) {
      const int64_t k = e >= 2 * Lr ? 2 : e >= Lr ? 1 : 0;
      d.fx[4 * (e - k * Lr) + k] = v;
    }
  };
  if ((pre == 3 && A == Lr) || (pre == 1 && A == 3 && post == Lr)) {
    // the mean of each decay's whole vector, or (the decay axis is the reduce axis) of each entry's three decays
    const bool whole = pre == 3 && A == Lr;
    for (int64_t i = gtid; i < Lr; i += A2_CL * THREADS) {
      const float v0 = fac_r[i], v1 = fac_r[Lr + i], v2 = fac_r[2 * Lr + i];
      const float own = (v0 + v1 + v2) / 3.0f;
      const float f0 = safe_rsqrt(v0 / ((whole ? s_tot[0] / (float)A : own) + 1e-9f));
      const float f1 = safe_rsqrt(v1 / ((whole ? s_tot[1] / (float)A : own) + 1e-9f));
      const float f2 = safe_rsqrt(v2 / ((whole ? s_tot[2] / (float)A : own) + 1e-9f));
      f_r[i] = f0; f_r[Lr + i] = f1; f_r[2 * Lr + i] = f2;
      if (d.fx && r_is_a) st4(d.fx + 4 * i, make_float4(f0, f1, f2, 0.f));
    }
  } else {   // a warp per mean (a thread per mean, one after the other, took 55 us for VeLO over 3x3 convolutions: 27 means of 512 entries)
    const int lane = tid & 31;
    for (int64_t o = gtid >> 5; o < pre * post; o += A2_CL * THREADS / 32) {
      const int64_t first = o / post * A * post + o % post;
      float m = 0.f;
#pragma unroll 4
      for (int64_t a = lane; a < A; a += 32) m += fac_r[first + a * post];
      m = __shfl_sync(0xffffffffu, warp_sum(m), 0) / (float)A;
      for (int64_t a = lane; a < A; a += 32) {
        const int64_t e = first + a * post;
        put(e, safe_rsqrt(fac_r[e] / (m + 1e-9f)));
      }
    }
  }
  // 5. closed-form sums of squares of the features that depend on one vector only: every vector entry is seen by
  //    n / L elements of the tensor
  if (rank == 0 && tid < PYLO_STAT_STRIDE) {
    const float mult_r = (float)(d.n / Lr), mult_c = (float)(d.n / (r_is_a ? Lb : La));
    float v = 0.f;
    if (tid >= F::R && tid < F::R + 3) v = s_tot[3 + tid - F::R] * mult_r;
    else if (tid >= F::RR && tid < F::RR + 3) v = s_tot[6 + tid - F::RR] * mult_r;
    else if (tid >= F::C && tid < F::C + 3) v = s_tot[9 + tid - F::C] * mult_c;
    else if (tid >= F::RC && tid < F::RC + 3) v = s_tot[12 + tid - F::RC] * mult_c;
    d.closed[tid] = v;
  }
}

// ================================================================================================
// Phase B: state update + per-tile sums of squares of the element-wise features
// ================================================================================================
template <int FAM>
struct BAcc {
  static constexpr int N = Fam<FAM>::NF + (FAM == PYLO_FAM_VELO ? 8 : 0);
};

template <int FAM, bool VECF>
__device__ __forceinline__ void accumulate(float (&acc)[BAcc<FAM>::N], const float* f) {
#pragma unroll
  for (int j = 0; j < Fam<FAM>::NF; ++j) {
    if (!VECF && is_vec_feature<FAM>(j)) continue;
    acc[j] = fmaf(f[j], f[j], acc[j]);
  }
}

template <int FAM>
__device__ __forceinline__ void velo_stats(float (&acc)[BAcc<FAM>::N], float m0, float m1, float m2, float v) {
  if (FAM == PYLO_FAM_VELO) {
    constexpr int B = Fam<FAM>::NF;
    acc[B + 0] += m0; acc[B + 1] += m1; acc[B + 2] += m2;
    acc[B + 3] = fmaf(m0, m0, acc[B + 3]); acc[B + 4] = fmaf(m1, m1, acc[B + 4]); acc[B + 5] = fmaf(m2, m2, acc[B + 5]);
    acc[B + 6] += v; acc[B + 7] = fmaf(v, v, acc[B + 7]);
  }
}

// Vectors: full-size accumulators updated element-wise (AdafacLO_cuda.py:349-360, velo_cuda.py:543-546).
template <int FAM, int THREADS>
__device__ __forceinline__ void vec1d_update(const pylo_tensor_desc& d, const pylo_step_params& prm, float gs, int64_t start, int cnt,
                                             float (&acc)[BAcc<FAM>::N]) {
  const int64_t n = d.n;
  const float *gp = d.g + start, *pp = d.p + start;
  float *m0p = d.m + start, *m1p = m0p + d.m_stride, *m2p = m1p + d.m_stride, *vp = d.v + start;
  float* ra = d.fac_a + start;
  float* rb = d.fac_b ? d.fac_b + start : nullptr;
  for (int i = threadIdx.x; i < cnt; i += THREADS) {
    const float g = xform_grad(gp[i], gs, prm.clip_val, prm.nan_to_num);
    float m0 = m0p[i], m1 = m1p[i], m2 = m2p[i], v = vp[i];
    velo_stats<FAM>(acc, m0, m1, m2, v);
    m0 = lerp_torch(m0, g, prm.w_m[0]);
    m1 = lerp_torch(m1, g, prm.w_m[1]);
    m2 = lerp_torch(m2, g, prm.w_m[2]);
    v = lerp_torch(v, g * g + prm.eps_v, prm.w_v);
    m0p[i] = m0; m1p[i] = m1; m2p[i] = m2; vp[i] = v;
    const float gsq = g * g + 1e-30f;
    float r[3], c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      r[k] = lerp_torch(ra[k * n + i], gsq, prm.w_f[k]);
      ra[k * n + i] = r[k];
      if (rb) { c[k] = lerp_torch(rb[k * n + i], gsq, prm.w_f[k]); rb[k * n + i] = c[k]; }
      else c[k] = r[k];
    }
    const float rs = rsqrtf(v + prm.eps_feat);
    float f[Fam<FAM>::NF];
    elem_features<FAM>(f, g, pp[i], m0, m1, m2, v, rs, safe_rsqrt(r[0] + 1e-9f), safe_rsqrt(r[1] + 1e-9f),
                       safe_rsqrt(r[2] + 1e-9f));
    vec_features<FAM>(f, r[0], r[1], r[2], c[0], c[1], c[2]);
    accumulate<FAM, true>(acc, f);
  }
}

// Bound by HBM on large models.  With RING, FAST2D tiles come through the ring of pylo_pipe.cuh: the copies run ahead over tile
// borders, so that neither the next loads nor the block reduction at a tile's end leave the memory idle.  Everything else is
// read into registers; without RING all tiles are, and the memory that the ring would take is the L1 cache in which the
// factor vectors of strided tensors are found.
template <int FAM, bool RING>
__global__ void __launch_bounds__(NT, 2) k_state_moments(const pylo_tensor_desc* __restrict__ descs,
                                                      const pylo_tile* __restrict__ tiles, int n_tiles, int reverse,
                                                      const pylo_step_params prm) {
  using F = Fam<FAM>;
  constexpr int NACC = BAcc<FAM>::N;
  extern __shared__ __align__(128) unsigned char pipe_raw[];
  PipeSmem& pipe = *reinterpret_cast<PipeSmem*>(pipe_raw);   // RING only
  __shared__ float s_red[NWARP * NACC];
  const int tid = threadIdx.x;
  if constexpr (RING) pipe_init(pipe);
  pdl_begin();
  uint32_t k = 0;   // stages consumed
  // the first warp's cursor, PIPE_STAGES - 1 stages ahead of the consumers: lane u < 6 copies stream u
  int ptt = blockIdx.x - gridDim.x, pc = 0, pcnt = 0;
  uint32_t pk = 0;
  const float* psrc = nullptr;
  auto produce = [&]() -> bool {
    while (pc >= pcnt) {   // on to the next FAST2D tile
      ptt += gridDim.x;
      if (ptt >= n_tiles) { ptt = n_tiles; return true; }
      const pylo_tile tl = tiles[reverse ? (n_tiles - 1 - ptt) : ptt];
      const pylo_tensor_desc& d = descs[tl.tensor];
      if (d.mode != PYLO_MODE_FAST2D) continue;
      pc = 0;
      pcnt = tile_count(tl, d.n);
      psrc = (tid == 0 ? d.g : tid == 1 ? d.p : tid == 5 ? d.v : d.m + (tid - 2) * d.m_stride) + tl.start;
    }
    const uint32_t bytes = 4u * min(PIPE_ELEMS, pcnt - pc);
    if (!pipe_begin(pipe, pk, PIPE_STREAMS * bytes)) return false;
    if (tid < PIPE_STREAMS) pipe_copy(pipe, pk, tid, 0, psrc + pc, bytes);
    pc += PIPE_ELEMS;
    ++pk;
    return true;
  };
  if (RING && tid < 32) {
    asm volatile("fence.proxy.async;" ::: "memory");   // what earlier kernels stored is read through the async proxy
    for (int s = 0; s < PIPE_STAGES - 1; ++s) produce();
  }
  bool dead = false;
  for (int tt = blockIdx.x; tt < n_tiles && !dead; tt += gridDim.x) {
    const int t = reverse ? (n_tiles - 1 - tt) : tt;
    const pylo_tile tl = tiles[t];
    const pylo_tensor_desc& d = descs[tl.tensor];
    const int64_t n = d.n, start = tl.start;
    const int cnt = tile_count(tl, n);
    const float gs = grad_scale_of(d, prm);
    const bool plain = plain_grad(gs, prm);
    float acc[NACC];
#pragma unroll
    for (int j = 0; j < NACC; ++j) acc[j] = 0.f;
    float* m0p = d.m + start;
    float* m1p = d.m + d.m_stride + start;
    float* m2p = d.m + 2 * d.m_stride + start;
    float* vp = d.v + start;
    const float* gp = d.g + start;
    const float* pp = d.p + start;

    if (d.mode == PYLO_MODE_FAST2D || (!RING && d.mode == PYLO_MODE_KERNEL)) {
      const uint32_t Y = RING ? d.Y : d.Y * d.I;
      // this thread's row and column (n < 2^31 here), moved on by a stage's length
      const uint32_t first = (uint32_t)start + tid * 4;
      uint32_t x = first / Y, y = first - x * Y;
      const uint32_t dx = PIPE_ELEMS / Y, dy = PIPE_ELEMS - dx * Y;
      const float* __restrict__ fxp = d.fx;
      const float* __restrict__ fbp = d.f_b;
      auto update4 = [&](int i, float4 g4, float4 p4, float4 a0, float4 a1, float4 a2, float4 v4, auto row, float4 b0, float4 b1, float4 b2) {
        float ge[4] = {g4.x, g4.y, g4.z, g4.w}, pe[4] = {p4.x, p4.y, p4.z, p4.w};
        float m0e[4] = {a0.x, a0.y, a0.z, a0.w}, m1e[4] = {a1.x, a1.y, a1.z, a1.w}, m2e[4] = {a2.x, a2.y, a2.z, a2.w};
        float ve[4] = {v4.x, v4.y, v4.z, v4.w};
        const float b0e[4] = {b0.x, b0.y, b0.z, b0.w}, b1e[4] = {b1.x, b1.y, b1.z, b1.w}, b2e[4] = {b2.x, b2.y, b2.z, b2.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float g = plain ? ge[u] : xform_grad(ge[u], gs, prm.clip_val, prm.nan_to_num);
          velo_stats<FAM>(acc, m0e[u], m1e[u], m2e[u], ve[u]);
          m0e[u] = lerp_torch(m0e[u], g, prm.w_m[0]);
          m1e[u] = lerp_torch(m1e[u], g, prm.w_m[1]);
          m2e[u] = lerp_torch(m2e[u], g, prm.w_m[2]);
          ve[u] = lerp_torch(ve[u], g * g + prm.eps_v, prm.w_v);
          const float rs = rsqrtf(ve[u] + prm.eps_feat);
          float f[F::NF];
          const float4 fa = row(u);
          elem_features<FAM>(f, g, pe[u], m0e[u], m1e[u], m2e[u], ve[u], rs, fa.x * b0e[u], fa.y * b1e[u], fa.z * b2e[u]);
          accumulate<FAM, false>(acc, f);
        }
        st4(m0p + i, make_float4(m0e[0], m0e[1], m0e[2], m0e[3]));
        st4(m1p + i, make_float4(m1e[0], m1e[1], m1e[2], m1e[3]));
        st4(m2p + i, make_float4(m2e[0], m2e[1], m2e[2], m2e[3]));
        st4(vp + i, make_float4(ve[0], ve[1], ve[2], ve[3]));
      };
      if (!RING && d.mode == PYLO_MODE_KERNEL) {   // the four columns are four positions in turn, each with row factors of its own
        const uint32_t I = d.I;
        uint32_t pos = y % I;
        const uint32_t dpos = dy % I;   // Y is a multiple of I
        for (int i = tid * 4; i < cnt; i += PIPE_ELEMS) {
          float4 fa[4];
#pragma unroll
          for (uint32_t u = 0; u < 4; ++u) {
            uint32_t q = pos + u;
            while (q >= I) q -= I;
            fa[u] = ld4(fxp + 4 * ((int64_t)x * I + q));
          }
          update4(i, ldg4(gp + i), ld4(pp + i), ld4(m0p + i), ld4(m1p + i), ld4(m2p + i), ld4(vp + i), [&](int u) { return fa[u]; }, ld4(fbp + y),
                  ld4(fbp + Y + y), ld4(fbp + 2 * (int64_t)Y + y));
          x += dx; y += dy; pos += dpos;
          if (y >= Y) { y -= Y; ++x; }
          if (pos >= I) pos -= I;
        }
      } else
      for (int i = tid * 4; i - tid * 4 < cnt; i += PIPE_ELEMS) {
        const bool ok = i < cnt;
        float4 fa = make_float4(0.f, 0.f, 0.f, 0.f), b0 = fa, b1 = fa, b2 = fa;
        if (ok) {
          fa = ld4(fxp + 4 * (int64_t)x);
          b0 = ld4(fbp + y); b1 = ld4(fbp + Y + y); b2 = ld4(fbp + 2 * (int64_t)Y + y);
        }
        x += dx; y += dy;
        if (y >= Y) { y -= Y; ++x; }
        if constexpr (RING) {
          if (tid < 32 && !produce()) { dead = true; break; }
          if (!pipe_wait_full(pipe, k)) { dead = true; break; }
          const float(*st)[PIPE_ELEMS] = pipe.st[k % PIPE_STAGES];
          if (ok) update4(i, ld4(&st[0][tid * 4]), ld4(&st[1][tid * 4]), ld4(&st[2][tid * 4]), ld4(&st[3][tid * 4]), ld4(&st[4][tid * 4]),
                          ld4(&st[5][tid * 4]), [&](int) { return fa; }, b0, b1, b2);
          pipe_release(pipe, k++);
        } else if (ok) {
          update4(i, ldg4(gp + i), ld4(pp + i), ld4(m0p + i), ld4(m1p + i), ld4(m2p + i), ld4(vp + i), [&](int) { return fa; }, b0, b1, b2);
        }
      }
    } else if (d.mode == PYLO_MODE_GENERIC || (RING && d.mode == PYLO_MODE_KERNEL)) {
      const int64_t La = d.La, Lb = d.Lb;
      const bool vecf = d.vec_elementwise != 0;
      GenPos pos(d, d.idx0 + start + tid, NT);
      constexpr int U = 4;   // elements of a thread in flight; their factors, from L1, are fetched when they are needed
      auto update = [&](float g, float& m0, float& m1, float& m2, float& v) {
        velo_stats<FAM>(acc, m0, m1, m2, v);
        m0 = lerp_torch(m0, g, prm.w_m[0]);
        m1 = lerp_torch(m1, g, prm.w_m[1]);
        m2 = lerp_torch(m2, g, prm.w_m[2]);
        v = lerp_torch(v, g * g + prm.eps_v, prm.w_v);
      };
      if (!vecf) {
        for (int i0 = tid; i0 < cnt; i0 += U * NT) {
          float g[U], p[U], m0[U], m1[U], m2[U], v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + u * NT;
            if (i < cnt) { g[u] = __ldg(gp + i); p[u] = pp[i]; m0[u] = m0p[i]; m1[u] = m1p[i]; m2[u] = m2p[i]; v[u] = vp[i]; }
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + u * NT;
            if (i < cnt) {
              const int64_t a = pos.a(), b = pos.b();
              const float k0 = __ldg(d.f_a + a) * __ldg(d.f_b + b), k1 = __ldg(d.f_a + La + a) * __ldg(d.f_b + Lb + b),
                          k2 = __ldg(d.f_a + 2 * La + a) * __ldg(d.f_b + 2 * Lb + b);
              const float gx = xform_grad(g[u], gs, prm.clip_val, prm.nan_to_num);
              update(gx, m0[u], m1[u], m2[u], v[u]);
              m0p[i] = m0[u]; m1p[i] = m1[u]; m2p[i] = m2[u]; vp[i] = v[u];
              float f[F::NF];
              elem_features<FAM>(f, gx, p[u], m0[u], m1[u], m2[u], v[u], rsqrtf(v[u] + prm.eps_feat), k0, k1, k2);
              accumulate<FAM, false>(acc, f);
            }
            pos.next();
          }
        }
      } else {
        const float* fac_r = d.r_is_a ? d.fac_a : d.fac_b;
        const float* fac_c = d.r_is_a ? d.fac_b : d.fac_a;
        for (int i = tid; i < cnt; i += NT, pos.next()) {
          const int64_t a = pos.a(), b = pos.b();
          const float g = xform_grad(gp[i], gs, prm.clip_val, prm.nan_to_num);
          float m0 = m0p[i], m1 = m1p[i], m2 = m2p[i], v = vp[i];
          update(g, m0, m1, m2, v);
          m0p[i] = m0; m1p[i] = m1; m2p[i] = m2; vp[i] = v;
          float f[F::NF];
          elem_features<FAM>(f, g, pp[i], m0, m1, m2, v, rsqrtf(v + prm.eps_feat), d.f_a[a] * d.f_b[b], d.f_a[La + a] * d.f_b[Lb + b],
                             d.f_a[2 * La + a] * d.f_b[2 * Lb + b]);
          const int64_t ir = d.r_is_a ? a : b, ic = d.r_is_a ? b : a;
          const int64_t Lr = d.r_is_a ? La : Lb, Lc = d.r_is_a ? Lb : La;
          vec_features<FAM>(f, fac_r[ir], fac_r[Lr + ir], fac_r[2 * Lr + ir], fac_c[ic], fac_c[Lc + ic], fac_c[2 * Lc + ic]);
          accumulate<FAM, true>(acc, f);
        }
      }
    } else {
      vec1d_update<FAM, NT>(d, prm, gs, start, cnt, acc);
    }
    float* out = d.tile_part + (int64_t)(t - d.tile0) * PYLO_STAT_STRIDE;
    block_reduce_store<NACC>(acc, s_red, out);
    if (tid >= NACC && tid < PYLO_STAT_STRIDE) out[tid] = 0.f;
    if constexpr (RING) dead = __syncthreads_or(dead);   // a warp whose wait ran out takes the whole CTA with it: the barriers above are everyone's
  }
  if constexpr (RING) {
    if (dead && (tid & 31) == 0) pipe_failed(prm);
    if (dead && tid < 32) pipe_drain(pipe, pk);
  }
}

// ================================================================================================
// Phase B2: per-tensor fixed-order reduction of the tile partials
// ================================================================================================
// A unit's sums from its tiles' partials, in a fixed order; valid in threads j < PYLO_STAT_STRIDE, which hold sum j.
// Latency-bound: a 58 M-element tensor leaves 3584 rows of 40 partials.  The rows are read as one stretch of memory, ROWS at
// a time, every thread keeping its column; eight rows ahead are in flight.
template <int ROWS>
__device__ __forceinline__ double unit_sum(const pylo_tensor_desc& d, double (&s_d)[ROWS][PYLO_STAT_STRIDE]) {
  const int j = threadIdx.x % PYLO_STAT_STRIDE, sub = threadIdx.x / PYLO_STAT_STRIDE;
  if (sub < ROWS) {
    double acc = 0.0;
    const float* __restrict__ src = d.tile_part + j;
    const int n = d.n_tiles;
#pragma unroll 8
    for (int t = sub; t < n; t += ROWS) acc += (double)src[(int64_t)t * PYLO_STAT_STRIDE];
    s_d[sub][j] = acc;
  }
  __syncthreads();
  double tot = 0.0;
  if (threadIdx.x < PYLO_STAT_STRIDE) {
    for (int q = 0; q < ROWS; ++q) tot += s_d[q][j];
    tot += (double)d.closed[j];
  }
  return tot;
}
__device__ __forceinline__ void store_unit_sum(const pylo_tensor_desc& d, double tot, int j = threadIdx.x) {
  const float hi = (float)tot;
  d.sums[j] = hi;
  if (j >= 30 && j < 38) d.sums[SUMS_LO + (j - 30)] = (float)(tot - (double)hi);
}
template <int ROWS>
__global__ void __launch_bounds__(ROWS * PYLO_STAT_STRIDE) k_finalize_moments(const pylo_tensor_desc* __restrict__ descs) {
  pdl_begin();
  __shared__ double s_d[ROWS][PYLO_STAT_STRIDE];
  const pylo_tensor_desc& d = descs[blockIdx.x];
  const double tot = unit_sum<ROWS>(d, s_d);
  if (threadIdx.x < PYLO_STAT_STRIDE) store_unit_sum(d, tot);
}

// ================================================================================================
// Phase P: fold normalisers (and time features) into the first layer; tabulate vector-feature terms
// ================================================================================================
template <int FAM>
__device__ __forceinline__ float w1_at(const float* w, int j, int k) {
  // first-layer weight for hidden unit j and input k in the family's own storage order
  if (FAM == PYLO_FAM_ADAFAC) return w[j * 39 + k];
  if (FAM == PYLO_FAM_CELO2) return w[k * 8 + j];
  return w[j * 30 + k];
}

// One work item is PREP_TABLE / H rows of a unit's "a" or "b" table (the "a" items first); item 0 of a unit also writes
// the folded network.  Items are dealt by the tables' sizes, so that a 50257-row table is spread over the GPU (a fixed
// number of CTAs per unit took 537 us for it).
// Latency-bound: an item's work is a few thousand operations, so everything it reads (the network, its entries' accumulators,
// the tile partials) is asked for at once, the first two as asynchronous copies into shared memory.  Read where it was used, each
// loop waited for its own loads: 7.5 us, now 5.2, for AdafacLO on a perceptron of 118 K parameters.
#define PREP_TABLE 2048
template <int FAM>
__global__ void __launch_bounds__(NT) k_prep_apply(const pylo_tensor_desc* __restrict__ descs,
                                                   const pylo_atile* __restrict__ items, const pylo_step_params prm) {
  pdl_begin();
  using F = Fam<FAM>;
  using L = Fold<FAM>;
  constexpr int H = F::H, NF = F::NF, NIN = F::NIN, PER = PREP_TABLE / H;
  // source offsets in the family layout
  constexpr int o_b1 = NIN * H, o_w2 = o_b1 + H, o_b2 = o_w2 + H * H, o_w3 = o_b2 + H, o_b3 = o_w3 + H * F::NOUT, o_end = o_b3 + F::NOUT;
  __shared__ float s_scale[NF];
  __shared__ double s_d[6][PYLO_STAT_STRIDE];
  __shared__ float s_net[o_end];
  __shared__ float s_fac[3][PER];
  __shared__ float s_w1[NF * H];
  __shared__ float s_b1[H];
  __shared__ float s_p2;
  const pylo_atile it = items[blockIdx.x];
  const pylo_tensor_desc& d = descs[it.tensor];
  const int tid = threadIdx.x;
  const float* const w = s_net;
  auto copy = [](float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  };
  for (int e = tid; e < o_end; e += NT) copy(s_net + e, d.w + e);
  // the table entries of this item: of the "a" or of the "b" index
  const int La = d.X, Lb = d.Y, items_a = (La + PER - 1) / PER;
  const bool tables = d.h_a && prm.no_tables != 1, of_a = it.strip < items_a;
  const int i0 = (of_a ? it.strip : it.strip - items_a) * PER, end = tables ? min(of_a ? La : Lb, i0 + PER) : 0;
  for (int e = tid; e < 3 * PER; e += NT) {
    const int k = e / PER, i = i0 + e % PER;
    if (i < end) copy(&s_fac[k][i - i0], (of_a ? d.fac_a + (int64_t)k * La : d.fac_b + (int64_t)k * Lb) + i);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (prm.sum_tiles) {   // small models: no finalize launch, every item adds its unit's few partials up itself
    const double tot = unit_sum<6>(d, s_d);
    if (tid < NF) s_scale[tid] = rsqrtf((float)tot / (float)d.n + prm.eps_norm);
    if (tid == 2) s_p2 = (float)tot;
    if (it.strip == 0 && tid < PYLO_STAT_STRIDE) store_unit_sum(d, tot);
  } else {
    if (tid < NF) s_scale[tid] = rsqrtf(d.sums[tid] / (float)d.n + prm.eps_norm);
    if (tid == 2) s_p2 = d.sums[2];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int e = tid; e < NF * H; e += NT) {
    const int k = e / H, j = e % H;
    s_w1[e] = w1_at<FAM>(w, j, k) * s_scale[k];
  }
  if (tid < H) {
    float b = w[o_b1 + tid];
    if (FAM == PYLO_FAM_ADAFAC) {
      const float tau[11] = {1.f, 3.f, 10.f, 30.f, 100.f, 300.f, 1000.f, 3000.f, 10000.f, 30000.f, 100000.f};
      const float step = d.step + prm.step_delta;
#pragma unroll
      for (int t = 0; t < 11; ++t) b = fmaf(w1_at<FAM>(w, tid, 28 + t), tanhf(step / tau[t] - 1.0f), b);
    }
    s_b1[tid] = b;
  }
  __syncthreads();
  if (it.strip == 0) {
    float* const o = d.wfold;
    for (int e = tid; e < NF * H; e += NT) o[L::W1 + e] = s_w1[e];
    if (tid < NF) o[L::SN + tid] = s_scale[tid];
    if (tid < H) o[L::B1 + tid] = s_b1[tid];
    for (int e = tid; e < H * H; e += NT) {
      const int k = e / H, j = e % H;
      o[L::W2 + e] = (FAM == PYLO_FAM_CELO2) ? w[o_w2 + k * H + j] : w[o_w2 + j * H + k];
    }
    if (tid < H) o[L::B2 + tid] = w[o_b2 + tid];
    for (int e = tid; e < H * 2; e += NT) {
      const int k = e / 2, q = e % 2;
      o[L::W3 + e] = (FAM == PYLO_FAM_CELO2) ? w[o_w3 + k * F::NOUT + q] : w[o_w3 + q * H + k];
    }
    if (tid < 2) o[L::B3 + tid] = w[o_b3 + tid];
    for (int e = tid; e < H * 2; e += NT) {  // pair-major copy of the output layer
      const int jp = e / 4, r = e % 4, k = 2 * jp + (r & 1), q = r >> 1;
      o[L::W3P + e] = (FAM == PYLO_FAM_CELO2) ? w[o_w3 + k * F::NOUT + q] : w[o_w3 + q * H + k];
    }
    if (tid == 0) {
      // VeLO: param_scale = sqrt(mean(p^2) + 1e-9) from the p feature's sum (velo_kernel.cu:297)
      o[L::SC + 0] = (FAM == PYLO_FAM_VELO) ? sqrtf(s_p2 / (float)d.n + 1e-9f) : 1.0f;
      o[L::SC + 1] = d.lr_mult ? d.lr * d.lr_mult[0] : d.lr;
    }
  }
  // first-layer contribution of the features that depend only on the "a" index (plus bias) / "b" index
  const int kr = of_a == (d.r_is_a != 0) ? F::R : F::C, krr = of_a == (d.r_is_a != 0) ? F::RR : F::RC;
  if (of_a) {
    const int j = tid % H;
    float w1[3], w2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) { w1[k] = s_w1[(kr + k) * H + j]; w2[k] = s_w1[(krr + k) * H + j]; }
#pragma unroll 4
    for (int i = i0 + tid / H; i < end; i += NT / H) {
      float acc = s_b1[j];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float r = s_fac[k][i - i0];
        acc = fmaf(w1[k], r, acc);
        acc = fmaf(w2[k], rsqrtf(r + 1e-8f), acc);
      }
      const int64_t e = (int64_t)i * H + j;
      if (FAM == PYLO_FAM_ADAFAC) d.h_a[e] = acc;
      else { d.h_a[2 * e] = acc; d.h_a[2 * e + 1] = acc; }  // stored as (v, v) pairs for the packed kernel
    }
    return;
  }
  for (int e = tid; e < PER * H; e += NT) {  // stored transposed, [H][Y]: a thread of the apply sweep reads its columns' terms with one float4
    const int i = i0 + e % PER, jj = e / PER;
    if (i >= end) continue;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float r = s_fac[k][i - i0];
      acc = fmaf(s_w1[(kr + k) * H + jj], r, acc);
      acc = fmaf(s_w1[(krr + k) * H + jj], rsqrtf(r + 1e-8f), acc);
    }
    d.h_b[(int64_t)jj * Lb + i] = acc;
  }
}

// What the tensor-core sweep reads of a unit (TcImage): the network as operands B, the features' normalisers as scales of operand A.
// One CTA per unit; latency-bound like the kernel above.
//
// Operands are two fp16 planes, so every operand gets a power of two that keeps it inside fp16's range whatever the gradients are.
// A feature over its root mean square is at most sqrt(n) (all of the tensor's sum of squares in one element), so 2^q sqrt(n) <= 2^15;
// a hidden unit's first-layer sum is at most its weights' magnitudes times sqrt(n), plus the bias, so 2^e1 times that is <= 2^15, with
// an e1 for every unit, which its column of the second layer undoes; and weights are
// taken as large as they go, up to 2^a = 2^(e1 + TC_SHIFT - q): the shift between is undone by the tensor core, which scales the
// sums by 2^-TC_SHIFT as it adds the bias.  What a network's units are scaled by (by s, and their columns by 1 / s) therefore changes
// nothing: with one e1 for all units, the largest one's, half of the units times 1e-4 were off by 5e-6 to 5e-5 of the sum of the terms'
// magnitudes at 16 M elements, now 5e-9 to 2e-8 (restated on the CPU, normal and heavy-tailed features).  A plane's last bit is 2^-25 of the scaled unit: of a feature 2^-(25 + q) of its root mean square
// (q = 6 up to 65 K elements, 2 at 16 M, 0 at 268 M), of a unit's activation 2^-(25 + e1), i.e. 2^-39 or less of its largest possible one.
#define TC_SHIFT 10
#define TC_SUM_ROWS 4   // of unit_sum, for what k_small_front leaves (up to 16 tiles): as the sweep's warpgroups do it where they add the partials up
// where a unit's column has features of its own for all rows (FAST2D, KERNEL), those come first
__device__ __forceinline__ bool tc_swap(const pylo_tensor_desc& d) { return (d.mode == PYLO_MODE_FAST2D || d.mode == PYLO_MODE_KERNEL) && d.r_is_a; }
__constant__ float TIME_SCALES[11] = {1.f, 3.f, 10.f, 30.f, 100.f, 300.f, 1000.f, 3000.f, 10000.f, 30000.f, 100000.f};
__device__ __forceinline__ int tc_room(float x) {   // the largest e (up to 60) for which x 2^e is known to be below 2^15
  return x > 0.f ? max(-60, min(60, 141 - (int)((__float_as_uint(x) >> 23) & 255))) : 60;
}
__device__ __forceinline__ float tc_pow2(int e) { return __uint_as_float((uint32_t)(127 + max(-126, min(127, e))) << 23); }
__device__ __forceinline__ uint32_t tc_plane(float x, float scale, float& rest) {   // fp16 of x; rest: what it leaves, scaled
  const __half h = __float2half_rn(x);
  rest = (x - __half2float(h)) * scale;
  return __half_as_ushort(h);
}
// The network's part of a unit's TcImage, and in sn[28] and [29] what undoes the scale of the second layer's sums and that of the features.  Called
// by all of a CTA's THREADS threads with room for TcNet in shared memory; the network is asked for by the caller (tc_ask_network).
struct TcNet {
  static constexpr int H = 32, NIN = 39, o_b1 = NIN * H, o_w2 = o_b1 + H, o_b2 = o_w2 + H * H, o_w3 = o_b2 + H, o_b3 = o_w3 + 2 * H, o_end = o_b3 + 2;
  float net[o_end + H];   // the second layer's rows are H + 1 apart, so that lanes on different rows do not collide
  float b1[H], row[H], column[H], pow[3];   // first layer's bias (scaled), scales of its rows and of the second layer's columns; see below
  float part[4][NT / 32][32];
  __host__ __device__ static constexpr int at(int e) { return e < o_w2 ? e : e < o_b2 ? e + (e - o_w2) / H : e + H; }
};
template <int THREADS>
__device__ __forceinline__ void tc_ask_network(const pylo_tensor_desc& d, TcNet& s) {
  for (int e = threadIdx.x; e < TcNet::o_end; e += THREADS)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(s.net + TcNet::at(e))), "l"(d.w + e) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int THREADS>
__device__ __forceinline__ void tc_network(const pylo_tensor_desc& d, const pylo_step_params& prm, TcNet& s) {
  using L = Fold<PYLO_FAM_ADAFAC>;
  using N = TcNet;
  constexpr int H = N::H, NF = Fam<PYLO_FAM_ADAFAC>::NF, PARTS = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (part < PARTS) {  // a hidden unit per lane, its inputs dealt to eight warps
    const float step = d.step + prm.step_delta;
    float sum = 0.f, most = 0.f, most2 = 0.f, time = 0.f;
    for (int k = part; k < NF; k += PARTS) {
      const float a = fabsf(s.net[lane * N::NIN + k]);
      sum += a;
      most = fmaxf(most, a);
    }
    for (int t = part; t < 11; t += PARTS) time = fmaf(s.net[lane * N::NIN + NF + t], tanhf(step / TIME_SCALES[t] - 1.0f), time);
    for (int k = part; k < H; k += PARTS) most2 = fmaxf(most2, fabsf(s.net[N::o_w2 + k * (H + 1) + lane]));   // of the unit's column
    s.part[0][part][lane] = sum; s.part[1][part][lane] = most; s.part[2][part][lane] = most2; s.part[3][part][lane] = time;
  }
  __syncthreads();
  if (part == 0) {
    float sum = 0.f, most = 0.f, most2 = 0.f, b1 = s.net[N::o_b1 + lane];
    for (int q = 0; q < PARTS; ++q) {
      sum += s.part[0][q][lane];
      most = fmaxf(most, s.part[1][q][lane]);
      most2 = fmaxf(most2, s.part[2][q][lane]);
      b1 += s.part[3][q][lane];
    }
    const float spread = sqrtf((float)d.n) * 1.001f, bound = fmaf(sum, spread, fabsf(b1));
    const int q = min(6, tc_room(spread));
    const int a = min(tc_room(bound) + TC_SHIFT - q, tc_room(most)), e1 = a + q - TC_SHIFT;
    // second-layer sums times 2^a2: as large as every column's weights, which get 2^(a2 - e1), and the biases allow
    int a2 = min(tc_room(most2) - 1 + e1, tc_room(fabsf(s.net[N::at(N::o_b2 + lane)])) + TC_SHIFT);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a2 = min(a2, __shfl_xor_sync(0xffffffffu, a2, o));
    s.b1[lane] = b1 * tc_pow2(e1); s.row[lane] = tc_pow2(a); s.column[lane] = tc_pow2(a2 - e1);
    if (lane == 0) { s.pow[0] = tc_pow2(q); s.pow[1] = tc_pow2(a2 - TC_SHIFT); s.pow[2] = tc_pow2(TC_SHIFT - a2); }
  }
  __syncthreads();
  TcImage& o = *reinterpret_cast<TcImage*>(d.wfold + TC_IMAGE);
  const bool swap = tc_swap(d);
  if (tid < 256) {  // both layers: a thread makes eight weights of one hidden unit, 16 bytes of each plane
    const int layer = tid >> 7, kc = part & 3;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      uint32_t h[2], l[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = kc * 8 + i + u;
        const float x = layer ? s.net[N::o_w2 + lane * (H + 1) + k] : k < NF ? s.net[lane * N::NIN + tc_slot_feature(k, swap)] : 0.f;
        float rest, none;
        h[u] = tc_plane(x * (layer ? s.column[k] : s.row[lane]), 1.f, rest);
        l[u] = tc_plane(rest, 0.f, none);
      }
      hi[i / 2] = h[0] | h[1] << 16;
      lo[i / 2] = l[0] | l[1] << 16;
    }
    char* b = reinterpret_cast<char*>(layer ? o.b2 : o.b1) + kc * 1024 + (lane >> 3) * 128 + (lane & 7) * 16;
    *reinterpret_cast<uint4*>(b) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(b + 512) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  if (part < 4) {
    const int layer = part >> 1, kc = part & 1;
    float rest, none;
    uint32_t word = tc_plane(layer ? s.net[N::at(N::o_b2 + lane)] * s.pow[1] : s.b1[lane], 2048.f, rest);
    word |= tc_plane(rest, 0.f, none) << 16;
    char* b = reinterpret_cast<char*>(layer ? o.bias2 : o.bias1) + kc * 512 + (lane >> 3) * 128 + (lane & 7) * 16;
    *reinterpret_cast<uint4*>(b) = make_uint4(kc ? 0u : word, 0u, 0u, 0u);
  } else if (part == 4) {
    if (lane < 2) {
      o.sn[NF + lane] = s.pow[lane ? 0 : 2];
      d.wfold[L::B3 + lane] = s.net[N::at(N::o_b3 + lane)];
    }
    if (lane == 2) d.wfold[L::SC + 1] = d.lr_mult ? d.lr * d.lr_mult[0] : d.lr;
  } else if (part < 7) {   // pair-major copy of the output layer
    const int e = lane + 32 * (part - 5), k = 2 * (e / 4) + (e & 1), q = (e % 4) >> 1;
    d.wfold[L::W3P + e] = s.net[N::at(N::o_w3 + q * H + k)];
  }
}
__global__ void __launch_bounds__(NT) k_prep_tc(const pylo_tensor_desc* __restrict__ descs, const pylo_atile* __restrict__ items,
                                                const pylo_step_params prm) {
  pdl_begin();
  constexpr int NF = Fam<PYLO_FAM_ADAFAC>::NF;
  __shared__ TcNet s;
  __shared__ float s_scale[NF];
  __shared__ double s_d[6][PYLO_STAT_STRIDE], s_few[TC_SUM_ROWS][PYLO_STAT_STRIDE];
  const pylo_atile it = items[blockIdx.x];
  if (it.strip) return;   // the whole CTA
  const pylo_tensor_desc& d = descs[it.tensor];
  const int tid = threadIdx.x;
  tc_ask_network<NT>(d, s);
  const float n = (float)d.n;
  if (prm.sum_tiles) {
    const double tot = d.n_tiles <= 16 ? unit_sum<TC_SUM_ROWS>(d, s_few) : unit_sum<6>(d, s_d);
    if (tid < NF) s_scale[tid] = rsqrtf((float)tot / n + prm.eps_norm);
    if (tid < PYLO_STAT_STRIDE) store_unit_sum(d, tot);
  } else if (tid < NF) {
    s_scale[tid] = rsqrtf(d.sums[tid] / n + prm.eps_norm);
  }
  tc_network<NT>(d, prm, s);
  if (tid < NF) reinterpret_cast<TcImage*>(d.wfold + TC_IMAGE)->sn[tid] = s_scale[tc_slot_feature(tid, tc_swap(d))] * s.pow[0];
}

// ================================================================================================
// Phase C: features -> network -> parameter / raw step
// ================================================================================================
// Network on E elements at once (weights are read from shared memory once per E elements).
// h1 comes in holding the bias (and, on the float4 path, the tabulated vector-feature terms);
// f holds the features in reference order.
template <int FAM, bool VECF, int E>
__device__ __forceinline__ void network(const uint32_t s_w, float (&h1)[E][Fam<FAM>::H],
                                        const float (&f)[E][Fam<FAM>::NF], float (&o0)[E], float (&o1)[E]) {
  using F = Fam<FAM>;
  using L = Fold<FAM>;
  constexpr int H = F::H;
  static_for<0, F::NF>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    if constexpr (VECF || !is_vec_feature<FAM>(k)) {
      static_for<0, H / 4>([&](auto jc) {
        constexpr int j = decltype(jc)::value * 4;
        const float4 w = lds4<L::W1 + k * H + j>(s_w);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const float fk = f[e][k];
          h1[e][j] = fmaf(w.x, fk, h1[e][j]); h1[e][j + 1] = fmaf(w.y, fk, h1[e][j + 1]);
          h1[e][j + 2] = fmaf(w.z, fk, h1[e][j + 2]); h1[e][j + 3] = fmaf(w.w, fk, h1[e][j + 3]);
        }
      });
    }
  });
  float h2[E][H];
  static_for<0, H / 4>([&](auto jc) {
    constexpr int j = decltype(jc)::value * 4;
    const float4 b = lds4<L::B2 + j>(s_w);
#pragma unroll
    for (int e = 0; e < E; ++e) { h2[e][j] = b.x; h2[e][j + 1] = b.y; h2[e][j + 2] = b.z; h2[e][j + 3] = b.w; }
  });
  static_for<0, H>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    float hk[E];
#pragma unroll
    for (int e = 0; e < E; ++e) hk[e] = fmaxf(h1[e][k], 0.f);
    static_for<0, H / 4>([&](auto jc) {
      constexpr int j = decltype(jc)::value * 4;
      const float4 w = lds4<L::W2 + k * H + j>(s_w);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        h2[e][j] = fmaf(w.x, hk[e], h2[e][j]); h2[e][j + 1] = fmaf(w.y, hk[e], h2[e][j + 1]);
        h2[e][j + 2] = fmaf(w.z, hk[e], h2[e][j + 2]); h2[e][j + 3] = fmaf(w.w, hk[e], h2[e][j + 3]);
      }
    });
  });
#pragma unroll
  for (int e = 0; e < E; ++e) { const float2 b3 = lds2<L::B3>(s_w); o0[e] = b3.x; o1[e] = b3.y; }
  static_for<0, H / 2>([&](auto kc) {
    constexpr int k = decltype(kc)::value * 2;
    const float4 w = lds4<L::W3 + 2 * k>(s_w);  // (k: dir, mag), (k+1: dir, mag)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float ha = fmaxf(h2[e][k], 0.f), hb = fmaxf(h2[e][k + 1], 0.f);
      o0[e] = fmaf(w.x, ha, o0[e]); o1[e] = fmaf(w.y, ha, o1[e]);
      o0[e] = fmaf(w.z, hb, o0[e]); o1[e] = fmaf(w.w, hb, o1[e]);
    }
  });
}

// The parameter's copies in the other ranks' buffers (peer-mapped memory reached by plain stores).
// The pointers are re-read from the descriptor at every store (they sit in L1) rather than held in
// fourteen registers; with n_peer == 0 the cost is one compare.
// n < 0: p[0] is a multicast address that maps every rank's buffer (NVLink switch multicast); one multimem
// store then reaches all of them and the switch does the replication, so the writer's link carries each value
// once instead of once per peer.
struct Peers {
  float* const* p;
  int n;
};
__device__ __forceinline__ Peers load_peers(const pylo_tensor_desc& d) { return Peers{d.p_peer, d.n_peer}; }
__device__ __forceinline__ void peer_store(const Peers& q, int64_t idx, float v) {
  if (q.n < 0) {
    asm volatile("multimem.st.relaxed.sys.global.f32 [%0], %1;" ::"l"(q.p[0] + idx), "f"(v) : "memory");
    return;
  }
#pragma unroll 1
  for (int k = 0; k < q.n; ++k) q.p[k][idx] = v;
}
__device__ __forceinline__ void peer_store4(const Peers& q, int64_t idx, float4 v) {
  if (q.n < 0) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};"
                 ::"l"(q.p[0] + idx), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    return;
  }
#pragma unroll 1
  for (int k = 0; k < q.n; ++k) st4(q.p[k] + idx, v);
}

// per-tensor scalars of the output stage, read once per tile
struct Fin {
  float exp_mult, step_mult, wd, lr, lr_eff, param_scale;
  int wd_mode;
};
__device__ __forceinline__ Fin make_fin(const pylo_tensor_desc& d, float param_scale, float lr_eff, int wd_mode) {
  return Fin{d.exp_mult, d.step_mult, d.wd, d.lr, lr_eff, param_scale, wd_mode};
}

template <int FAM>
__device__ __forceinline__ float finish(float p, float o0, float o1, const Fin& c) {
  if (FAM == PYLO_FAM_CELO2) return o0 * __expf(o1 * c.exp_mult);
  if (FAM == PYLO_FAM_ADAFAC) {
    const float upd = o0 * __expf(o1 * c.exp_mult) * c.step_mult;
    float pn = p - c.lr_eff * upd;
    if (c.wd_mode == 1) pn = fmaf(-(c.wd * c.lr), pn, pn);
    else if (c.wd_mode == 2) pn = fmaf(-(c.wd * c.lr), p, pn);
    return pn;
  }
  const float upd = c.param_scale * o0 * __expf(o1 * c.exp_mult) * c.step_mult;
  float pn = p - c.lr_eff * upd;
  if (c.wd > 0.f) pn = pn - c.wd * c.lr_eff * pn;
  return pn;
}

// word: of the step's status (0 for CELO2, whose parameters k_post_apply writes); block, blocks: of those that share the tiles
template <int FAM>
__device__ __forceinline__ void apply_tiles(const pylo_tensor_desc* __restrict__ descs, const pylo_tile* __restrict__ tiles, int n_tiles,
                                            int reverse, const pylo_step_params& prm, int word, int block, int blocks) {
  using F = Fam<FAM>;
  using L = Fold<FAM>;
  constexpr int H = F::H;
  __shared__ __align__(16) float s_w[L::SIZE + 4];
  const int tid = threadIdx.x;
  const uint32_t s_wa = smem_addr(s_w);
  int loaded = -1;
  for (int tt = block; tt < n_tiles; tt += blocks) {
    const int t = reverse ? (n_tiles - 1 - tt) : tt;
    const pylo_tile tl = tiles[t];
    const pylo_tensor_desc& d = descs[tl.tensor];
    if (loaded != tl.tensor) {
      __syncthreads();
#pragma unroll 4
      for (int e = tid; e < L::SIZE; e += NT) s_w[e] = __ldg(d.wfold + e);
      loaded = tl.tensor;
      __syncthreads();
      if (word) {
        pass_on(word, prm.host_status);
        return;
      }
    }
    const int64_t n = d.n, start = tl.start;
    const int cnt = tile_count(tl, n);
    const float gs = grad_scale_of(d, prm);
    const Fin fin = make_fin(d, s_w[L::SC], s_w[L::SC + 1], prm.wd_mode);
    const Peers peers = load_peers(d);
    const float* gp = d.g + start;
    float* pp = d.p + start;
    float* op = (FAM == PYLO_FAM_CELO2) ? d.out + start : pp;
    const float* m0p = d.m + start;
    const float* m1p = d.m + d.m_stride + start;
    const float* m2p = d.m + 2 * d.m_stride + start;
    const float* vp = d.v + start;

    {
      // E elements of a thread side by side: every weight read from shared memory serves all of them.  Two where the
      // network is small; the 32-wide one (reached with mlp_precision="fp32" only) has no registers for a second.
      constexpr int E = FAM == PYLO_FAM_ADAFAC ? 1 : 2;
      const bool vec1d = d.mode == PYLO_MODE_VEC1D;
      const int64_t La = vec1d ? n : d.La, Lb = vec1d ? n : d.Lb;
      const float* fac_r = d.r_is_a ? d.fac_a : d.fac_b;
      const float* fac_c = d.r_is_a ? d.fac_b : d.fac_a;
      GenPos pos(d, vec1d ? 0 : d.idx0 + start + tid, NT);
      for (int i0 = tid; i0 < cnt; i0 += E * NT) {
        float f[E][F::NF], p[E], h1[E][H], o0[E], o1[E];
#pragma unroll
        for (int u = 0; u < E; ++u) {
          const bool ok = i0 + u * NT < cnt;
          const int i = ok ? i0 + u * NT : i0;   // a thread without a second element repeats its first (in bounds)
          const float g = xform_grad(gp[i], gs, prm.clip_val, prm.nan_to_num);
          const float m0 = m0p[i], m1 = m1p[i], m2 = m2p[i], v = vp[i];
          p[u] = pp[i];
          const float rs = rsqrtf(v + prm.eps_feat);
          if (vec1d) {
            const int64_t e = start + i;
            const float r0 = d.fac_a[e], r1 = d.fac_a[n + e], r2 = d.fac_a[2 * n + e];
            const float* cb = d.fac_b ? d.fac_b : d.fac_a;
            elem_features<FAM>(f[u], g, p[u], m0, m1, m2, v, rs, safe_rsqrt(r0 + 1e-9f), safe_rsqrt(r1 + 1e-9f), safe_rsqrt(r2 + 1e-9f));
            vec_features<FAM>(f[u], r0, r1, r2, cb[e], cb[n + e], cb[2 * n + e]);
          } else {
            const int64_t a = ok ? pos.a() : 0, b = ok ? pos.b() : 0;
            pos.next();
            elem_features<FAM>(f[u], g, p[u], m0, m1, m2, v, rs, d.f_a[a] * d.f_b[b], d.f_a[La + a] * d.f_b[Lb + b],
                               d.f_a[2 * La + a] * d.f_b[2 * Lb + b]);
            const int64_t ir = d.r_is_a ? a : b, ic = d.r_is_a ? b : a;
            const int64_t Lr = d.r_is_a ? La : Lb, Lc = d.r_is_a ? Lb : La;
            vec_features<FAM>(f[u], fac_r[ir], fac_r[Lr + ir], fac_r[2 * Lr + ir], fac_c[ic], fac_c[Lc + ic], fac_c[2 * Lc + ic]);
          }
#pragma unroll
          for (int j = 0; j < H; ++j) h1[u][j] = s_w[L::B1 + j];
        }
        network<FAM, true, E>(s_wa, h1, f, o0, o1);
#pragma unroll
        for (int u = 0; u < E; ++u) {
          const int i = i0 + u * NT;
          if (i < cnt) {
            const float pn = finish<FAM>(p[u], o0[u], o1[u], fin);
            op[i] = pn;
            if (FAM != PYLO_FAM_CELO2) peer_store(peers, start + i, pn);
          }
        }
      }
    }
  }
}
template <int FAM>
__global__ void __launch_bounds__(NT) k_apply(const pylo_tensor_desc* __restrict__ descs,
                                              const pylo_tile* __restrict__ tiles, int n_tiles, int reverse,
                                              const pylo_step_params prm) {
  pdl_begin();
  apply_tiles<FAM>(descs, tiles, n_tiles, reverse, prm, FAM == PYLO_FAM_CELO2 ? 0 : reported(prm.status), blockIdx.x, gridDim.x);
}

// ================================================================================================
// Phase C for AdafacLO / ELO on FAST2D tensors: thread-owns-column kernel.
//
// The 39-32-32-2 network costs ~1600 fp32 FMAs per element once the vector-only features and
// the time features are folded away, so this sweep is bound by FMA issue, not by HBM.  Layout:
//   * a CTA takes a tile of RT rows x CW columns; a thread keeps ONE column for all its rows, so
//     the column's tabulated first-layer term (32 floats) and its three column factors stay in
//     registers, and the rows' terms sit in shared memory;
//   * two rows are processed at once so every weight read from shared memory feeds two elements;
//   * all multiply-adds are packed fma.rn.f32x2 (two fp32 FMAs per instruction) over pairs of
//     adjacent hidden units, which halves the issue slots the FMAs need;
//   * the first hidden layer's activations are staged through shared memory so that the second
//     layer can run as a short loop over k instead of 1000+ unrolled instructions;
//   * the next pair's operands are loaded while the current pair is computed.
// ================================================================================================
#define CC_TILE_ROWS 32   // rows per tile

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

#define CC_E 2            // rows a thread processes at once (each weight read feeds CC_E elements)
#define CC_CTAS_PER_SM 2  // 128 registers per thread

__device__ __forceinline__ float ldg_early(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

struct CcSmem {
  float w[Fold<PYLO_FAM_ADAFAC>::SIZE + 12];  // folded network
  float ha[CC_TILE_ROWS][32];                 // first-layer terms of the tile's rows (bias included)
  float fx[CC_TILE_ROWS][4];                  // the rows' three factors
  float hb[16][NT][2];                        // first-layer terms of the tile's columns, hidden-unit pairs
  float h1[32][NT][CC_E];                     // staged first-layer activations of the rows in flight
};

__global__ void __launch_bounds__(NT, CC_CTAS_PER_SM) k_apply_adafac_cols(const pylo_tensor_desc* __restrict__ descs,
                                                              const pylo_atile* __restrict__ ctiles, int n_ctiles,
                                                              const pylo_step_params prm) {
  pdl_begin();
  using F = Fam<PYLO_FAM_ADAFAC>;
  using L = Fold<PYLO_FAM_ADAFAC>;
  constexpr int E = CC_E;
  extern __shared__ __align__(16) unsigned char cc_raw[];
  CcSmem& sm = *reinterpret_cast<CcSmem*>(cc_raw);
  const int tid = threadIdx.x;
  const int word = reported(prm.status);
  pass_on(word, prm.host_status);
  if (word) return;
  int loaded = -1;
  for (int t = blockIdx.x; t < n_ctiles; t += gridDim.x) {
    const pylo_atile ct = ctiles[t];
    const pylo_tensor_desc& d = descs[ct.tensor];
    const int X = d.X, Y = d.Y;
    const int cw = ct.pad_ & 0xffff;                 // columns per CTA: 32, 64, 128 or 256
    const int n_sub = ct.pad_ >> 16;                 // the work item covers n_sub sub-tiles of CC_TILE_ROWS rows
    const int ng = NT / cw;                          // row groups
    const int rt = CC_TILE_ROWS;                     // rows per sub-tile
    const int rows_per_thread = rt / ng;             // 32, 16, 8 or 4
    const int y0 = ct.cb * cw;
    const int col = tid % cw, rg = tid / cw;
    const int y = y0 + col;
    const bool colok = y < Y;
    const int yc = colok ? y : 0;
    __syncthreads();
    if (loaded != ct.tensor) {
      for (int e = tid; e < L::SIZE; e += NT) sm.w[e] = d.wfold[e];
      loaded = ct.tensor;
    }
    // this column's first-layer term (stored transposed, [32][Y]); each thread keeps its own slot, and it
    // serves every sub-tile of the work item
#pragma unroll 4
    for (int j = 0; j < 16; ++j) {
      sm.hb[j][tid][0] = d.h_b[(int64_t)(2 * j) * Y + yc];
      sm.hb[j][tid][1] = d.h_b[(int64_t)(2 * j + 1) * Y + yc];
    }
    const float fb0 = d.f_b[yc], fb1 = d.f_b[Y + yc], fb2 = d.f_b[2 * (int64_t)Y + yc];
    const float gs = grad_scale_of(d, prm);
    const int64_t n = d.n;
    const float* __restrict__ gp = d.g;
    float* __restrict__ pp = d.p;
    const float* __restrict__ mp = d.m;
    const float* __restrict__ vp = d.v;
    const Peers peers = load_peers(d);
    for (int sub = 0; sub < n_sub; ++sub) {
    const int x0 = (ct.strip * n_sub + sub) * rt;
    if (x0 >= X) break;
    __syncthreads();  // the previous sub-tile's rows are no longer read
    for (int e = tid; e < rt * 32; e += NT) {
      const int r = e >> 5, x = x0 + r;
      sm.ha[r][e & 31] = x < X ? d.h_a[(int64_t)x * 32 + (e & 31)] : 0.f;
    }
    for (int e = tid; e < rt * 4; e += NT) {
      const int r = e >> 2, x = x0 + r;
      sm.fx[r][e & 3] = x < X ? d.fx[(int64_t)x * 4 + (e & 3)] : 0.f;
    }
    __syncthreads();
    const Fin fin = make_fin(d, 1.0f, sm.w[L::SC + 1], prm.wd_mode);
    float cg[E], cp[E], cm0[E], cm1[E], cm2[E], cv[E];
    auto load_rows = [&](int q, float* g, float* p, float* m0, float* m1, float* m2, float* v) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int x = x0 + rg + ng * (q + e);
        const bool ok = colok && x < X;
        const int64_t idx = ok ? (int64_t)x * Y + y : 0;
        // issued as volatile loads so that they stay here, a whole row pair ahead of their use
        g[e] = ldg_early(gp + idx); p[e] = ldg_early(pp + idx); m0[e] = ldg_early(mp + idx);
        m1[e] = ldg_early(mp + n + idx); m2[e] = ldg_early(mp + 2 * n + idx); v[e] = ldg_early(vp + idx);
      }
    };
    load_rows(0, cg, cp, cm0, cm1, cm2, cv);
#pragma unroll 1
    for (int q = 0; q < rows_per_thread; q += E) {
      float ng_[E], np_[E], nm0[E], nm1[E], nm2[E], nv[E];
      const bool more = q + E < rows_per_thread;
      if (more) load_rows(q + E, ng_, np_, nm0, nm1, nm2, nv);
      // ---- features of the rows in flight
      float f[E][F::NF];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int r = rg + ng * (q + e);
        const float g = xform_grad(cg[e], gs, prm.clip_val, prm.nan_to_num);
        const float rs = rsqrt_pos(cv[e] + prm.eps_feat);
        const float4 fa = ld4(&sm.fx[r][0]);
        elem_features<PYLO_FAM_ADAFAC>(f[e], g, cp[e], cm0[e], cm1[e], cm2[e], cv[e], rs, fa.x * fb0, fa.y * fb1, fa.z * fb2);
      }
      // ---- first layer in two halves of 16 hidden units
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint64_t h1[E][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint64_t b = *reinterpret_cast<const uint64_t*>(&sm.hb[half * 8 + j][tid][0]);
#pragma unroll
          for (int e = 0; e < E; ++e)
            h1[e][j] = add2(*reinterpret_cast<const uint64_t*>(&sm.ha[rg + ng * (q + e)][half * 16 + 2 * j]), b);
        }
        static_for<0, F::NF>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          if constexpr (!is_vec_feature<PYLO_FAM_ADAFAC>(k)) {
            uint64_t fk[E];
#pragma unroll
            for (int e = 0; e < E; ++e) fk[e] = pack2(f[e][k], f[e][k]);
            const ulonglong2* wrow = reinterpret_cast<const ulonglong2*>(&sm.w[L::W1 + k * 32 + half * 16]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const ulonglong2 w = wrow[j];
#pragma unroll
              for (int e = 0; e < E; ++e) {
                h1[e][2 * j] = fma2(w.x, fk[e], h1[e][2 * j]);
                h1[e][2 * j + 1] = fma2(w.y, fk[e], h1[e][2 * j + 1]);
              }
            }
          }
        });
        // stage relu(h1), the E rows of one hidden unit side by side, for the second layer's dynamic index
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float lo[E], hi[E];
#pragma unroll
          for (int e = 0; e < E; ++e) { unpack2(h1[e][j], lo[e], hi[e]); lo[e] = fmaxf(lo[e], 0.f); hi[e] = fmaxf(hi[e], 0.f); }
          if constexpr (E == 4) {
            st4(&sm.h1[half * 16 + 2 * j][tid][0], make_float4(lo[0], lo[1], lo[2], lo[3]));
            st4(&sm.h1[half * 16 + 2 * j + 1][tid][0], make_float4(hi[0], hi[1], hi[2], hi[3]));
          } else {
            *reinterpret_cast<float2*>(&sm.h1[half * 16 + 2 * j][tid][0]) = make_float2(lo[0], lo[1]);
            *reinterpret_cast<float2*>(&sm.h1[half * 16 + 2 * j + 1][tid][0]) = make_float2(hi[0], hi[1]);
          }
        }
      }
      // ---- second layer: h2 = b2 + W2^T relu(h1)
      uint64_t h2[E][16];
      {
        const ulonglong2* brow = reinterpret_cast<const ulonglong2*>(&sm.w[L::B2]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const ulonglong2 b = brow[j];
#pragma unroll
          for (int e = 0; e < E; ++e) { h2[e][2 * j] = b.x; h2[e][2 * j + 1] = b.y; }
        }
      }
      {
        // the staged activations of unit k+1 are requested while unit k is multiplied in
        float2 cur = *reinterpret_cast<const float2*>(&sm.h1[0][tid][0]);
#pragma unroll 4
        for (int k = 0; k < 32; ++k) {
          const float2 nxt = *reinterpret_cast<const float2*>(&sm.h1[(k + 1) & 31][tid][0]);
          const uint64_t hk0 = pack2(cur.x, cur.x), hk1 = pack2(cur.y, cur.y);
          const ulonglong2* wrow = reinterpret_cast<const ulonglong2*>(&sm.w[L::W2 + k * 32]);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const ulonglong2 w = wrow[j];
            h2[0][2 * j] = fma2(w.x, hk0, h2[0][2 * j]); h2[0][2 * j + 1] = fma2(w.y, hk0, h2[0][2 * j + 1]);
            h2[1][2 * j] = fma2(w.x, hk1, h2[1][2 * j]); h2[1][2 * j + 1] = fma2(w.y, hk1, h2[1][2 * j + 1]);
          }
          cur = nxt;
        }
      }
      // ---- output layer: direction and magnitude as packed dot products over hidden-unit pairs, two
      //      partial accumulators each so that no dependent chain is longer than eight FMAs
      uint64_t od[E][2], om[E][2];
#pragma unroll
      for (int e = 0; e < E; ++e) { od[e][0] = od[e][1] = 0ull; om[e][0] = om[e][1] = 0ull; }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&sm.w[L::W3P + 4 * j]);  // (dir pair, mag pair)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          float a, b;
          unpack2(h2[e][j], a, b);
          const uint64_t r = pack2(fmaxf(a, 0.f), fmaxf(b, 0.f));
          od[e][j & 1] = fma2(w.x, r, od[e][j & 1]);
          om[e][j & 1] = fma2(w.y, r, om[e][j & 1]);
        }
      }
      float o0v[E], o1v[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        float a, b, c, dd;
        unpack2(add2(od[e][0], od[e][1]), a, b);
        unpack2(add2(om[e][0], om[e][1]), c, dd);
        o0v[e] = (a + b) + sm.w[L::B3];
        o1v[e] = (c + dd) + sm.w[L::B3 + 1];
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int x = x0 + rg + ng * (q + e);
        if (colok && x < X) {
          const float pn = finish<PYLO_FAM_ADAFAC>(cp[e], o0v[e], o1v[e], fin);
          pp[(int64_t)x * Y + y] = pn;
          peer_store(peers, (int64_t)x * Y + y, pn);
        }
      }
      if (more) {
#pragma unroll
        for (int e = 0; e < E; ++e) { cg[e] = ng_[e]; cp[e] = np_[e]; cm0[e] = nm0[e]; cm1[e] = nm1[e]; cm2[e] = nm2[e]; cv[e] = nv[e]; }
      }
    }
    }  // sub-tiles
  }
}

#include "pylo_small_front.cuh"
#include "pylo_apply_tc.cuh"
#include "pylo_ns_gemm.cuh"
#include "pylo_ns_f16.cuh"
#include "pylo_ns_cluster.cuh"

// ================================================================================================
// Phase C for CELO2 / ELO_CELO2 / VeLO on FAST2D tensors: packed kernel.
//
// These networks are small (30-8-8-3, 30-4-4-3), so the sweep should run at HBM speed; what stands
// in the way is the work per element.  218 M CELO2 parameters (a Llama block) take 2197 us (2747 before constant weights and
// early requests), 10.1 ps per element, of which the multiply-adds' pipe needs 8; 355 M VeLO parameters (GPT-2-medium) 1986 us
// (2345) = 5.0 TB/s.
//   * all arithmetic is done on PAIRS OF ADJACENT ELEMENTS with packed fp32x2 instructions: a
//     float4 load already is two such pairs, so no register moves are needed to form them;
//   * a weight is a pair (w, w) of one register, or of a constant: four weights per read from shared memory, each feeds four elements;
//   * a thread keeps four columns for all rows of its tile, so the columns' tabulated first-layer
//     terms and factors stay in registers; the rows' terms arrive as broadcast loads;
//   * the next row's six float4 operands are requested before the current row is computed;
//   * a packed multiply-add with three operands in registers occupies the pipe for 3.3 cycles (six registers to read), with one
//     of them a constant for 2.3: where one network serves all units (CELO2) its weights are arguments of the launch, and the
//     eighteen features are normalised instead of the weights; where every tensor has its own (VeLO) a weight is one register
//     taken twice (3.0 cycles), and a read from shared memory brings four of them, not two;
//   * the rows' first-layer terms and factors are staged in shared memory, up to 256 rows at a time: read from global memory
//     row by row, every row began with their latency.
// ================================================================================================
template <int FAM>
struct PkW {  // the network in shared memory (floats), or as an argument of the launch
  static constexpr int H = Fam<FAM>::H, NE = 18;  // NE: element-wise features
  static constexpr int W1 = 0;                    // [NE][H]
  static constexpr int W2 = W1 + NE * H;          // [H][H], k-major
  static constexpr int B2 = W2 + H * H;           // [H]
  static constexpr int W3 = B2 + H;               // [H][2]
  static constexpr int B3 = W3 + H * 2;           // [2], two unused
  static constexpr int SIZE = B3 + 4;
};
template <int FAM>
struct PkNet { float w[PkW<FAM>::SIZE]; };
// place of an element-wise feature among them
__host__ __device__ constexpr int pk_index(int k) { return k < 15 ? k : k - 12; }

struct PkBase {  // packed per-pair operands the features are made of
  uint64_t g, cg, p, m0, m1, m2, v, rs, k0, k1, k2;
};

template <int K>
__device__ __forceinline__ uint64_t pk_feature(const PkBase& b) {
  if constexpr (K == 0) return b.g;
  else if constexpr (K == 1) return b.cg;
  else if constexpr (K == 2) return b.p;
  else if constexpr (K == 3) return b.m0;
  else if constexpr (K == 4) return b.m1;
  else if constexpr (K == 5) return b.m2;
  else if constexpr (K == 6) return b.v;
  else if constexpr (K == 7) return mul2(b.m0, b.rs);
  else if constexpr (K == 8) return mul2(b.m1, b.rs);
  else if constexpr (K == 9) return mul2(b.m2, b.rs);
  else if constexpr (K == 10) return b.rs;
  else if constexpr (K == 11) return mul2(b.k0, b.g);
  else if constexpr (K == 12) return mul2(b.k1, b.g);
  else if constexpr (K == 13) return mul2(b.k2, b.g);
  else if constexpr (K == 14) return mul2(b.g, b.rs);
  else if constexpr (K == 27) return mul2(b.k0, b.m0);
  else if constexpr (K == 28) return mul2(b.k1, b.m1);
  else return mul2(b.k2, b.m2);
}

// a 128-bit load issued where it is written: the compiler moves the next row's loads down to their use (CELO2 3023 us instead of 2197)
__device__ __forceinline__ float4 ld4_early(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
#define PK_ROWS 16  // rows per thread in a tile, unless the tag's upper half says otherwise
#define PK_STAGE 256  // rows staged at once

#ifndef PK_CTAS_VELO
#define PK_CTAS_VELO 2
#endif
#ifndef PK_CTAS_CELO2
#define PK_CTAS_CELO2 1   // its 8-wide layers want registers more than a second CTA (224 bytes of spills: 2357 -> 2435 us over a Llama block)
#endif
// ARG: one network for all units, which comes as an argument of the launch; the features are normalised instead of the weights.
// RAGGED: matrices whose rows do not start on 16-byte boundaries: a thread's four columns are a tile's quarter apart, so that a
// warp's single accesses are to neighbouring elements.
template <int FAM, bool ARG, bool RAGGED>
__device__ __forceinline__ void packed_tiles(const pylo_tensor_desc* __restrict__ descs, const pylo_atile* __restrict__ ctiles, int n_ctiles,
                                             const pylo_step_params& prm, const PkNet<FAM>& net, int word, int block, int blocks) {
  using F = Fam<FAM>;
  using L = Fold<FAM>;
  using W = PkW<FAM>;
  constexpr int H = F::H;
  constexpr int RP = 2 * H + 4;     // floats of a staged row: H pairs (v, v), then its three factors
  __shared__ __align__(16) float s_w[ARG ? 20 : W::SIZE];   // ARG: the normalisers of the element-wise features
  __shared__ __align__(16) float s_row[PK_STAGE * RP];
  __shared__ float s_sc[2];
  __shared__ float s_red[40];
  float* const squares = FAM == PYLO_FAM_CELO2 ? prm.step_squares : nullptr;
  const int tid = threadIdx.x;
  const uint32_t s_wa = smem_addr(s_w);
  int loaded = -1;
  for (int t = block; t < n_ctiles; t += blocks) {
    const pylo_atile ct = ctiles[t];
    const pylo_tensor_desc& d = descs[ct.tensor];
    const int X = d.X, Y = d.Y;
    const int tpr = ct.pad_ & 0xffff; // threads per row: 8 .. 256 (a thread owns 4 columns)
    const int rpt = ct.pad_ >> 16 ? ct.pad_ >> 16 : PK_ROWS;   // rows per thread
    const int ng = NT / tpr;          // row groups
    const int rt = rpt * ng;          // rows per tile
    const int x0 = ct.strip * rt, y0 = ct.cb * tpr * 4;
    if (loaded != ct.tensor) {
      __syncthreads();
      const float* __restrict__ wf = d.wfold;
      if (ARG) {
        if (tid < W::NE) s_w[tid] = __ldg(wf + L::SN + (tid < 15 ? tid : tid + 12));
      } else {
        for (int e = tid; e < W::NE * H; e += NT) { const int k = e / H; s_w[W::W1 + e] = __ldg(wf + L::W1 + (k < 15 ? e : e + 12 * H)); }
        for (int e = tid; e < H * H; e += NT) s_w[W::W2 + e] = __ldg(wf + L::W2 + e);
        if (tid < H) s_w[W::B2 + tid] = __ldg(wf + L::B2 + tid);
        if (tid < H * 2) s_w[W::W3 + tid] = __ldg(wf + L::W3 + tid);
        if (tid < 2) s_w[W::B3 + tid] = __ldg(wf + L::B3 + tid);
      }
      if (tid < 2) s_sc[tid] = __ldg(wf + L::SC + tid);
      loaded = ct.tensor;
      __syncthreads();
      if (word) {
        pass_on(word, prm.host_status);
        return;
      }
    }
    const int y = y0 + (RAGGED ? tid % tpr : 4 * (tid % tpr)), rg = tid / tpr;
    const bool colok = y < Y;
    const int yc = colok ? y : 0;
    int yu[4];   // RAGGED: the thread's columns, or 0 where there is none
#pragma unroll
    for (int u = 0; u < 4; ++u) yu[u] = y + u * tpr < Y ? y + u * tpr : 0;
    auto columns = [&](const float* p) { return RAGGED ? make_float4(__ldg(p + yu[0]), __ldg(p + yu[1]), __ldg(p + yu[2]), __ldg(p + yu[3])) : ldg4(p + yc); };
    // VeLO: p + rate * (...), then + decay * that (lr_eff may have either sign)
    const float exp_mult = d.exp_mult, rate = -(s_sc[1] * s_sc[0] * d.step_mult), decay = d.wd > 0.f ? -(d.wd * s_sc[1]) : 0.f;
    const float gs = grad_scale_of(d, prm);
    const float eps_feat = prm.eps_feat, clip = prm.clip_val;
    const int64_t n = d.n;
    // the four columns' first-layer terms and factors: pairs (col, col+1) and (col+2, col+3)
    uint64_t hb[2][H], fb[2][3];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const float4 q = columns(d.h_b + (int64_t)j * Y);
      hb[0][j] = pack2(q.x, q.y);
      hb[1][j] = pack2(q.z, q.w);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 q = columns(d.f_b + (int64_t)k * Y);
      fb[0][k] = pack2(q.x, q.y);
      fb[1][k] = pack2(q.z, q.w);
    }
    const float* __restrict__ gp = d.g;
    float* __restrict__ pp = d.p;
    float* __restrict__ op = (FAM == PYLO_FAM_CELO2) ? d.out : d.p;
    const float* __restrict__ mp = d.m;
    const float* __restrict__ vp = d.v;
    const float* __restrict__ hap = d.h_a;
    const float* __restrict__ fxp = d.fx;
    const Peers peers = load_peers(d);

    float4 cg, cp, cm0, cm1, cm2, cv;
    auto load_row = [&](int q, float4& g, float4& p, float4& m0, float4& m1, float4& m2, float4& v) {
      const int x = x0 + rg + ng * q;
      if constexpr (RAGGED) {
        const int64_t at = x < X ? (int64_t)x * Y : 0;
        auto four = [&](const float* p) { return make_float4(ldg_early(p + yu[0]), ldg_early(p + yu[1]), ldg_early(p + yu[2]), ldg_early(p + yu[3])); };
        g = four(gp + at); p = four(pp + at); m0 = four(mp + at); m1 = four(mp + n + at); m2 = four(mp + 2 * n + at); v = four(vp + at);
      } else {
        const int64_t idx = (colok && x < X) ? (int64_t)x * Y + y : 0;
        g = ld4_early(gp + idx); p = ld4_early(pp + idx); m0 = ld4_early(mp + idx); m1 = ld4_early(mp + n + idx); m2 = ld4_early(mp + 2 * n + idx); v = ld4_early(vp + idx);
      }
    };
    load_row(0, cg, cp, cm0, cm1, cm2, cv);
    float sq = 0.f;   // CELO2: of this thread's raw steps
    const int sub = min(PK_ROWS, PK_STAGE / ng);   // rows per thread and stage
#pragma unroll 1
    for (int q = 0; q < rpt; ++q) {
      if (x0 + q * ng >= X) break;   // the same for the whole CTA
      if (q % sub == 0) {
        __syncthreads();   // the previous stage is no longer read
        const int first = x0 + q * ng, rows = min(sub * ng, X - first);
        for (int e = tid; e < rows * (RP / 4); e += NT) {
          const int r = e / (RP / 4), k = e - r * (RP / 4);
          st4(s_row + r * RP + 4 * k, k < H / 2 ? ldg4(hap + (int64_t)(first + r) * 2 * H + 4 * k) : ldg4(fxp + 4 * (int64_t)(first + r)));
        }
        __syncthreads();
      }
      float4 ng_, np_, nm0, nm1, nm2, nv;
      if (q + 1 < rpt) load_row(q + 1, ng_, np_, nm0, nm1, nm2, nv);
      const int x = x0 + rg + ng * q;
      const float* const row = s_row + (x < X ? rg + ng * (q % sub) : 0) * RP;
      const float4 fa = ld4(row + 2 * H);
      PkBase b[2];
      {
        float ge[4] = {cg.x, cg.y, cg.z, cg.w};
        float rs[4] = {rsqrt_pos(cv.x + eps_feat), rsqrt_pos(cv.y + eps_feat), rsqrt_pos(cv.z + eps_feat), rsqrt_pos(cv.w + eps_feat)};
        float cl[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { ge[u] = xform_grad(ge[u], gs, clip, prm.nan_to_num); cl[u] = fminf(fmaxf(ge[u], -0.1f), 0.1f); }
        const uint64_t a0 = pack2(fa.x, fa.x), a1 = pack2(fa.y, fa.y), a2 = pack2(fa.z, fa.z);
        b[0] = PkBase{pack2(ge[0], ge[1]), pack2(cl[0], cl[1]), pack2(cp.x, cp.y), pack2(cm0.x, cm0.y), pack2(cm1.x, cm1.y),
                      pack2(cm2.x, cm2.y), pack2(cv.x, cv.y), pack2(rs[0], rs[1]), mul2(a0, fb[0][0]), mul2(a1, fb[0][1]), mul2(a2, fb[0][2])};
        b[1] = PkBase{pack2(ge[2], ge[3]), pack2(cl[2], cl[3]), pack2(cp.z, cp.w), pack2(cm0.z, cm0.w), pack2(cm1.z, cm1.w),
                      pack2(cm2.z, cm2.w), pack2(cv.z, cv.w), pack2(rs[2], rs[3]), mul2(a0, fb[1][0]), mul2(a1, fb[1][1]), mul2(a2, fb[1][2])};
      }
      // first layer: h1 = (row term + column term) + sum_k W1[k] f_k
      uint64_t h1[2][H];
#pragma unroll
      for (int j = 0; j < H; j += 2) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row + 2 * j);
        h1[0][j] = add2(hb[0][j], a.x); h1[0][j + 1] = add2(hb[0][j + 1], a.y);
        h1[1][j] = add2(hb[1][j], a.x); h1[1][j + 1] = add2(hb[1][j + 1], a.y);
      }
      // four weights at a time, each as a pair (w, w): constants where they are an argument, which leaves a product two operands
      // to read from registers (three cost it 3.3 cycles instead of 2.3), else from shared memory
      auto weights = [&](auto at) -> float4 {
        constexpr int A = decltype(at)::value;
        if constexpr (ARG) return make_float4(net.w[A], net.w[A + 1], net.w[A + 2], net.w[A + 3]);
        else return lds4<A>(s_wa);
      };
      float4 scales;
      static_for<0, F::NF>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        if constexpr (!is_vec_feature<FAM>(k)) {
          constexpr int i = pk_index(k);
          uint64_t f0 = pk_feature<k>(b[0]), f1 = pk_feature<k>(b[1]);
          if constexpr (ARG) {
            if constexpr (i % 4 == 0) scales = lds4<i>(s_wa);
            const float sc = i % 4 == 0 ? scales.x : i % 4 == 1 ? scales.y : i % 4 == 2 ? scales.z : scales.w;
            f0 = mul2(f0, pack2(sc, sc));
            f1 = mul2(f1, pack2(sc, sc));
          }
          static_for<0, H / 4>([&](auto jc) {
            constexpr int j = decltype(jc)::value * 4;
            const float4 w = weights(std::integral_constant<int, W::W1 + i * H + j>{});
            const uint64_t w0 = pack2(w.x, w.x), w1 = pack2(w.y, w.y), w2 = pack2(w.z, w.z), w3 = pack2(w.w, w.w);
            h1[0][j] = fma2(w0, f0, h1[0][j]); h1[1][j] = fma2(w0, f1, h1[1][j]);
            h1[0][j + 1] = fma2(w1, f0, h1[0][j + 1]); h1[1][j + 1] = fma2(w1, f1, h1[1][j + 1]);
            h1[0][j + 2] = fma2(w2, f0, h1[0][j + 2]); h1[1][j + 2] = fma2(w2, f1, h1[1][j + 2]);
            h1[0][j + 3] = fma2(w3, f0, h1[0][j + 3]); h1[1][j + 3] = fma2(w3, f1, h1[1][j + 3]);
          });
        }
      });
      // second layer
      uint64_t h2[2][H];
      static_for<0, H / 4>([&](auto jc) {
        constexpr int j = decltype(jc)::value * 4;
        const float4 w = weights(std::integral_constant<int, W::B2 + j>{});
#pragma unroll
        for (int e = 0; e < 2; ++e) { h2[e][j] = pack2(w.x, w.x); h2[e][j + 1] = pack2(w.y, w.y); h2[e][j + 2] = pack2(w.z, w.z); h2[e][j + 3] = pack2(w.w, w.w); }
      });
      static_for<0, H>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        uint64_t r[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float lo, hi;
          unpack2(h1[e][k], lo, hi);
          r[e] = pack2(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
        }
        static_for<0, H / 4>([&](auto jc) {
          constexpr int j = decltype(jc)::value * 4;
          const float4 w = weights(std::integral_constant<int, W::W2 + k * H + j>{});
          const uint64_t w0 = pack2(w.x, w.x), w1 = pack2(w.y, w.y), w2 = pack2(w.z, w.z), w3 = pack2(w.w, w.w);
          h2[0][j] = fma2(w0, r[0], h2[0][j]); h2[1][j] = fma2(w0, r[1], h2[1][j]);
          h2[0][j + 1] = fma2(w1, r[0], h2[0][j + 1]); h2[1][j + 1] = fma2(w1, r[1], h2[1][j + 1]);
          h2[0][j + 2] = fma2(w2, r[0], h2[0][j + 2]); h2[1][j + 2] = fma2(w2, r[1], h2[1][j + 2]);
          h2[0][j + 3] = fma2(w3, r[0], h2[0][j + 3]); h2[1][j + 3] = fma2(w3, r[1], h2[1][j + 3]);
        });
      });
      // output layer: direction and magnitude
      const float4 b3 = weights(std::integral_constant<int, W::B3>{});
      uint64_t o0[2] = {pack2(b3.x, b3.x), pack2(b3.x, b3.x)}, o1[2] = {pack2(b3.y, b3.y), pack2(b3.y, b3.y)};
      static_for<0, H / 2>([&](auto kc) {
        constexpr int k = decltype(kc)::value * 2;
        const float4 w = weights(std::integral_constant<int, W::W3 + k * 2>{});   // (dir, mag) of two units
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float lo, hi;
          unpack2(h2[e][k], lo, hi);
          uint64_t r = pack2(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
          o0[e] = fma2(pack2(w.x, w.x), r, o0[e]);
          o1[e] = fma2(pack2(w.y, w.y), r, o1[e]);
          unpack2(h2[e][k + 1], lo, hi);
          r = pack2(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
          o0[e] = fma2(pack2(w.z, w.z), r, o0[e]);
          o1[e] = fma2(pack2(w.w, w.w), r, o1[e]);
        }
      });
      if (colok && x < X) {
        float d0, d1, d2, d3, m0, m1, m2, m3;
        unpack2(o0[0], d0, d1); unpack2(o0[1], d2, d3);
        unpack2(o1[0], m0, m1); unpack2(o1[1], m2, m3);
        float4 res;
        if constexpr (FAM == PYLO_FAM_VELO) {   // finish(), two elements at a time and its constants made once per tile
          auto two = [&](float p0, float p1, float a, float b, float m, float n, float& r0, float& r1) {
            uint64_t pn = fma2(mul2(pack2(a, b), pack2(__expf(m * exp_mult), __expf(n * exp_mult))), pack2(rate, rate), pack2(p0, p1));
            if (decay != 0.f) pn = fma2(pack2(decay, decay), pn, pn);
            unpack2(pn, r0, r1);
          };
          two(cp.x, cp.y, d0, d1, m0, m1, res.x, res.y);
          two(cp.z, cp.w, d2, d3, m2, m3, res.z, res.w);
        } else {
          res = make_float4(d0 * __expf(m0 * exp_mult), d1 * __expf(m1 * exp_mult), d2 * __expf(m2 * exp_mult), d3 * __expf(m3 * exp_mult));
          if constexpr (RAGGED) {
            sq += res.x * res.x;
            if (y + tpr < Y) sq += res.y * res.y;
            if (y + 2 * tpr < Y) sq += res.z * res.z;
            if (y + 3 * tpr < Y) sq += res.w * res.w;
          } else {
            sq += res.x * res.x + res.y * res.y + res.z * res.z + res.w * res.w;
          }
        }
        if constexpr (RAGGED) {
          const float r4[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (y + u * tpr < Y) {
              const int64_t at = (int64_t)x * Y + y + u * tpr;
              op[at] = r4[u];
              if (FAM != PYLO_FAM_CELO2) peer_store(peers, at, r4[u]);
            }
        } else {
          st4(op + (int64_t)x * Y + y, res);
          if (FAM != PYLO_FAM_CELO2) peer_store4(peers, (int64_t)x * Y + y, res);
        }
      }
      if (q + 1 < rpt) { cg = ng_; cp = np_; cm0 = nm0; cm1 = nm1; cm2 = nm2; cv = nv; }
    }
    if (FAM == PYLO_FAM_CELO2 && squares) {
      sq = block_sum(sq, s_red);
      if (tid == 0) squares[t] = sq;
    }
  }
}
// VeLO: the items on the first `packed` CTAs and other units' tiles (those of k_apply) on the rest, at the same time, instead of two
// launches one after the other, 7.5 and 4.7 us on a perceptron of 118 K: one of 7.6 us (step 48.3 -> 44.5 us; unaligned 1001-wide
// layers 127 -> 123, 110 M transformer 726 -> 721, convolutions with five tiles per item 318 -> 316).  Not CELO2: its vectors are not
// in the plan, and tiles at one CTA per SM, which its items want, are slow (convolutions 15.6 -> 24.9 ms).
template <int FAM, bool ARG, bool RAGGED>
__global__ void __launch_bounds__(NT, FAM == PYLO_FAM_VELO ? PK_CTAS_VELO : PK_CTAS_CELO2) k_apply_packed(const pylo_tensor_desc* __restrict__ descs,
                                                        const pylo_atile* __restrict__ ctiles, int n_ctiles, int packed,
                                                        const pylo_tile* __restrict__ tiles, int n_tiles,
                                                        const pylo_step_params prm, const __grid_constant__ PkNet<FAM> net) {
  pdl_begin();
  if constexpr (FAM == PYLO_FAM_VELO) {
    const int word = reported(prm.status);
    if ((int)blockIdx.x < packed) packed_tiles<FAM, ARG, RAGGED>(descs, ctiles, n_ctiles, prm, net, word, blockIdx.x, packed);
    else apply_tiles<FAM>(descs, tiles, n_tiles, 0, prm, word, blockIdx.x - packed, gridDim.x - packed);
  } else {
    packed_tiles<FAM, ARG, RAGGED>(descs, ctiles, n_ctiles, prm, net, 0, blockIdx.x, gridDim.x);   // k_post_apply writes the parameters
  }
}

// ================================================================================================
// CELO2 tail: second-moment normaliser over a matrix, then the parameter update
// ================================================================================================
// From the last tile to the first: what the sweep before wrote last is still in L2, and k_post_apply, which goes the other way,
// finds the first steps there.
__global__ void __launch_bounds__(NT) k_post_sums(const pylo_post_item* __restrict__ items,
                                                  const pylo_tile* __restrict__ tiles, int n_tiles) {
  pdl_begin();
  __shared__ float s_red[40];
  for (int tt = blockIdx.x; tt < n_tiles; tt += gridDim.x) {
    const int t = n_tiles - 1 - tt;
    const pylo_tile tl = tiles[t];
    const pylo_post_item& it = items[tl.tensor];
    const float* s = it.step + tl.start;
    const int cnt = tile_count(tl, it.n);
    float acc = 0.f;
    if (((((uintptr_t)s) & 15) == 0)) {
      const int c4 = cnt & ~3;
      for (int i = threadIdx.x * 4; i < c4; i += NT * 4) {
        const float4 q = ld4(s + i);
        acc += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
      }
      for (int i = c4 + threadIdx.x; i < cnt; i += NT) acc += s[i] * s[i];
    } else {
      for (int i = threadIdx.x; i < cnt; i += NT) acc += s[i] * s[i];
    }
    const float tot = block_sum(acc, s_red);
    if (threadIdx.x == 0) it.part[t - it.tile0] = tot;
  }
}

// block, blocks: of those that share the tiles
__device__ __forceinline__ void post_apply_tiles(const pylo_post_item* __restrict__ items, const pylo_tile* __restrict__ tiles, int n_tiles,
                                                 int word, int* __restrict__ host_status, int block, int blocks) {
  __shared__ float s_scale;
  for (int t = block; t < n_tiles; t += blocks) {
    const pylo_tile tl = tiles[t];
    const pylo_post_item& it = items[tl.tensor];
    __syncthreads();
    if (threadIdx.x < 32) {  // every tile re-reduces the item's partials in the same fixed order
      double acc = 0.0;
      for (int q = threadIdx.x; q < it.n_tiles; q += 32) acc += (double)it.part[q];
      acc = warp_sum_d(acc);
      if (threadIdx.x == 0) s_scale = rsqrtf(1e-9f + (float)acc / (float)it.n) * it.rmsmult;
    }
    __syncthreads();
    if (word) {
      pass_on(word, host_status);
      return;
    }
    const float sc = s_scale, lr = it.lr, wd = it.wd;
    const float* s = it.step + tl.start;
    float* p = it.p + tl.start;
    const int cnt = tile_count(tl, it.n);
    const bool al = (((((uintptr_t)s) | ((uintptr_t)p)) & 15) == 0);
    const int c4 = al ? (cnt & ~3) : 0;
    for (int i = threadIdx.x * 4; i < c4; i += NT * 4) {
      const float4 q = ld4(s + i);
      float4 w = ld4(p + i);
      w.x = fmaf(-lr, fmaf(q.x, sc, wd * w.x), w.x);
      w.y = fmaf(-lr, fmaf(q.y, sc, wd * w.y), w.y);
      w.z = fmaf(-lr, fmaf(q.z, sc, wd * w.z), w.z);
      w.w = fmaf(-lr, fmaf(q.w, sc, wd * w.w), w.w);
      st4(p + i, w);
    }
    for (int i = c4 + threadIdx.x; i < cnt; i += NT) p[i] = fmaf(-lr, fmaf(s[i], sc, wd * p[i]), p[i]);
  }
}
__global__ void __launch_bounds__(NT) k_post_apply(const pylo_post_item* __restrict__ items,
                                                   const pylo_tile* __restrict__ tiles, int n_tiles,
                                                   const int* __restrict__ status, int* __restrict__ host_status) {
  pdl_begin();
  post_apply_tiles(items, tiles, n_tiles, reported(status), host_status, blockIdx.x, gridDim.x);
}

// ================================================================================================
// AdamW branch
// ================================================================================================
// Bound by HBM (28 or 44 B per element): float4 where every stream allows it, two pieces of a thread in flight.  262 M
// elements: 1829 us (4.0 TB/s) with scalar loads before.
struct Adam { float beta1, omb1, beta2, omb2, eps, bc1, bc2; };
template <bool INDEPENDENT>
__device__ __forceinline__ void adamw_tiles(const pylo_adam_item* __restrict__ items, const pylo_tile* __restrict__ tiles, int n_tiles, const Adam& q,
                                            const pylo_step_params& prm, int block, int blocks) {
  const float beta1 = q.beta1, omb1 = q.omb1, beta2 = q.beta2, omb2 = q.omb2, eps = q.eps, bc1_all = q.bc1, bc2_all = q.bc2;
  constexpr int NM = INDEPENDENT ? 1 : 3;
  for (int t = block; t < n_tiles; t += blocks) {
    const pylo_tile tl = tiles[t];
    const pylo_adam_item& it = items[tl.tensor];
    const int64_t n = it.n;
    const int cnt = tile_count(tl, n);
    float gs = 1.0f;
    if (it.clip_norm > 0.f && prm.gnorm_sq) {
      const float denom = fmaxf(sqrtf(*prm.gnorm_sq), it.clip_norm);
      gs = denom > 0.f ? it.clip_norm / denom : 1.0f;
    }
    const float bc1 = bc1_all > 0.f ? bc1_all : it.bc1, bc2 = bc1_all > 0.f ? bc2_all : it.bc2;
    const float lr = it.lr, wd = it.wd;
    const float* __restrict__ gp = it.g + tl.start;
    float* __restrict__ pp = it.p + tl.start;
    float* __restrict__ vp = it.v + tl.start;
    float* __restrict__ mp = it.m + tl.start;
    auto element = [&](float g, float& p, float& v, float (&m)[NM]) {
      g = xform_grad(g, gs, prm.clip_val, prm.nan_to_num);
      if (INDEPENDENT) {  // exp_avg.mul_(b1).add_(g, alpha=1-b1); exp_avg_sq.mul_(b2).addcmul_(g, g, value=1-b2)
        m[0] = fmaf(g, omb1, m[0] * beta1);
        v = fmaf(g * g, omb2, v * beta2);
      } else {  // shared accumulators: all three momenta advance, the step uses decay 0
#pragma unroll
        for (int k = 0; k < NM; ++k) m[k] = lerp_torch(m[k], g, prm.w_m[k]);
        v = lerp_torch(v, g * g, prm.w_v);
      }
      const float upd = (m[0] / bc1) / (sqrtf(v / bc2) + eps);
      p = fmaf(-lr, fmaf(wd, p, upd), p);
    };
    const bool al = ((((uintptr_t)gp | (uintptr_t)pp | (uintptr_t)vp | (uintptr_t)mp) & 15) == 0) && (INDEPENDENT || (n & 3) == 0);
    const int c4 = al ? (cnt & ~3) : 0;
#pragma unroll 2
    for (int i = threadIdx.x * 4; i < c4; i += NT * 4) {
      const float4 g4 = ldg4(gp + i), p4 = ld4(pp + i), v4 = ld4(vp + i);
      float4 m4[NM];
#pragma unroll
      for (int k = 0; k < NM; ++k) m4[k] = ld4(mp + k * n + i);
      float g[4] = {g4.x, g4.y, g4.z, g4.w}, p[4] = {p4.x, p4.y, p4.z, p4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w}, m[4][NM];
#pragma unroll
      for (int k = 0; k < NM; ++k) { m[0][k] = m4[k].x; m[1][k] = m4[k].y; m[2][k] = m4[k].z; m[3][k] = m4[k].w; }
#pragma unroll
      for (int u = 0; u < 4; ++u) element(g[u], p[u], v[u], m[u]);
      st4(pp + i, make_float4(p[0], p[1], p[2], p[3]));
      st4(vp + i, make_float4(v[0], v[1], v[2], v[3]));
#pragma unroll
      for (int k = 0; k < NM; ++k) st4(mp + k * n + i, make_float4(m[0][k], m[1][k], m[2][k], m[3][k]));
    }
    for (int i = c4 + threadIdx.x; i < cnt; i += NT) {
      float p = pp[i], v = vp[i], m[NM];
#pragma unroll
      for (int k = 0; k < NM; ++k) m[k] = mp[k * n + i];
      element(gp[i], p, v, m);
      pp[i] = p;
      vp[i] = v;
#pragma unroll
      for (int k = 0; k < NM; ++k) mp[k * n + i] = m[k];
    }
  }
}
template <bool INDEPENDENT>
__global__ void __launch_bounds__(NT) k_adamw(const pylo_adam_item* __restrict__ items, const pylo_tile* __restrict__ tiles, int n_tiles, const Adam q,
                                              const pylo_step_params prm) {
  pdl_begin();
  adamw_tiles<INDEPENDENT>(items, tiles, n_tiles, q, prm, blockIdx.x, gridDim.x);
}
// A small model's last two launches in one (neither reads what the other writes): the first n_post_ctas CTAs take the matrices' tiles.
// Perceptron, us per step: 101.2 -> 98.5.
template <bool INDEPENDENT>
__global__ void __launch_bounds__(NT) k_post_adamw(const pylo_post_item* __restrict__ post, const pylo_tile* __restrict__ post_tiles, int n_post, int n_post_ctas,
                                                   const int* __restrict__ status, int* __restrict__ host_status,
                                                   const pylo_adam_item* __restrict__ items, const pylo_tile* __restrict__ tiles, int n_tiles, const Adam q,
                                                   const pylo_step_params prm) {
  pdl_begin();
  if ((int)blockIdx.x < n_post_ctas) post_apply_tiles(post, post_tiles, n_post, reported(status), host_status, blockIdx.x, n_post_ctas);
  else adamw_tiles<INDEPENDENT>(items, tiles, n_tiles, q, prm, blockIdx.x - n_post_ctas, gridDim.x - n_post_ctas);
}

// ================================================================================================
// VeLO front end
// ================================================================================================
__device__ __forceinline__ float clip_log_abs10(float v) {
  return fminf(fmaxf(logf(1e-8f + fabsf(v * 10.0f)), -5.f), 5.f) * 0.5f;
}

// BufferLossAccumulators.update followed by .features (velo_cuda.py:183-211); one warp.  loss9 (may be shared memory, may be
// NULL) gets the features, the buffer is advanced where `write` says so.
__device__ __forceinline__ void velo_loss_update(const pylo_velo_loss& b, float* loss9, bool write) {
  __shared__ float s_cor[10];
  const int j = threadIdx.x & 31;
  const int it = *b.iteration;
  const float loss_in = b.loss ? b.loss[0] : b.value;
  float cor = -CUDART_INF_F;
  if (j < 10) cor = b.means[j] / (1.0f - powf(b.decays[j], (float)(it + 1)));
  float mx = cor;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float approx_max = it == 0 ? loss_in : mx;
  const float loss = fminf(fabsf(approx_max) * 2.0f, loss_in);
  float rmin = 0.f;
  if (j < 10) {
    const float dj = b.decays[j];
    const float mnew = b.means[j] * dj + loss * (1.0f - dj);
    const float c2 = mnew / (1.0f - powf(dj, (float)(it + 1)));  // features() uses iteration after the increment
    rmin = fminf(b.running_min[j], c2);
    if (write) {
      b.means[j] = mnew;
      b.running_min[j] = rmin;
    }
    s_cor[j] = c2;
  }
  __syncwarp();
  if (loss9 && j < 9) {
    const float den = fmaxf(1e-8f, s_cor[j + 1] - rmin);
    float f = fminf(fmaxf((s_cor[j] - rmin) / den - 1.0f, -1.f), 1.f);
    loss9[j] = (it + 1 <= 2) ? f * 0.f : f;
  }
  __syncwarp();
  if (write && j == 0) *b.iteration = it + 1;
}

__global__ void k_velo_loss(const pylo_velo_loss b, float* __restrict__ loss9) {
  pdl_begin();
  velo_loss_update(b, loss9, true);
}

// Entry `lane` (< 30) of a tensor's LSTM inputs from its sums (s_sum, 40 of them) and the loss features.
__device__ __forceinline__ float velo_feature(int lane, const pylo_tensor_desc& d, const double* s_sum, const float* s_loss9, const float* rank_onehot,
                                              float fraction) {
  const double n = (double)d.n;
  // as the stored sums have them: 32 bits, the VeLO statistics 32 + 32
  auto stat = [&](int j) { const float hi = (float)s_sum[30 + j]; return (double)hi + (double)(float)(s_sum[30 + j] - (double)hi); };
  const float mean_p2 = (float)((double)(float)s_sum[2] / n);
  const double norm = (double)rsqrtf(fmaxf(mean_p2, 1e-9f));
  const double mean_v = stat(6) / n, e_v2 = stat(7) / n;
  float o = 0.f;
  if (lane < 9) {  // tanh((x - t) * 10) (velo_cuda.py:155-162)
    const float at[9] = {0.03f, 0.1f, 0.2f, 0.4f, 0.6f, 0.8f, 0.9f, 1.0f, 1.1f};
#pragma unroll
    for (int j = 0; j < 9; ++j) if (lane == j) o = tanhf((fraction - at[j]) * 10.0f);
  }
  else if (lane < 18) o = s_loss9[lane - 9];
  else if (lane == 18) o = clip_log_abs10((float)(norm * mean_v));
  else if (lane < 24) o = rank_onehot[lane - 19];
  else if (lane < 30) {
    const int k = (lane - 24) % 3;
    const double mu = stat(k) / n, e_m2 = stat(3 + k) / n;
    const double var = lane < 27 ? fmax(e_m2 - mu * mu, 0.0)
                                : fmax(e_v2 - 2.0 * mu * mean_v + mu * mu, 0.0);  // mean((rms - mean_m)^2), velo_cuda.py:243
    o = clip_log_abs10((float)(norm * norm * var));
  }
  return o;
}

// The 30 LSTM inputs of a tensor from the statistics gathered in phase B (velo_cuda.py:213-252).  One CTA per tensor, which
// first does phase B2 for it (a launch less), while its last warp works out the loss features: every CTA for itself and
// without advancing the loss buffer, which is left to a kernel that runs when all of them are done (k_velo_xmix).
template <int ROWS>
__global__ void __launch_bounds__(ROWS * PYLO_STAT_STRIDE + 32) k_velo_tensor_features(const pylo_tensor_desc* __restrict__ descs,
                                       const int32_t* __restrict__ layer_of, int T,
                                       const float* __restrict__ rank_onehot, float fraction,
                                       const pylo_velo_loss lossbuf, float* __restrict__ x_in) {
  pdl_begin();
  __shared__ double s_d[ROWS][PYLO_STAT_STRIDE];
  __shared__ double s_sum[PYLO_STAT_STRIDE];
  __shared__ float s_loss9[9];
  const int t = blockIdx.x, tid = threadIdx.x;
  const pylo_tensor_desc& d = descs[t];
  if (tid >= ROWS * PYLO_STAT_STRIDE) velo_loss_update(lossbuf, s_loss9, false);
  const double tot = unit_sum<ROWS>(d, s_d);
  if (tid < PYLO_STAT_STRIDE) {
    store_unit_sum(d, tot);
    s_sum[tid] = tot;
  }
  __syncthreads();
  if (tid >= 32) return;
  const int layer = layer_of ? layer_of[t] : t;  // position of this tensor among all T tensors of the model
  const float o = velo_feature(tid, d, s_sum, s_loss9, rank_onehot + t * 5, fraction);
  if (tid < 30) x_in[(int64_t)(T - 1 - layer) * 30 + tid] = o;  // rows are flipped (velo_cuda.py:422)
}

// x' = final_mix(x) + max_t relu(mix2(x)).  One warp per hidden unit, lanes along the tensors (one thread per unit walked
// through all tensors by itself: 203 us at 292 tensors).
__global__ void __launch_bounds__(NT) k_velo_xmix(const pylo_velo_rnn r, const pylo_velo_loss lossbuf) {
  pdl_begin();
  if (lossbuf.means && blockIdx.x == 0 && threadIdx.x < 32) velo_loss_update(lossbuf, nullptr, !reported(r.status));
  const int h = blockIdx.x * NWARP + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= r.H) return;
  float best = 0.f;   // relu
  const float b2 = r.mix2_b[h], bf = r.fmix_b[h];
  const float2* __restrict__ w2 = reinterpret_cast<const float2*>(r.mix2_w + h * 30);
  const float2* __restrict__ wf = reinterpret_cast<const float2*>(r.fmix_w + h * 30);
  for (int t = lane; t < r.T; t += 32) {
    const float2* __restrict__ x = reinterpret_cast<const float2*>(r.x_in + t * 30);
    float m = b2, f = bf;
#pragma unroll
    for (int k = 0; k < 15; ++k) {
      const float2 v = x[k], a = w2[k], c = wf[k];
      m = fmaf(a.y, v.y, fmaf(a.x, v.x, m));
      f = fmaf(c.y, v.y, fmaf(c.x, v.x, f));
    }
    best = fmaxf(best, m);
    r.xmix[(int64_t)t * r.H + h] = f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  for (int t = lane; t < r.T; t += 32) r.xmix[(int64_t)t * r.H + h] += best;
}

// The two above in one launch for small models (up to VI_TENSORS tensors, best of up to VI_TILES tiles): every CTA makes all tensors' inputs for itself,
// from sums in the order of unit_sum, and its eight hidden units' x'.  The loss buffer, which all CTAs read here, is written by
// k_velo_lstm.  Latency-bound; in place of two launches: perceptron, us per step 44.4 -> 42.2.
#define VI_TENSORS 16
#define VI_TILES 16
__global__ void __launch_bounds__(NT) k_velo_inputs(const pylo_tensor_desc* __restrict__ descs, const int32_t* __restrict__ layer_of,
                                                    const float* __restrict__ rank_onehot, float fraction, const pylo_velo_loss lossbuf,
                                                    const pylo_velo_rnn r) {
  pdl_begin();
  __shared__ double s_sum[VI_TENSORS][PYLO_STAT_STRIDE];
  __shared__ float s_x[VI_TENSORS][31], s_loss9[9];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j = tid % PYLO_STAT_STRIDE, T = r.T;
  const int h = blockIdx.x * NWARP + warp;
  const bool unit = h < r.H;
  const float w2 = unit && lane < 30 ? __ldg(r.mix2_w + h * 30 + lane) : 0.f, wf = unit && lane < 30 ? __ldg(r.fmix_w + h * 30 + lane) : 0.f;
  const float b2 = unit ? __ldg(r.mix2_b + h) : 0.f, bf = unit ? __ldg(r.fmix_b + h) : 0.f;
  if (tid < 5 * PYLO_STAT_STRIDE) {
    for (int t = tid / PYLO_STAT_STRIDE; t < T; t += 5) {
      const pylo_tensor_desc& d = descs[t];
      const float* __restrict__ src = d.tile_part + j;
      const int n = d.n_tiles;
      float v[VI_TILES];
#pragma unroll
      for (int q = 0; q < VI_TILES; ++q) v[q] = q < n ? src[q * PYLO_STAT_STRIDE] : 0.f;
      double tot = 0.0;
#pragma unroll
      for (int q = 0; q < VI_TILES; ++q) tot += (double)v[q];
#pragma unroll 1
      for (int q = VI_TILES; q < n; ++q) tot += (double)src[(int64_t)q * PYLO_STAT_STRIDE];   // none in the plans of small models
      tot += (double)d.closed[j];
      s_sum[t][j] = tot;
      if (blockIdx.x == 0) store_unit_sum(d, tot, j);
    }
  } else if (warp == NWARP - 1) {
    velo_loss_update(lossbuf, s_loss9, false);
  }
  __syncthreads();
  for (int t = warp; t < T; t += NWARP) {
    const int row = T - 1 - (layer_of ? layer_of[t] : t);  // rows are flipped (velo_cuda.py:422)
    const float o = velo_feature(lane, descs[t], s_sum[t], s_loss9, rank_onehot + t * 5, fraction);
    if (lane < 30) {
      s_x[row][lane] = o;
      if (blockIdx.x == 0) r.x_in[row * 30 + lane] = o;
    }
  }
  __syncthreads();
  float m = b2, f = bf;
  const float* x = s_x[lane < T ? lane : 0];   // a lane per tensor
#pragma unroll
  for (int k = 0; k < 30; ++k) {
    const float v = x[k];
    m = fmaf(__shfl_sync(0xffffffffu, w2, k), v, m);
    f = fmaf(__shfl_sync(0xffffffffu, wf, k), v, f);
  }
  float best = lane < T ? fmaxf(m, 0.f) : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if (unit && lane < T) r.xmix[(int64_t)lane * r.H + h] = f + best;
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }
// cell update of one hidden unit; gate order i, g, f, o with f + 1 (VeLO_RNN.py:57-65)
__device__ __forceinline__ float velo_cell(float i, float g, float f, float o, float& c) {
  c = sigmoidf_(f + 1.0f) * c + sigmoidf_(i) * tanhf(g);
  return sigmoidf_(o) * tanhf(c);
}

// The LSTM's gates, gates[t][q] = lstm_b[q] + sum_k lstm_w[q][k] * cat(x', h)[t][k], a [T x 2H] x [2H x 4H] product, fp32
// throughout, and its cell.
//
// For few tensors it is a read of the 8.4 MB of weights, for a few hundred ~0.6 G FMAs.  A warp keeps the four weight rows of a
// hidden unit (one half of their columns: those that meet x', or those that meet h) in registers and takes eight tensors at a time
// from shared memory: 512 FMAs per lane on 32 shared-memory reads, then the 32 sums are reduced over the lanes together, 31
// shuffles in all, and lane l ends with the sum of tensor l / 4 and gate l % 4.  The other half's sums come from the warp beside
// it, the four gates of a tensor from the lanes beside.  512 hidden units, the gates alone: 6 tensors 3.6 us, 292 tensors 46, in the
// tiled kernel below, which is for hidden sizes that are not multiples of 128 or above 512, 68.6 and 124; with the cell, which
// would be another launch of 2.8, 6.7 and 57 as launches by themselves under the profiler.  Other CTAs still read h: the new one is
// left in `gates` ([T][H]), k_velo_mix takes it over.
#define GR_UNITS 4   // hidden units per CTA: one per pair of warps
template <int NI>    // float4 per lane and row: H = 128 * NI
__global__ void __launch_bounds__(NT, 2) k_velo_lstm(const pylo_velo_rnn r, const pylo_velo_loss lossbuf, int groups_per_cta) {
  pdl_begin();
  extern __shared__ __align__(16) float s_x[];   // [2][8][2H]
  __shared__ float s_half[GR_UNITS][32];
  constexpr int H = 128 * NI;
  const int tid = threadIdx.x, lane = tid & 31, half = (tid >> 5) & 1, unit = tid >> 6, h = blockIdx.x * GR_UNITS + unit;
  const int word = reported(r.status);
  if (lossbuf.means && blockIdx.x == 0 && blockIdx.y == 0 && tid < 32) velo_loss_update(lossbuf, nullptr, !word);   // behind k_velo_inputs
  const int groups = (r.T + 7) / 8, g0 = blockIdx.y * groups_per_cta, g1 = min(g0 + groups_per_cta, groups);
  auto stage = [&](int g) {
    float* dst = s_x + (g & 1) * 16 * H;
    for (int e = tid; e < 8 * 2 * (H / 4); e += NT) {
      const int c = e % (H / 2), t = g * 8 + e / (H / 2);   // 2H / 4 pieces per tensor
      const float* src = c < H / 4 ? r.xmix + (int64_t)t * H + 4 * c : r.h + (int64_t)t * H + 4 * (c - H / 4);
      const uint32_t bytes = t < r.T ? 16 : 0;              // past the last tensor: zeros
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst + 4 * e)), "l"(t < r.T ? src : r.xmix), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (g0 < g1) stage(g0);
  float4 w[4][NI];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int i = 0; i < NI; ++i) w[u][i] = ldg4(r.lstm_w + (int64_t)(u * H + h) * 2 * H + half * H + (i * 32 + lane) * 4);
  const float bias = r.lstm_b[(lane & 3) * H + h];
  for (int g = g0; g < g1; ++g) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this group has arrived, and the buffer of the next one is no longer read
    if (g + 1 < g1) stage(g + 1);
    const int t = g * 8 + (lane >> 2);
    const float c_old = !half && t < r.T ? r.c[(int64_t)t * H + h] : 0.f;
    const float* x = s_x + (g & 1) * 16 * H + half * H + lane * 4;
    float acc[32];     // tensor * 4 + gate
#pragma unroll
    for (int t = 0; t < 8; ++t) {
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[t * 4 + u] = 0.f;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const float4 v = ld4(x + t * 2 * H + i * 128);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          acc[t * 4 + u] = fmaf(w[u][i].w, v.w, fmaf(w[u][i].z, v.z, fmaf(w[u][i].y, v.y, fmaf(w[u][i].x, v.x, acc[t * 4 + u]))));
      }
    }
    const float sum = warp_fold<0, 32>(acc);
    if (half) s_half[unit][lane] = sum;
    __syncthreads();
    if (!half) {
      const float gate = (sum + bias) + s_half[unit][lane];
      const int first = lane & ~3;
      const float gi = __shfl_sync(0xffffffffu, gate, first), gg = __shfl_sync(0xffffffffu, gate, first + 1),
                  gf = __shfl_sync(0xffffffffu, gate, first + 2), go = __shfl_sync(0xffffffffu, gate, first + 3);
      if ((lane & 3) == 0 && t < r.T && !word) {
        float c = c_old;
        r.gates[(int64_t)t * H + h] = velo_cell(gi, gg, gf, go, c);
        r.c[(int64_t)t * H + h] = c;
      }
    }
  }
}

// Shared-memory tiled, 64 x 64 outputs per CTA, 16 deep, 4 x 4 outputs per thread.
#define GT 64
#define GK 16
__global__ void __launch_bounds__(NT) k_velo_gates(const pylo_velo_rnn r) {
  pdl_begin();
  __shared__ float s_a[GK][GT + 4];
  __shared__ float s_w[GK][GT + 4];
  const int H = r.H, Q = 4 * H, K = 2 * H, T = r.T;
  const int t0 = blockIdx.y * GT, q0 = blockIdx.x * GT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 x 16 threads
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += GK) {
    // each thread loads 4 elements of each operand tile: rows (threadIdx.x / 16 + 16 * u), column threadIdx.x % 16
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int row = ty + 16 * u, kk = k0 + tx;
      const int t = t0 + row, q = q0 + row;
      float av = 0.f, wv = 0.f;
      if (t < T && kk < K) av = kk < H ? r.xmix[(int64_t)t * H + kk] : r.h[(int64_t)t * H + (kk - H)];
      if (q < Q && kk < K) wv = r.lstm_w[(int64_t)q * K + kk];
      s_a[tx][row] = av;
      s_w[tx][row] = wv;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      const float4 a = ld4(&s_a[kk][ty * 4]);
      const float4 w = ld4(&s_w[kk][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = t0 + ty * 4 + i;
    if (t >= T) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = q0 + tx * 4 + j;
      if (q < Q) r.gates[(int64_t)t * Q + q] = acc[i][j] + r.lstm_b[q];
    }
  }
}

// the cell behind k_velo_gates
__global__ void k_velo_cell(const pylo_velo_rnn r) {
  pdl_begin();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)r.T * r.H) return;
  const int word = reported(r.status);
  const int t = (int)(e / r.H), h = (int)(e % r.H), H = r.H;
  const float* g4 = r.gates + (int64_t)t * 4 * H + h;
  float c = r.c[e];
  const float hn = velo_cell(g4[0], g4[H], g4[2 * H], g4[3 * H], c);
  if (word) return;
  r.c[e] = c;
  r.h[e] = hn;
}

// controls[t][b] and lr_mult[t]; one warp per output
// h: r.h, or where k_velo_lstm has left the new one
__global__ void __launch_bounds__(NT) k_velo_heads(const pylo_velo_rnn r, const float* __restrict__ h) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int64_t wid = (int64_t)blockIdx.x * NWARP + (threadIdx.x >> 5);
  const int H = r.H, B1 = r.B + 1;
  if (wid >= (int64_t)r.T * B1) return;
  const int t = (int)(wid / B1), b = (int)(wid % B1);
  const float* wrow = b < r.B ? r.ctrl_w + (int64_t)b * H : r.step_w;
  float acc = 0.f;
  for (int k = lane; k < H; k += 32) acc = fmaf(wrow[k], h[(int64_t)t * H + k], acc);
  acc = warp_sum(acc);
  if (lane == 0) {
    if (b < r.B) r.controls[(int64_t)t * r.B + b] = acc + r.ctrl_b[b];
    else r.lr_mult[r.T - 1 - t] = acc + r.step_b[0];  // row t of the flipped input belongs to tensor T-1-t
  }
}

// weights[tensor][e] = mean_b(control[b] * bank[b][e]) * 100 (VeLO_MLP.py:92-126).  Latency-bound: a block takes a quarter of a
// tensor's 159 weights and deals the bank to sixteen groups of threads, whose sixteen reads of the usual bank are in flight
// together (a block per tensor and four groups, eight reads at a time: 7.3 us, now 3.5; as one launch with the heads, a cluster per tensor, the two took 12.5 instead of 7.4).
#define MIX_GROUPS 16
#define MIX_OUT 40
__global__ void __launch_bounds__(MIX_OUT * MIX_GROUPS) k_velo_mix(const pylo_velo_rnn r, const float* __restrict__ h_new) {
  pdl_begin();
  if (h_new != r.h && !reported(r.status)) {   // nobody reads the old h any more
    for (int k = blockIdx.y * blockDim.x + threadIdx.x; k < r.H; k += gridDim.y * blockDim.x) r.h[(int64_t)blockIdx.x * r.H + k] = h_new[(int64_t)blockIdx.x * r.H + k];
  }
  extern __shared__ float s_ctrl[];
  __shared__ float s_part[MIX_GROUPS][MIX_OUT];
  const int tensor = blockIdx.x, row = r.T - 1 - tensor;
  for (int b = threadIdx.x; b < r.B; b += blockDim.x) s_ctrl[b] = r.controls[(int64_t)row * r.B + b];
  __syncthreads();
  const int c = threadIdx.x % MIX_OUT, e = blockIdx.y * MIX_OUT + c, grp = threadIdx.x / MIX_OUT;
  float acc = 0.f;
  if (e < 159) {
#pragma unroll 16
    for (int b = grp; b < r.B; b += MIX_GROUPS) acc = fmaf(s_ctrl[b], __ldg(r.bank + (int64_t)b * 159 + e), acc);
  }
  s_part[grp][c] = acc;
  __syncthreads();
  if (threadIdx.x < MIX_OUT && e < 159) {
    acc = 0.f;
#pragma unroll
    for (int q = 0; q < MIX_GROUPS; ++q) acc += s_part[q][c];
    r.weights[(int64_t)tensor * 160 + e] = acc / (float)r.B * 100.0f;
  }
}

// ================================================================================================
// C ABI
// ================================================================================================
// Opt-in limits and caches are kept per device: the library may be used on every GPU of a box from one process.
#define PYLO_MAX_DEVICES 64
static int g_sm_count[PYLO_MAX_DEVICES] = {0};
static int sm_count() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PYLO_MAX_DEVICES) return 148;
  if (g_sm_count[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    g_sm_count[dev] = n > 0 ? n : 148;
  }
  return g_sm_count[dev];
}
static int grid_for(int n_items, int ctas_per_sm) {
  const int cap = sm_count() * ctas_per_sm;
  return n_items < cap ? n_items : cap;
}
static int launch_status() { return (int)cudaGetLastError(); }

// Every kernel of this library is launched so that it may become resident while its predecessor in the stream drains
// (programmatic dependent launch) and waits in pdl_begin() until that one is complete.  A step is a chain of small launches;
// on a small model the gaps between them are as long as the kernels (AdafacLO over a 118 K MLP: 47.5 -> 38.8 us per step).
// On large ones there is nothing to gain (GPT-2-medium shapes: 0.7 % slower with it), so a step of more than 134 M elements
// launches plainly: PlainLaunches says so for the calls of one scope on one host thread.
static thread_local bool t_plain_launches = false;
struct PlainLaunches {
  bool before;
  explicit PlainLaunches(int n_tiles) : before(t_plain_launches) { t_plain_launches = before || n_tiles > 8192; }
  ~PlainLaunches() { t_plain_launches = before; }
};
// The SMs' memory is split between L1 cache and shared memory anew only when they are idle, which programmatic launches never
// let them be: the kernels after one with a large share of shared memory would run with what L1 it left (the apply sweep of
// 6 x 4096 x 4096 VeLO parameters: 921 us after the state sweep's ring, 755 us without).  Such a kernel has itself and the next
// launch of its thread made plainly.
static thread_local bool t_plain_next = false;
template <class... P, class... A>
static void launch_clusters(void (*kernel)(P...), dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (!t_plain_launches && !t_plain_next) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  t_plain_next = false;
  if (cluster >= 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
static void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  launch_clusters(kernel, grid, block, 0, smem, stream, static_cast<A&&>(args)...);
}

// Opt a kernel in to more than 48 KB of dynamic shared memory, once per device (the attribute belongs to the
// device's copy of the function); flags[] is the caller's per-kernel record.
template <class K>
static int allow_dynamic_smem(K kernel, int bytes, bool (&flags)[PYLO_MAX_DEVICES]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < PYLO_MAX_DEVICES && flags[dev]) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < PYLO_MAX_DEVICES) flags[dev] = true;
  return 0;
}

// The same for clusters of more than eight CTAs.
template <class K>
static int allow_wide_clusters(K kernel, bool (&flags)[PYLO_MAX_DEVICES]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < PYLO_MAX_DEVICES && flags[dev]) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < PYLO_MAX_DEVICES) flags[dev] = true;
  return 0;
}

#define CHECK_ARG(cond) \
  do {                  \
    if (!(cond)) return -1; \
  } while (0)

template <int BM, int BN>
static long long ns_deal(nf_group& grp) {
  long long tiles = 0;
  for (int k = 0; k < grp.n; ++k) {
    nf_args& g = grp.p[k].g;
    g.per = nf_tiles_per_matrix<BM, BN>(g.M, g.N, g.symmetric);
    g.tile0 = (int)tiles;
    tiles += (long long)g.per * g.batch;
  }
  grp.tiles = (int)tiles;
  return tiles;
}
template <class Smem, void (*kernel)(nf_group, int*)>
static int ns_launch(nf_group& grp, int ctas, int* status, cudaStream_t s, int cluster = 0) {
  static bool configured[PYLO_MAX_DEVICES] = {};
  constexpr int smem = (int)sizeof(Smem) + 1024;  // room to start the stages on a 1024-byte boundary
  if (int rc = allow_dynamic_smem(kernel, smem, configured)) return rc;
  launch_clusters(kernel, ctas, NF_THREADS, cluster, smem, s, grp, status);
  return launch_status();
}
// The tile by what fills the GPU: a launch is as long as the SM with the most tiles, and a pair's tile of 256 x 256 is worth it
// from about one per pair of SMs on; below, tiles of 128 x 128 on single SMs, the longest contractions split.
static int ns_gemm(nf_group& grp, int* status, cudaStream_t s) {
  const int sms = sm_count();
  long long tiles = ns_deal<256, 256>(grp);
  if (tiles > 0x3fffffff) return -1;
  if (tiles * 8 >= sms / 2 * 7) {
    const int ctas = (int)(2 * tiles < sms ? 2 * tiles : sms & ~1);
    return ns_launch<NfSmem<256, true>, k_gemm_f16x2_pair>(grp, ctas, status, s);
  }
  tiles = ns_deal<NF_BM, 128>(grp);
  // An SM fetches a K block of 64 in half a microsecond or more, so a few tiles with a long contraction are shared by clusters
  // of CTAs: from eight blocks each on (below, bringing the sums together costs what is gained: 197 x 768, 12 blocks, 171 us
  // per chain unsplit, 174 in two), as far as three quarters of the SMs go (1001 x 1433 in 36 clusters of four found no room
  // for all of them at once: 342 -> 446).  768 x 2304: 308 -> 259 us; 128 x 3000 (now k_ns_cluster's): 293 -> 194.
  int blocks = 0, split = 1;
  for (int k = 0; k < grp.n; ++k) blocks = max(blocks, (grp.p[k].g.K + NF_BK - 1) / NF_BK);
  while (split < 8 && blocks >= 16 * split && tiles * 2 * split <= sms * 3 / 4) split *= 2;
  if (split > 1) return ns_launch<NfSmem<128, false>, k_gemm_f16x2_split>(grp, (int)tiles * split, status, s, split);
  return ns_launch<NfSmem<128, false>, k_gemm_f16x2>(grp, (int)(tiles < sms ? tiles : sms), status, s);
}

template <int FAM>
static void factor_update_launch(const pylo_tensor_desc* descs, const int32_t* mats, int n, int threads, const pylo_step_params& prm, cudaStream_t s) {
  if (threads == A2_NT) launch(k_factor_update<FAM, A2_NT>, n * A2_CL, A2_NT, 0, s, descs, mats, prm);
  else launch(k_factor_update<FAM, A2_NT / 2>, n * A2_CL, A2_NT / 2, 0, s, descs, mats, prm);
}

template <int FAM>
static int state_moments_launch(const pylo_tensor_desc* descs, const pylo_tile* tiles, int n_tiles, int reverse,
                                const pylo_step_params& prm, cudaStream_t s) {
  if (!prm.bulk_copies) {
    launch(k_state_moments<FAM, false>, grid_for(n_tiles, 4), NT, 0, s, descs, tiles, n_tiles, reverse, prm);
    return 0;
  }
  static bool configured[PYLO_MAX_DEVICES] = {};
  if (int rc = allow_dynamic_smem(k_state_moments<FAM, true>, (int)sizeof(PipeSmem), configured)) return rc;
  t_plain_next = true;
  launch(k_state_moments<FAM, true>, grid_for(n_tiles, 2), NT, sizeof(PipeSmem), s, descs, tiles, n_tiles, reverse, prm);
  t_plain_next = true;
  return 0;
}

static long long ns_small_floats(int rows, int cols) {
  const long long r = rows < cols ? rows : cols, c = rows < cols ? cols : rows;
  return 2 * r * (c + 1) + 2 * r * (r + 1);
}
// One CTA does about 1e5 FMAs per microsecond: beyond a few million, or where it does not fit into shared memory, the
// tensor-core chain (15 launches of 4 us at least) is faster.
static bool ns_is_small(int rows, int cols, int iters) {
  const long long r = rows < cols ? rows : cols, c = rows < cols ? cols : rows;
  return r <= 64 && iters * (2 * r * r * c + r * r * r) <= 3000000 && ns_small_floats(rows, cols) * 4 <= 200 * 1024;
}

// How a stack is run: 0, by single CTAs in plain fp32; 1 to 16, by so many CTAs a matrix (k_ns_cluster); -1, as a chain of
// launches.  Alone, what fits clusters is faster there for any number of matrices (us per chain, launches / clusters, two of each run
// within 1 %: 128 x 784 155 / 64, 128 x 3072 184 / 83, 24 x 128 x 1000 288 / 140, 48 x 128 x 1000 413 / 280, 400 x 128 x 128
// 833 / 120, 300 x 64 x 256 642 / 205), with as few CTAs a matrix as hold it (48 matrices of 128 x 128 to 128 x 512, with
// up to 192 columns per CTA 73, with 128 125).
static int ns_parts(int rows, int cols, int iters) {
  if (ns_is_small(rows, cols, iters)) return 0;
  const int r = rows < cols ? rows : cols, c = rows < cols ? cols : rows;
  if (r > NC_SIDE || c > 16 * NC_COLS) return -1;
  int parts = 1;
  while ((c + parts - 1) / parts > NC_COLS) parts *= 2;
  return parts;
}
struct NsWork {   // byte offsets into the workspace, every buffer on a 1024-byte boundary
  int64_t xp[2], ap, bp, a, x, part, inv, total;
  int r, c, ldx, lda_p, lda, slices;
};
static NsWork ns_work(int rows, int cols, int batch) {
  NsWork w = {};
  w.r = rows < cols ? rows : cols;
  w.c = rows < cols ? cols : rows;
  w.ldx = (cols + 7) / 8 * 8;
  w.lda_p = (w.r + 7) / 8 * 8;
  w.lda = (w.r + 3) / 4 * 4;
  const int64_t n = (int64_t)rows * cols;
  w.slices = (int)((n + NF_SLICE - 1) / NF_SLICE);
  int64_t at = 0;
  auto take = [&](int64_t bytes) { const int64_t o = at; at += (bytes + 1023) / 1024 * 1024; return o; };
  const int64_t planes_x = (int64_t)batch * rows * w.ldx * 4, planes_a = (int64_t)batch * w.r * w.lda_p * 4;
  w.xp[0] = take(planes_x);
  w.xp[1] = take(planes_x);
  w.ap = take(planes_a);
  w.bp = take(planes_a);
  w.a = take((int64_t)batch * w.r * w.lda * 4);
  w.x = take((int64_t)batch * n * 4);
  w.part = take((int64_t)batch * w.slices * 4);
  w.inv = take((int64_t)batch * 4);
  w.total = at;
  return w;
}

// Where a stack goes: the chain of launches, the launch of clusters, or a launch of single CTAs of its own.
enum NsRoute { NS_CHAIN, NS_CLUSTERS, NS_SINGLE };
struct NsRoutes {
  bool chain = false, clusters = false;   // whether a stack needs the chain; whether there is a launch of clusters
  long long fitting = 0;                  // matrices that would fit clusters
  NsRoutes(const pylo_ns_desc* descs, int n) {
    for (int k = 0; k < n; ++k) {
      const int parts = ns_parts(descs[k].rows, descs[k].cols, descs[k].iters);
      chain |= parts < 0;
      if (parts > 0) fitting += descs[k].batch;
    }
    for (int k = 0; k < n; ++k) clusters |= by_size(descs[k]) == NS_CLUSTERS;
  }
  // Whether a stack goes with the chain: where it must, and beside larger ones also where it would fit clusters, as long as it is
  // no more than a few tiles in launches that are there anyway: a launch of clusters before them costs its own 40 to 80 us (us per
  // call, clusters first / riding: 512 x 512, 128 x 512, 1792 x 512 299 / 233; 512 x 784, 512 x 512, 100 x 512 285 / 219; 16 of
  // 768 rows and one 50 x 768 1245 / 1167; 256 x 256 and 48 of 128 x 128 186 / 152).  64 matrices make the symmetric products take
  // tiles of 256 x 256, three quarters of each for padding, and clusters are the better place (256 x 256 and 64 of 128 x 128 187 /
  // 247, of 128 x 512 284 / 318; 512 x 512 and 400 of 128 x 128 308 / 909).
  bool rides(int parts) const { return parts < 0 || (parts > 0 && chain && fitting < 64); }
  // What has no workspace for the chain and fits clusters stays there.
  NsRoute by_size(const pylo_ns_desc& d) const {
    const int parts = ns_parts(d.rows, d.cols, d.iters);
    if (parts == 0) return NS_SINGLE;
    if (parts < 0) return NS_CHAIN;
    return rides(parts) && d.work && ((uintptr_t)d.work & 255) == 0 && d.work_bytes >= ns_work(d.rows, d.cols, d.batch).total ? NS_CHAIN : NS_CLUSTERS;
  }
  // A launch of clusters takes a few small matrices along.
  NsRoute operator()(const pylo_ns_desc& d) const {
    const NsRoute to = by_size(d);
    return to == NS_SINGLE && clusters && d.batch <= 16 ? NS_CLUSTERS : to;
  }
};

// One launch: clusters as large as the most CTAs that share a matrix.
template <int COLS>
static int nc_launch(const nc_group& grp, int ctas, int cluster, int* status, cudaStream_t s) {
  static bool configured[PYLO_MAX_DEVICES] = {}, wide[PYLO_MAX_DEVICES] = {};
  constexpr int smem = (int)sizeof(NcSmem<COLS>) + 1024;   // room to start the boxes on a 1024-byte boundary
  if (int rc = allow_dynamic_smem(k_ns_cluster<COLS>, smem, configured)) return rc;
  if (cluster > 8)
    if (int rc = allow_wide_clusters(k_ns_cluster<COLS>, wide)) return rc;
  launch_clusters(k_ns_cluster<COLS>, ctas, NC_THREADS, cluster, smem, s, grp, status);
  return launch_status();
}
static int ns_clusters(nc_group& grp, int* status, cudaStream_t s) {
  int cluster = 1;
  for (int k = 0; k < grp.n; ++k) cluster = max(cluster, grp.p[k].parts);
  long long ctas = 0;
  bool wide = false;   // whether 128 columns per CTA (a register less in three: 64 instead of 69 us for 128 x 784) do not do
  for (int k = 0; k < grp.n; ++k) {
    nc_item& p = grp.p[k];
    const int c = max(p.rows, p.cols);
    p.cta0 = (int)ctas;
    ctas += ((long long)p.batch * max(1, p.parts) + cluster - 1) / cluster * cluster;
    wide |= p.parts ? (c + p.parts - 1) / p.parts > 128 : ns_small_floats(p.rows, p.cols) * 4 > (long long)offsetof(NcSmem<128>, red);
  }
  if (ctas > 0x7fffffff) return -1;
  return wide ? nc_launch<NC_COLS>(grp, (int)ctas, cluster, status, s) : nc_launch<128>(grp, (int)ctas, cluster, status, s);
}

template <int FAM>
static int small_front_launch(const pylo_tensor_desc* descs, int n, int cluster, const SfShape& q, int networks, const pylo_step_params& prm, cudaStream_t s) {
  static bool configured[PYLO_MAX_DEVICES] = {}, wide[PYLO_MAX_DEVICES] = {};
  if (int rc = allow_dynamic_smem(k_small_front<FAM>, PYLO_SMALL_FLOATS * 4, configured)) return rc;
  if (cluster > 8)
    if (int rc = allow_wide_clusters(k_small_front<FAM>, wide)) return rc;
  size_t smem = (size_t)sf_floats(q) * 4;
  if (networks && smem < sizeof(TcNet)) smem = sizeof(TcNet);
  launch_clusters(k_small_front<FAM>, (n + networks) * cluster, SF_NT, cluster, smem, s, descs, n, q, prm);
  return launch_status();
}

extern "C" {

int pylo_b200_abi_version(void) { return PYLO_B200_ABI_VERSION; }
int pylo_b200_sizeof_desc(void) { return (int)sizeof(pylo_tensor_desc); }
int pylo_b200_sizeof_params(void) { return (int)sizeof(pylo_step_params); }

int pylo_b200_workspace_layout(int family, int mode, int64_t n, int64_t La, int64_t Lb, int32_t X, int32_t Y,
                               pylo_ws_layout* out) {
  CHECK_ARG(out && n > 0);
  CHECK_ARG(family == PYLO_FAM_ADAFAC || family == PYLO_FAM_CELO2 || family == PYLO_FAM_VELO);
  CHECK_ARG(mode == PYLO_MODE_FAST2D || mode == PYLO_MODE_GENERIC || mode == PYLO_MODE_VEC1D || mode == PYLO_MODE_KERNEL);
  const int64_t H = family == PYLO_FAM_ADAFAC ? 32 : (family == PYLO_FAM_CELO2 ? 8 : 4);
  pylo_ws_layout w = {};
  if (mode != PYLO_MODE_VEC1D) {
    CHECK_ARG(La > 0 && Lb > 0);
    w.f_a = 3 * La; w.f_b = 3 * Lb; w.sum_a = La; w.sum_b = Lb;
  }
  if (mode == PYLO_MODE_GENERIC && X <= 0) {
    CHECK_ARG(n % Lb == 0);
    const int64_t rows = n / Lb;   // X
    // rows per strip of the column sums: one thread adds up a strip's rows, and 256 columns are one item
    w.rb = rows <= 512 ? 16 : (rows <= 2048 ? 32 : PYLO_A_ROWS_MAX);
    w.n_strips = (int32_t)((rows + w.rb - 1) / w.rb);
    w.part_b = w.n_strips * Lb;
  } else if (mode != PYLO_MODE_VEC1D) {
    const bool kernel = mode == PYLO_MODE_KERNEL;
    CHECK_ARG(X > 0 && Y > 0 && (La == X || (kernel && La % X == 0 && La / X <= 32)) && Lb == Y && (Y % 4 == 0 || mode == PYLO_MODE_GENERIC));
    // rows per strip: about X / 128, a multiple of 8, within [32, 128].  Up to 512 rows a tensor gives too few strips of
    // 32 to fill the GPU and the launch is all latency: strips of 8 (one or two rows per warp) there.
    int rb = (((X + 127) / 128 + 7) / 8) * 8;
    rb = X <= 512 ? 8 : (rb < 32 ? 32 : (rb > PYLO_A_ROWS_MAX ? PYLO_A_ROWS_MAX : rb));
    w.rb = rb;
    w.n_strips = (X + rb - 1) / rb;
    w.n_cb = (Y + PYLO_A_COLS - 1) / PYLO_A_COLS;
    w.part_a = kernel ? 2 * La * w.n_cb : (int64_t)X * w.n_cb;
    w.part_b = (int64_t)w.n_strips * Y;
    if (kernel) {
      w.fx = 4 * La;
    } else if (mode == PYLO_MODE_FAST2D || family != PYLO_FAM_ADAFAC) {   // what the tiled apply sweeps read
      w.fx = 4 * La;
      w.h_a = La * H * 2;
      w.h_b = Lb * H;
    }
  }
  w.closed = PYLO_STAT_STRIDE;
  w.n_tiles = (int32_t)((n + PYLO_TILE_ELEMS - 1) / PYLO_TILE_ELEMS);
  w.sums = SUMS_STRIDE;
  switch (family) {   // the tensor cores' operands are behind the network for ADAFAC alone; CELO2 has a unit per matrix, down to 3 x 3
    case PYLO_FAM_ADAFAC: w.wfold = PYLO_WFOLD_STRIDE; break;
    case PYLO_FAM_CELO2: w.wfold = Fold<PYLO_FAM_CELO2>::SN + Fam<PYLO_FAM_CELO2>::NF; break;
    default: w.wfold = Fold<PYLO_FAM_VELO>::SN + Fam<PYLO_FAM_VELO>::NF; break;
  }
  w.tile_part = (int64_t)w.n_tiles * PYLO_STAT_STRIDE;
  *out = w;
  return 0;
}

int64_t pylo_b200_workspace_bytes(const pylo_ws_layout* w, int tensor_part, int unit_part) {
  if (!w) return -1;
  auto pad = [](int64_t floats) { return (floats + 63) / 64 * 64 * 4; };
  int64_t bytes = 0;
  if (tensor_part)
    bytes += pad(w->f_a) + pad(w->f_b) + pad(w->sum_a) + pad(w->sum_b) + pad(w->fx) + pad(w->part_a) + pad(w->part_b) +
             pad(w->h_a) + pad(w->h_b) + pad(w->closed);
  if (unit_part) bytes += pad(w->sums) + pad(w->wfold) + pad(w->tile_part);
  return bytes;
}

int pylo_b200_grad_sumsq(const pylo_gvec* descs, const pylo_tile* tiles, int n_tiles, float* scratch,
                         float* out, void* stream) {
  CHECK_ARG(descs && tiles && scratch && out && n_tiles >= 0);
  cudaStream_t s = (cudaStream_t)stream;
  if (n_tiles > 0) launch(k_grad_sumsq, grid_for(n_tiles, 8), NT, 0, s, descs, tiles, n_tiles, scratch);
  launch(k_sum_final, 1, 1024, 0, s, scratch, n_tiles, out);
  return launch_status();
}

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of pylo_b200_grad_sumsq.
//
// Some hosts of this library cannot hand it scratch memory: a language binding that links only this
// .so and has no device allocator of its own, or a step loop whose rules forbid cudaMalloc because it
// synchronises the device.  For them the per-tile partial sums live in the fixed array below instead
// of a caller buffer.  The array is part of the loaded module, so every GPU that loads the library
// carries its 256 KiB until the process exits.
//
// In host code the name `g_static_sumsq_scratch` is only a handle for the symbol, not a pointer the
// device can follow, so the device address is looked up with cudaGetSymbolAddress, once per device,
// with that device current, and that address is what the kernels receive.
// ------------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_static_sumsq_scratch[PYLO_STATIC_SCRATCH_TILES];

static float* g_static_scratch_addr[PYLO_MAX_DEVICES] = {nullptr};
static std::mutex g_static_scratch_mutex;

static int static_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= PYLO_MAX_DEVICES) return -3;
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (g_static_scratch_addr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_static_sumsq_scratch);
    if (e != cudaSuccess) return (int)e;
    if (p == nullptr) return -3;
    g_static_scratch_addr[dev] = p;
  }
  *out = g_static_scratch_addr[dev];
  return 0;
}

int pylo_b200_grad_sumsq_static(const pylo_gvec* items, const pylo_tile* tiles, int n_tiles, float* out,
                                void* stream) {
  CHECK_ARG(items && tiles && out && n_tiles >= 0);
  if (n_tiles > PYLO_STATIC_SCRATCH_TILES) return PYLO_ERR_STATIC_SCRATCH_TOO_SMALL;
  float* scratch = nullptr;
  const int rc = static_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  // every slot that the final sum reads is written by the partial kernel of this same call, so
  // nothing left over from an earlier call needs clearing
  if (n_tiles > 0) launch(k_grad_sumsq, grid_for(n_tiles, 8), NT, 0, s, items, tiles, n_tiles, scratch);
  launch(k_sum_final, 1, 1024, 0, s, scratch, n_tiles, out);
  return launch_status();
}

int pylo_b200_rowcol_sums(const pylo_tensor_desc* descs, const pylo_atile* atiles, int n_atiles, int n_ragged, int n_kernel,
                          const pylo_atile* gitems, int n_gitems, const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && prm && n_ragged >= 0 && n_kernel >= 0 && n_atiles >= n_ragged + n_kernel && n_gitems >= 0 && (atiles || !n_atiles));
  cudaStream_t s = (cudaStream_t)stream;
  CHECK_ARG(gitems || !n_gitems);
  const pylo_atile* fast = atiles + n_ragged;
  const int n_fast = n_atiles - n_ragged;
  if (n_ragged > 0) launch(k_rowcol_fast<false, false>, grid_for(n_ragged, 3), NT, 0, s, descs, atiles, n_ragged, gitems, 0, *prm);
  // how many of the aligned items go with the variant that takes KERNEL and GENERIC tensors along: all of a small model's, else the KERNEL ones
  const int most = n_kernel > 0 ? PYLO_ROWCOL_KERNEL_APART : PYLO_ROWCOL_ONE_LAUNCH;
  const int mixed = n_fast - n_kernel > most ? n_kernel : n_kernel > 0 || n_gitems > 0 ? n_fast : 0;
  if (mixed > 0) launch(k_rowcol_fast<true, true>, n_gitems + grid_for(mixed, 3), NT, 0, s, descs, fast, mixed, gitems, n_gitems, *prm);
  else if (n_gitems > 0) launch(k_rowcol_generic, n_gitems, NT, 0, s, descs, gitems, *prm);
  if (n_fast > mixed) launch(k_rowcol_fast<true, false>, grid_for(n_fast - mixed, 4), NT, 0, s, descs, fast + mixed, n_fast - mixed, gitems, 0, *prm);
  return launch_status();
}

int pylo_b200_factor_update(const pylo_tensor_desc* descs, const int32_t* mats, int n_tensors, int threads, const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && prm && n_tensors >= 0 && (threads == A2_NT || threads == A2_NT / 2));
  if (n_tensors == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  switch (prm->family) {
    case PYLO_FAM_ADAFAC: factor_update_launch<PYLO_FAM_ADAFAC>(descs, mats, n_tensors, threads, *prm, s); break;
    case PYLO_FAM_CELO2: factor_update_launch<PYLO_FAM_CELO2>(descs, mats, n_tensors, threads, *prm, s); break;
    case PYLO_FAM_VELO: factor_update_launch<PYLO_FAM_VELO>(descs, mats, n_tensors, threads, *prm, s); break;
    default: return -2;
  }
  return launch_status();
}

int pylo_b200_state_moments(const pylo_tensor_desc* descs, const pylo_tile* tiles, int n_tiles, int reverse,
                            const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && tiles && prm && n_tiles >= 0);
  if (n_tiles == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  int rc = 0;
  switch (prm->family) {
    case PYLO_FAM_ADAFAC: rc = state_moments_launch<PYLO_FAM_ADAFAC>(descs, tiles, n_tiles, reverse, *prm, s); break;
    case PYLO_FAM_CELO2: rc = state_moments_launch<PYLO_FAM_CELO2>(descs, tiles, n_tiles, reverse, *prm, s); break;
    case PYLO_FAM_VELO: rc = state_moments_launch<PYLO_FAM_VELO>(descs, tiles, n_tiles, reverse, *prm, s); break;
    default: return -2;
  }
  if (rc) return rc;
  return launch_status();
}

int pylo_b200_small_front(const pylo_tensor_desc* descs, int n_tensors, int cluster, int slice, int rows, int cols, int networks,
                          const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && prm && n_tensors >= 0 && networks >= 0 && (networks == 0 || prm->family == PYLO_FAM_ADAFAC));
  CHECK_ARG(((uintptr_t)descs & 15) == 0);   // a descriptor is read in pieces of 16 bytes
  CHECK_ARG(cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8 || cluster == 16);
  const SfShape q = {(slice + 3) & ~3, (rows + 3) & ~3, (cols + 3) & ~3};   // the arrays start on 16-byte boundaries
  CHECK_ARG(slice >= 0 && rows >= 0 && cols >= 0 && slice <= SF_SLICE && sf_floats(q) <= PYLO_SMALL_FLOATS);
  if (n_tensors == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  switch (prm->family) {
    case PYLO_FAM_ADAFAC: return small_front_launch<PYLO_FAM_ADAFAC>(descs, n_tensors, cluster, q, networks, *prm, s);
    case PYLO_FAM_CELO2: return small_front_launch<PYLO_FAM_CELO2>(descs, n_tensors, cluster, q, 0, *prm, s);
    case PYLO_FAM_VELO: return small_front_launch<PYLO_FAM_VELO>(descs, n_tensors, cluster, q, 0, *prm, s);
    default: return -2;
  }
}

int pylo_b200_finalize_moments(const pylo_tensor_desc* descs, int n_tensors, void* stream) {
  CHECK_ARG(descs && n_tensors >= 0);
  if (n_tensors == 0) return 0;
  // many units (the slices of a CELO2 tensor) have few tiles each: small CTAs then
  if (n_tensors > 512) launch(k_finalize_moments<6>, n_tensors, 6 * PYLO_STAT_STRIDE, 0, (cudaStream_t)stream, descs);
  else launch(k_finalize_moments<25>, n_tensors, 25 * PYLO_STAT_STRIDE, 0, (cudaStream_t)stream, descs);
  return launch_status();
}

int pylo_b200_prep_apply(const pylo_tensor_desc* descs, const pylo_atile* items, int n_items, const pylo_step_params* prm,
                         void* stream) {
  CHECK_ARG(descs && items && prm && n_items >= 0);
  if (n_items == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  switch (prm->family) {
    case PYLO_FAM_ADAFAC:
      if (prm->no_tables != 2) launch(k_prep_apply<PYLO_FAM_ADAFAC>, n_items, NT, 0, s, descs, items, *prm);
      if (prm->no_tables == 2 || prm->no_tables == 0) launch(k_prep_tc, n_items, NT, 0, s, descs, items, *prm);
      break;
    case PYLO_FAM_CELO2: launch(k_prep_apply<PYLO_FAM_CELO2>, n_items, NT, 0, s, descs, items, *prm); break;
    case PYLO_FAM_VELO: launch(k_prep_apply<PYLO_FAM_VELO>, n_items, NT, 0, s, descs, items, *prm); break;
    default: return -2;
  }
  return launch_status();
}

int pylo_b200_apply(const pylo_tensor_desc* descs, const pylo_tile* tiles, int n_tiles, int reverse,
                    const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && tiles && prm && n_tiles >= 0);
  if (n_tiles == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  switch (prm->family) {
    case PYLO_FAM_ADAFAC: launch(k_apply<PYLO_FAM_ADAFAC>, grid_for(n_tiles, 2), NT, 0, s, descs, tiles, n_tiles, reverse, *prm); break;
    case PYLO_FAM_CELO2: launch(k_apply<PYLO_FAM_CELO2>, grid_for(n_tiles, 4), NT, 0, s, descs, tiles, n_tiles, reverse, *prm); break;
    case PYLO_FAM_VELO: launch(k_apply<PYLO_FAM_VELO>, grid_for(n_tiles, 4), NT, 0, s, descs, tiles, n_tiles, reverse, *prm); break;
    default: return -2;
  }
  return launch_status();
}

int pylo_b200_apply_adafac_cols(const pylo_tensor_desc* descs, const pylo_atile* ctiles, int n_ctiles,
                                const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && ctiles && prm && n_ctiles >= 0 && prm->family == PYLO_FAM_ADAFAC);
  if (n_ctiles == 0) return 0;
  static bool configured[PYLO_MAX_DEVICES] = {};
  if (int rc = allow_dynamic_smem(k_apply_adafac_cols, (int)sizeof(CcSmem), configured)) return rc;
  launch(k_apply_adafac_cols, grid_for(n_ctiles, CC_CTAS_PER_SM), NT, sizeof(CcSmem), (cudaStream_t)stream, descs, ctiles, n_ctiles, *prm);
  return launch_status();
}

int pylo_b200_apply_adafac_tc(const pylo_tensor_desc* descs, const pylo_atile* ttiles, int n_ttiles, int generic,
                              const pylo_step_params* prm, int* status, int* host_status, void* stream) {
  CHECK_ARG(descs && ttiles && prm && n_ttiles >= 0 && prm->family == PYLO_FAM_ADAFAC);
  if (n_ttiles == 0) return 0;
  CHECK_ARG(generic || prm->no_tables != 4);   // the other variant makes no scales
  // more than half an SM's shared memory is requested: one CTA per SM, which then owns all of the SM's tensor memory
  constexpr int smem = sizeof(TcSmem) > 120 * 1024 ? (int)sizeof(TcSmem) : 120 * 1024;
  static bool configured[4][PYLO_MAX_DEVICES] = {};
  TcHeads heads = {};
  if (prm->w_host) {   // w_in[32][39] b_in[32] w_h[32][32] b_h[32] w_out[2][32] b_out[2]
    const float* w = prm->w_host + 32 * 39 + 32 + 32 * 32 + 32;
    for (int k = 0; k < 32; ++k)
      for (int q = 0; q < 2; ++q) heads.w[4 * (k / 2) + 2 * q + k % 2] = w[32 * q + k];
    heads.b[0] = w[64];
    heads.b[1] = w[65];
  }
  auto kernel = prm->w_host ? (generic ? k_apply_adafac_tc<true, true> : k_apply_adafac_tc<false, true>)
                            : (generic ? k_apply_adafac_tc<true, false> : k_apply_adafac_tc<false, false>);
  if (int rc = allow_dynamic_smem(kernel, smem, configured[(generic ? 1 : 0) + (prm->w_host ? 2 : 0)])) return rc;
  launch(kernel, grid_for(n_ttiles, 1), TC_NT, smem, (cudaStream_t)stream, descs, ttiles, n_ttiles, *prm, status, host_status, heads);
  return launch_status();
}

int pylo_b200_gemm_tn_3xtf32(const pylo_gemm_desc* g, int* status, void* stream) {
  CHECK_ARG(g && g->A && g->B && g->C);
  CHECK_ARG(g->M > 0 && g->N > 0 && g->K > 0 && g->batch > 0);
  // rows are moved in 16-byte pieces
  CHECK_ARG(g->K % 4 == 0 && g->N % 4 == 0 && g->lda % 4 == 0 && g->ldb % 4 == 0 && g->ldc % 4 == 0);
  CHECK_ARG(g->lda >= g->K && g->ldb >= g->K && g->ldc >= g->N);
  CHECK_ARG(((uintptr_t)g->A | (uintptr_t)g->B | (uintptr_t)g->C | (uintptr_t)g->D) % 16 == 0);
  CHECK_ARG(g->strideA % 4 == 0 && g->strideB % 4 == 0 && g->strideC % 4 == 0);
  if (g->D) CHECK_ARG(g->ldd % 4 == 0 && g->ldd >= g->N && g->strideD % 4 == 0 && g->D != g->C);
  static_assert(sizeof(pylo_gemm_desc) == sizeof(pylo_gemm_args), "pylo_gemm_desc and the kernel's argument block differ");
  pylo_gemm_args a;
  memcpy(&a, g, sizeof(a));
  if (g->symmetric) CHECK_ARG(g->M == g->N);
  const long long tiles = (long long)ns_tiles_per_matrix((g->M + NS_BM - 1) / NS_BM, (g->N + NS_BN - 1) / NS_BN, g->symmetric) * g->batch;
  static bool configured[PYLO_MAX_DEVICES] = {};
  constexpr int smem = (int)sizeof(NsSmem) + 1024;  // room to start the tiles on a 1024-byte boundary
  if (int rc = allow_dynamic_smem(k_gemm_tn_3xtf32, smem, configured)) return rc;
  const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
  launch(k_gemm_tn_3xtf32, grid, NS_THREADS, smem, (cudaStream_t)stream, a, status);
  return launch_status();
}

int pylo_b200_transpose(const float* src, float* dst, int rows, int cols, int ld_src, int ld_dst, int64_t stride_src,
                        int64_t stride_dst, int batch, int mirror, void* stream) {
  CHECK_ARG(src && dst && rows > 0 && cols > 0 && batch > 0 && batch <= 65535 && ld_src >= cols);
  if (mirror) CHECK_ARG(rows == cols && src == dst && ld_src == ld_dst);
  else CHECK_ARG(src != dst && ld_dst >= rows);
  const dim3 grid((cols + 31) / 32, (rows + 31) / 32, batch);
  CHECK_ARG(grid.y <= 65535);
  launch(k_transpose32, grid, 256, 0, (cudaStream_t)stream, src, dst, rows, cols, ld_src, ld_dst, stride_src, stride_dst, mirror ? 1 : 0);
  return launch_status();
}

// ------------------------------------------------------------------------------------------------
// Newton-Schulz chain
// ------------------------------------------------------------------------------------------------
int64_t pylo_b200_newton_schulz_workspace(int rows, int cols, int batch, int iters) {
  if (rows <= 0 || cols <= 0 || batch <= 0 || iters < 0) return -1;
  return ns_parts(rows, cols, iters) >= 0 ? 0 : ns_work(rows, cols, batch).total;
}

int pylo_b200_newton_schulz_workspaces(const pylo_ns_desc* descs, int n, int64_t* bytes) {
  CHECK_ARG(descs && bytes && n >= 0);
  for (int k = 0; k < n; ++k) CHECK_ARG(descs[k].rows > 0 && descs[k].cols > 0 && descs[k].batch > 0 && descs[k].iters >= 0);
  const NsRoutes route(descs, n);
  for (int k = 0; k < n; ++k)
    bytes[k] = route.rides(ns_parts(descs[k].rows, descs[k].cols, descs[k].iters)) ? ns_work(descs[k].rows, descs[k].cols, descs[k].batch).total : 0;
  return 0;
}

typedef CUresult (*TensorMapEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TensorMapEncode tensor_map_encode() {
  static TensorMapEncode fn = [] {   // initialised once, also with several threads
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return (TensorMapEncode)p;
  }();
  return fn;
}
// planes [2][batch][rows][ld] of fp16, boxes of 64 x 64; what a box reaches beyond a matrix reads as zero
static int ns_map(CUtensorMap* map, void* base, int rows, int cols, int ld, int batch) {
  TensorMapEncode fn = tensor_map_encode();
  if (!fn) return -5;
  const cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch, 2};
  const cuuint64_t strides[3] = {(cuuint64_t)ld * 2, (cuuint64_t)rows * ld * 2, (cuuint64_t)batch * rows * ld * 2};
  const cuuint32_t box[4] = {64, 64, 1, 1}, unit[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -5;
}

// the chain of up to NF_GROUP stacks of matrices, step by step side by side
static int ns_chain(const pylo_ns_desc* const* ds, int n, int* status, cudaStream_t s) {
  struct Stack { NsWork w; CUtensorMap x[2], a, b; char* base; };
  Stack st[NF_GROUP];
  // |x|, |a|, |b| stay below about 1.3, 1.5 and 3 for the usual coefficients and below 10, 15 and 15 for whatever this is
  // called with (the caller checks): 2^12 keeps them inside fp16's range
  constexpr float SX = 4096.f, SA = 4096.f, SB = 4096.f;
  nf_prep_group prep = {};
  prep.n = n;
  long long ctas = 0;
  for (int k = 0; k < n; ++k) {
    const pylo_ns_desc& d = *ds[k];
    Stack& t = st[k];
    t.w = ns_work(d.rows, d.cols, d.batch);
    t.base = (char*)d.work;
    for (int q = 0; q < 2; ++q)
      if (int rc = ns_map(&t.x[q], t.base + t.w.xp[q], d.rows, d.cols, t.w.ldx, d.batch)) return rc;
    if (int rc = ns_map(&t.a, t.base + t.w.ap, t.w.r, t.w.r, t.w.lda_p, d.batch)) return rc;
    if (int rc = ns_map(&t.b, t.base + t.w.bp, t.w.r, t.w.r, t.w.lda_p, d.batch)) return rc;
    nf_prep& p = prep.p[k];
    p.x = d.x; p.n = (long long)d.rows * d.cols;
    p.part = (float*)(t.base + t.w.part); p.inv = (float*)(t.base + t.w.inv); p.P = (__half*)(t.base + t.w.xp[0]);
    p.sP = (long long)d.rows * t.w.ldx; p.planeP = p.sP * d.batch;
    p.cols = d.cols; p.ldp = t.w.ldx; p.slices = t.w.slices; p.cta0 = (int)ctas; p.eps = d.eps; p.scale = SX;
    ctas += (long long)t.w.slices * d.batch;
  }
  if (ctas > 0x7fffffff) return -1;
  launch(k_ns_sumsq, (int)ctas, NT, 0, s, prep);
  launch(k_ns_split, (int)ctas, NT, 0, s, prep);
  const int iters = ds[0]->iters;
  nf_group grp;
  grp.n = n;
  for (int it = 0; it < iters; ++it) {
    const int cur = it & 1;
    const bool last = it == iters - 1;
    for (int step = 0; step < 3; ++step) {
      for (int k = 0; k < n; ++k) {
        const pylo_ns_desc& d = *ds[k];
        Stack& t = st[k];
        const NsWork& w = t.w;
        const bool wide = d.rows <= d.cols;
        const long long size = (long long)d.rows * d.cols, sA = (long long)w.r * w.lda, sAp = (long long)w.r * w.lda_p;
        nf_problem& q = grp.p[k];
        nf_args g = {};
        g.batch = d.batch;
        if (step == 0) {          // a = x x^T (wide), x^T x (tall)
          q.A = q.B = t.x[cur];
          g.C = (float*)(t.base + w.a); g.sC = sA; g.ldc = w.lda;
          g.P = (__half*)(t.base + w.ap); g.sP = sAp; g.ldp = w.lda_p; g.planeP = sAp * d.batch;
          g.M = g.N = w.r; g.K = w.c;
          g.alpha = 1.0f / (SX * SX); g.scale = SA; g.a_mn = g.b_mn = !wide; g.symmetric = 1;
        } else if (step == 1) {   // b = c1 a + c2 a a
          q.A = q.B = t.a;
          g.D = (float*)(t.base + w.a); g.sD = sA; g.ldd = w.lda;
          g.P = (__half*)(t.base + w.bp); g.sP = sAp; g.ldp = w.lda_p; g.planeP = sAp * d.batch;
          g.M = g.N = g.K = w.r;
          g.alpha = d.c2 / (SA * SA); g.beta = d.c1; g.scale = SB; g.symmetric = 1;
          if (d.c2 == 0.f) { g.K = 0; g.alpha = 1.0f; }   // no product: b = c1 a
        } else {                  // x' = c0 x + b x (wide), c0 x + x b (tall); the first round's x is d.x times inv
          q.A = wide ? t.b : t.x[cur];
          q.B = wide ? t.x[cur] : t.b;
          float* const even = (float*)(t.base + w.x);
          g.C = ((iters - it) & 1) ? d.out : even; g.sC = size; g.ldc = d.cols;   // the last round writes d.out
          g.D = it == 0 ? d.x : ((iters - it) & 1) ? even : d.out; g.sD = size; g.ldd = d.cols;
          g.d_scale = it == 0 ? (float*)(t.base + w.inv) : nullptr;
          if (!last) { g.P = (__half*)(t.base + w.xp[cur ^ 1]); g.sP = (long long)d.rows * w.ldx; g.ldp = w.ldx; g.planeP = g.sP * d.batch; }
          g.M = d.rows; g.N = d.cols; g.K = w.r;
          g.alpha = 1.0f / (SB * SX); g.beta = d.c0; g.scale = SX; g.b_mn = wide;
        }
        q.g = g;
      }
      if (int rc = ns_gemm(grp, status, s)) return rc;
    }
  }
  return 0;
}

int pylo_b200_newton_schulz(const pylo_ns_desc* descs, int n, int* status, void* stream) {
  CHECK_ARG(descs && n >= 0);
  cudaStream_t s = (cudaStream_t)stream;
  for (int k = 0; k < n; ++k) {
    const pylo_ns_desc& d = descs[k];
    CHECK_ARG(d.x && d.out && d.x != d.out && d.rows > 0 && d.cols > 0 && d.batch > 0 && d.iters >= 1 && d.iters == descs[0].iters);
    CHECK_ARG(d.cols % 4 != 0 || (((uintptr_t)d.x | (uintptr_t)d.out) & 15) == 0);   // rows are moved in 16-byte pieces where they can
    if (ns_parts(d.rows, d.cols, d.iters) < 0) CHECK_ARG(d.work && ((uintptr_t)d.work & 255) == 0 && d.work_bytes >= ns_work(d.rows, d.cols, d.batch).total);
  }
  // what clusters take goes first, and with it, beside it, what single CTAs take
  const pylo_ns_desc* group[NF_GROUP];
  int m = 0;
  nc_group small = {};
  small.iters = n ? descs[0].iters : 0;
  auto run_clusters = [&]() { const int rc = small.n ? ns_clusters(small, status, s) : 0; small.n = 0; return rc; };
  const NsRoutes route(descs, n);
  for (int k = 0; k < n; ++k) {
    const pylo_ns_desc& d = descs[k];
    const NsRoute to = route(d);
    if (to == NS_CLUSTERS) {
      small.p[small.n++] = {d.x, d.out, d.rows, d.cols, d.batch, ns_parts(d.rows, d.cols, d.iters), 0, d.c0, d.c1, d.c2, d.eps};
      if (small.n == NF_GROUP)
        if (int rc = run_clusters()) return rc;
    } else if (to == NS_SINGLE) {
      static bool configured[PYLO_MAX_DEVICES] = {};
      if (int rc = allow_dynamic_smem(k_ns_small, 200 * 1024, configured)) return rc;
      launch(k_ns_small, d.batch, NT, (size_t)ns_small_floats(d.rows, d.cols) * 4, s, d.x, d.out, d.rows, d.cols, d.iters, d.c0, d.c1, d.c2, d.eps);
    } else {
      group[m++] = &d;
      if (m == NF_GROUP) {
        if (int rc = ns_chain(group, m, status, s)) return rc;
        m = 0;
      }
    }
  }
  if (int rc = run_clusters()) return rc;
  if (m)
    if (int rc = ns_chain(group, m, status, s)) return rc;
  return launch_status();
}

int pylo_b200_newton_schulz_launches(const pylo_ns_desc* descs, int n) {
  CHECK_ARG(descs && n >= 0);
  const NsRoutes route(descs, n);
  int of[3] = {};
  for (int k = 0; k < n; ++k) ++of[route(descs[k])];
  auto groups = [](int m) { return (m + NF_GROUP - 1) / NF_GROUP; };
  return groups(of[NS_CLUSTERS]) + of[NS_SINGLE] + groups(of[NS_CHAIN]) * (2 + 3 * (n ? descs[0].iters : 0));
}

int pylo_b200_apply_packed(const pylo_tensor_desc* descs, const pylo_atile* ctiles, int n_ctiles, int ragged,
                           const pylo_tile* tiles, int n_tiles, const pylo_step_params* prm, void* stream) {
  CHECK_ARG(descs && (ctiles || !n_ctiles) && (tiles || !n_tiles) && prm && n_ctiles >= 0 && n_tiles >= 0);
  if (n_ctiles == 0) return n_tiles ? pylo_b200_apply(descs, tiles, n_tiles, 0, prm, stream) : 0;
  cudaStream_t s = (cudaStream_t)stream;
  switch (prm->family) {
    case PYLO_FAM_CELO2: {
      PkNet<PYLO_FAM_CELO2> net = {};
      if (prm->w_host) {
        using W = PkW<PYLO_FAM_CELO2>;
        const float* w = prm->w_host;   // w_in[30][8] b_in[8] w_h[8][8] b_h[8] w_out[8][3] b_out[3]
        for (int e = 0; e < 18 * 8; ++e) net.w[W::W1 + e] = w[e < 15 * 8 ? e : e + 12 * 8];
        for (int e = 0; e < 64; ++e) net.w[W::W2 + e] = w[248 + e];
        for (int e = 0; e < 8; ++e) { net.w[W::B2 + e] = w[312 + e]; net.w[W::W3 + 2 * e] = w[320 + 3 * e]; net.w[W::W3 + 2 * e + 1] = w[321 + 3 * e]; }
        net.w[W::B3] = w[344]; net.w[W::B3 + 1] = w[345];
      }
      auto kernel = prm->w_host ? (ragged ? k_apply_packed<PYLO_FAM_CELO2, true, true> : k_apply_packed<PYLO_FAM_CELO2, true, false>)
                                : (ragged ? k_apply_packed<PYLO_FAM_CELO2, false, true> : k_apply_packed<PYLO_FAM_CELO2, false, false>);
      const int packed = grid_for(n_ctiles, PK_CTAS_CELO2);
      launch(kernel, packed, NT, 0, s, descs, ctiles, n_ctiles, packed, (const pylo_tile*)nullptr, 0, *prm, net);
      if (n_tiles) return pylo_b200_apply(descs, tiles, n_tiles, 0, prm, stream);
      break;
    }
    // four times the CTAs that fit: an SM that is done takes the next (17 M parameters: 341 -> 327 us per step, 67 M: 1104 ->
    // 1091); CELO2's larger network is loaded by every CTA, which costs more than that gives
    case PYLO_FAM_VELO: {
      const int packed = grid_for(n_ctiles, 4 * PK_CTAS_VELO);
      launch(ragged ? k_apply_packed<PYLO_FAM_VELO, false, true> : k_apply_packed<PYLO_FAM_VELO, false, false>, packed + grid_for(n_tiles, 4), NT, 0, s,
             descs, ctiles, n_ctiles, packed, tiles, n_tiles, *prm, PkNet<PYLO_FAM_VELO>{});
      break;
    }
    default: return -2;
  }
  return launch_status();
}

int pylo_b200_celo2_post_sums(const pylo_post_item* items, const pylo_tile* tiles, int n_tiles, void* stream) {
  CHECK_ARG(items && tiles && n_tiles >= 0);
  if (n_tiles == 0) return 0;
  const PlainLaunches plain(n_tiles);
  launch(k_post_sums, grid_for(n_tiles, 8), NT, 0, (cudaStream_t)stream, items, tiles, n_tiles);
  return launch_status();
}

int pylo_b200_celo2_post_apply(const pylo_post_item* items, const pylo_tile* tiles, int n_tiles, const int* status, int* host_status,
                               void* stream) {
  CHECK_ARG(items && tiles && n_tiles >= 0);
  if (n_tiles == 0) return 0;
  const PlainLaunches plain(n_tiles);
  launch(k_post_apply, grid_for(n_tiles, 8), NT, 0, (cudaStream_t)stream, items, tiles, n_tiles, status, host_status);
  return launch_status();
}

int pylo_b200_adamw(const pylo_adam_item* items, const pylo_tile* tiles, int n_tiles, int independent, float beta1,
                    float one_minus_beta1, float beta2, float one_minus_beta2, float eps, float bc1, float bc2,
                    const pylo_step_params* prm, void* stream) {
  CHECK_ARG(items && tiles && prm && n_tiles >= 0);
  if (n_tiles == 0) return 0;
  const PlainLaunches plain(n_tiles);
  launch(independent ? k_adamw<true> : k_adamw<false>, grid_for(n_tiles, 8), NT, 0, (cudaStream_t)stream, items, tiles, n_tiles,
         Adam{beta1, one_minus_beta1, beta2, one_minus_beta2, eps, bc1, bc2}, *prm);
  return launch_status();
}

int pylo_b200_celo2_tail(const pylo_post_item* post, const pylo_tile* post_tiles, int n_post, const int* status, int* host_status,
                         const pylo_adam_item* items, const pylo_tile* tiles, int n_tiles, int independent, float beta1, float one_minus_beta1,
                         float beta2, float one_minus_beta2, float eps, float bc1, float bc2, const pylo_step_params* prm, void* stream) {
  CHECK_ARG(post && post_tiles && items && tiles && prm && n_post > 0 && n_tiles > 0);
  launch(independent ? k_post_adamw<true> : k_post_adamw<false>, grid_for(n_post, 4) + grid_for(n_tiles, 4), NT, 0, (cudaStream_t)stream, post, post_tiles,
         n_post, grid_for(n_post, 4), status, host_status, items, tiles, n_tiles,
         Adam{beta1, one_minus_beta1, beta2, one_minus_beta2, eps, bc1, bc2}, *prm);
  return launch_status();
}

int pylo_b200_velo_tensor_features(const pylo_tensor_desc* descs, int n_local, const int32_t* layer_of,
                                   int n_total, const float* rank_onehot, float fraction,
                                   const pylo_velo_loss* lossbuf, float* x_in, void* stream) {
  CHECK_ARG(descs && rank_onehot && x_in && n_local > 0 && n_total >= n_local);
  CHECK_ARG(lossbuf && lossbuf->means && lossbuf->iteration && lossbuf->running_min && lossbuf->decays);
  launch(k_velo_tensor_features<20>, n_local, 20 * PYLO_STAT_STRIDE + 32, 0, (cudaStream_t)stream, descs, layer_of, n_total,
         rank_onehot, fraction, *lossbuf, x_in);
  return launch_status();
}

int pylo_b200_velo_inputs(const pylo_tensor_desc* descs, const int32_t* layer_of, const float* rank_onehot, float fraction,
                          const pylo_velo_loss* lossbuf, const pylo_velo_rnn* rnn, void* stream) {
  CHECK_ARG(descs && rank_onehot && rnn && rnn->T > 0 && rnn->T <= VI_TENSORS && rnn->x_in && rnn->xmix);
  CHECK_ARG(lossbuf && lossbuf->means && lossbuf->iteration && lossbuf->running_min && lossbuf->decays);
  launch(k_velo_inputs, (rnn->H + NWARP - 1) / NWARP, NT, 0, (cudaStream_t)stream, descs, layer_of, rank_onehot, fraction, *lossbuf, *rnn);
  return launch_status();
}

int pylo_b200_velo_rnn(const pylo_velo_rnn* rnn, const pylo_velo_loss* lossbuf, void* stream) {
  CHECK_ARG(rnn && rnn->T > 0 && rnn->H > 0 && rnn->B > 0 && rnn->B <= 1024);
  cudaStream_t s = (cudaStream_t)stream;
  const pylo_velo_rnn r = *rnn;
  const int64_t TH = (int64_t)r.T * r.H;
  const pylo_velo_loss none = {};
  const bool tiled = !(r.H % 128 == 0 && r.H <= 512);   // the LSTM's other kernels
  CHECK_ARG(!r.mixed || !tiled);
  if (!r.mixed) launch(k_velo_xmix, (r.H + NWARP - 1) / NWARP, NT, 0, s, r, lossbuf ? *lossbuf : none);
  const float* h = r.h;   // the new one
  if (!tiled) {
    const int gx = r.H / GR_UNITS, groups = (r.T + 7) / 8;
    const int gy = groups * gx <= 2 * sm_count() ? groups : (2 * sm_count() / gx > 0 ? 2 * sm_count() / gx : 1);   // two CTAs per SM
    const int per = (groups + gy - 1) / gy, smem = 2 * 8 * 2 * r.H * (int)sizeof(float);
    static bool configured[4][PYLO_MAX_DEVICES] = {};
    auto kernel = r.H == 128 ? k_velo_lstm<1> : r.H == 256 ? k_velo_lstm<2> : r.H == 384 ? k_velo_lstm<3> : k_velo_lstm<4>;
    if (int rc = allow_dynamic_smem(kernel, smem, configured[r.H / 128 - 1])) return rc;
    launch(kernel, dim3(gx, gy), NT, smem, s, r, r.mixed && lossbuf ? *lossbuf : none, per);
    h = r.gates;
  } else {
    launch(k_velo_gates, dim3((4 * r.H + GT - 1) / GT, (r.T + GT - 1) / GT), NT, 0, s, r);
    launch(k_velo_cell, (unsigned)((TH + 255) / 256), 256, 0, s, r);
  }
  const int64_t hw = (int64_t)r.T * (r.B + 1);
  launch(k_velo_heads, (unsigned)((hw + NWARP - 1) / NWARP), NT, 0, s, r, h);
  launch(k_velo_mix, dim3(r.T, 160 / MIX_OUT), MIX_OUT * MIX_GROUPS, r.B * sizeof(float), s, r, h);
  return launch_status();
}

int pylo_b200_velo_loss_features(float* means, int32_t* iteration, float* running_min, const float* decays,
                                 const float* loss, float* loss9, void* stream) {
  CHECK_ARG(means && iteration && running_min && decays && loss && loss9);
  const pylo_velo_loss b = {means, iteration, running_min, decays, loss, 0.f, 0};
  launch(k_velo_loss, 1, 32, 0, (cudaStream_t)stream, b, loss9);
  return launch_status();
}

// ------------------------------------------------------------------------------------------------
// A step's phases in one call, for hosts whose own call overhead counts (a ctypes call costs about as much as a launch).
// ------------------------------------------------------------------------------------------------
int pylo_b200_step(const pylo_step_plan* p, const pylo_step_params* prm, int phases, void* stream) {
  CHECK_ARG(p && prm);
  const PlainLaunches plain(p->n_tiles);
  int rc = 0;
  constexpr int front = PYLO_STEP_SUMS | PYLO_STEP_FACTORS | PYLO_STEP_STATE;
  if (p->small_cluster && (phases & front) == front) {
    if ((rc = pylo_b200_small_front(p->tdesc, p->n_tensors, p->small_cluster, p->small_slice, p->small_rows, p->small_cols, p->small_networks, prm, stream))) return rc;
    phases &= ~front;
  }
  if ((phases & PYLO_STEP_SUMS) && (p->n_atiles || p->n_gitems))
    if ((rc = pylo_b200_rowcol_sums(p->tdesc, p->atiles, p->n_atiles, p->n_ragged, p->n_kernel, p->gitems, p->n_gitems, prm, stream))) return rc;
  if (phases & PYLO_STEP_FACTORS)
    if ((rc = pylo_b200_factor_update(p->tdesc, p->mats, p->n_mats, p->factor_threads, prm, stream))) return rc;
  if (phases & PYLO_STEP_STATE)
    if ((rc = pylo_b200_state_moments(p->desc, p->tiles, p->n_tiles, 1, prm, stream))) return rc;
  if ((phases & PYLO_STEP_STATE) && p->small_networks) {   // the phases one by one: what the launch of all of them would have left
    pylo_step_params q = *prm;
    q.no_tables = 2;
    q.sum_tiles = 1;
    if ((rc = pylo_b200_prep_apply(p->desc, p->pitems, p->n_pitems, &q, stream))) return rc;
  }
  if ((phases & PYLO_STEP_MOMENTS) && !p->sum_tiles)
    if ((rc = pylo_b200_finalize_moments(p->desc, p->n_units, stream))) return rc;
  if (!(phases & PYLO_STEP_BACK)) return 0;
  pylo_step_params q = *prm;
  q.sum_tiles = p->sum_tiles && q.family != PYLO_FAM_VELO;
  q.no_tables = p->small_networks ? 4 : p->tensor_cores ? 2 : 3;
  if ((phases & PYLO_STEP_PREP) && !p->small_networks)
    if ((rc = pylo_b200_prep_apply(p->desc, p->pitems, p->n_pitems, &q, stream))) return rc;
  const bool main = phases & PYLO_STEP_APPLY, rest = phases & PYLO_STEP_APPLY_REST;
  if (p->tensor_cores) {
    // small models: one launch; large ones: what is not FAST2D first, then the others through the leaner variant
    const int first = p->n_ctiles - p->n_ctiles_gen < PYLO_TC_ONE_LAUNCH ? 0 : p->n_ctiles_gen;
    if (rest && (rc = pylo_b200_apply_adafac_tc(p->desc, p->ctiles, first, 1, &q, p->status, p->host_status, stream))) return rc;
    if (main && (rc = pylo_b200_apply_adafac_tc(p->desc, p->ctiles + first, p->n_ctiles - first, p->n_ctiles_gen > first || p->small_networks, &q, p->status, p->host_status, stream))) return rc;
    return 0;
  }
  if (q.family == PYLO_FAM_ADAFAC) {
    if (main && p->n_ctiles && (rc = pylo_b200_apply_adafac_cols(p->desc, p->ctiles, p->n_ctiles, &q, stream))) return rc;
    return rest && p->n_tiles_slow ? pylo_b200_apply(p->desc, p->tiles_slow, p->n_tiles_slow, 0, &q, stream) : 0;
  }
  // the tiles go with the first launch of packed items that there is
  int n_slow = rest ? p->n_tiles_slow : 0;
  if (main && p->n_ctiles) {
    if ((rc = pylo_b200_apply_packed(p->desc, p->ctiles, p->n_ctiles, 0, p->tiles_slow, n_slow, &q, stream))) return rc;
    n_slow = 0;
  }
  return rest ? pylo_b200_apply_packed(p->desc, p->rtiles, p->n_rtiles, 1, p->tiles_slow, n_slow, &q, stream) : 0;
}

int pylo_b200_advance_steps(double* const* steps, int n, double* first, int* equal) {
  CHECK_ARG(steps && n >= 0 && first && equal);
  *first = n ? *steps[0] : 0.0;
  *equal = 1;
  for (int i = 0; i < n; ++i) {
    if (*steps[i] != *first) *equal = 0;
    *steps[i] += 1.0;
  }
  return 0;
}

}  // extern "C"
