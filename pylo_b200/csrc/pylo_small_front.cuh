// Phases A, A2 and B of a small model in one launch, a cluster of CTAs per tensor (included by pylo_kernels.cu).
//
// On a small model each phase is a few dependent reads of descriptors and data from L2 and a launch: 4, 6.5 and 4 us for the
// 118 K parameters of a perceptron, whose data an SM reads in 2.  All that the three exchange belongs to one tensor, so a cluster
// can do them together: every CTA takes a run of the tensor's rows, copies its part of the gradient and of the state into shared
// memory at the start (the state arrives while the sums are made), and the CTAs exchange column sums and the tensor's fifteen
// sums through distributed shared memory.  It takes 11.3 us there: a step of 33.9 us takes 27.3.  Bound by latency (descriptor and
// copies 2 us, sums 1.5, the two exchanges 2.5, factors 1) and, in the state update (2.5), by the issue slots of a tensor's
// sixteen SMs.
// AdafacLO, ELO: clusters behind the tensors' make the networks of the tensor-core sweep meanwhile, which then only needs the features'
// scales; it adds the few partials up itself, and there is no launch in between (perceptron: us per step 23.5 -> 19.5).
// The host chooses it (LoPlan) where every tensor is a vector or a plain matrix whose share fits.
#pragma once

#define SF_NT 512
#define SF_SLICE 8192   // elements of a CTA's share of a tensor at most

struct SfShape { int slice, rows, cols; };   // largest share, its rows, columns of a matrix: the arrays below
__host__ __device__ inline int sf_floats(const SfShape& q) { return 6 * q.slice + 4 * q.rows + 5 * q.cols; }

template <bool VEC>
__device__ __forceinline__ void sf_copy(float* dst, const float* src, int cnt) {
  if constexpr (VEC) {
    for (int i = threadIdx.x * 4; i < cnt; i += SF_NT * 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst + i)), "l"(src + i) : "memory");
  } else {
    for (int i = threadIdx.x; i < cnt; i += SF_NT)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst + i)), "l"(src + i) : "memory");
  }
}

template <int FAM>
__global__ void __launch_bounds__(SF_NT, 1) k_small_front(const pylo_tensor_desc* __restrict__ descs, int n_tensors, const SfShape shape,
                                                          const pylo_step_params prm) {
  pdl_begin();
  using F = Fam<FAM>;
  constexpr int NACC = BAcc<FAM>::N, WARPS = SF_NT / 32, NS = 15;   // NS: as in k_factor_update
  extern __shared__ __align__(16) float sf[];
  __shared__ float s_red[WARPS * NACC];
  __shared__ float s_warp[WARPS][NS], s_cta[16][NS + 1], s_tot[NS + 1], s_scr[SF_NT];
  const int tid = threadIdx.x, lane = tid & 31, rank = (int)cluster_rank(), parts = (int)cluster_size();
  if constexpr (FAM == PYLO_FAM_ADAFAC) {
    // further clusters: the tensors' networks as the tensor-core sweep reads them, which need nothing that is made here
    const int first = n_tensors * parts;
    if ((int)blockIdx.x >= first) {
      TcNet& net = *reinterpret_cast<TcNet*>(sf);
      for (int u = blockIdx.x - first; u < n_tensors; u += gridDim.x - first) {
        tc_ask_network<SF_NT>(descs[u], net);
        tc_network<SF_NT>(descs[u], prm, net);
        __syncthreads();
      }
      return;
    }
  }
  __shared__ pylo_tensor_desc d;   // all of it at once: read field by field between the copies it costs a trip to L2 each time
  static_assert(sizeof(d) % 16 == 0 && sizeof(d) / 16 <= SF_NT, "a thread per 16 bytes");
  if (tid < (int)(sizeof(d) / 16)) reinterpret_cast<uint4*>(&d)[tid] = __ldg(reinterpret_cast<const uint4*>(descs + blockIdx.x / parts) + tid);
  __syncthreads();
  const float gs = grad_scale_of(d, prm);
  float acc[NACC];
#pragma unroll
  for (int j = 0; j < NACC; ++j) acc[j] = 0.f;
  float* const out = d.tile_part + (int64_t)rank * PYLO_STAT_STRIDE;
  if (d.mode == PYLO_MODE_VEC1D) {   // the same for all CTAs of the cluster
    const int per = ((int)d.n + parts - 1) / parts, start = rank * per;
    vec1d_update<FAM, SF_NT>(d, prm, gs, start, min(per, (int)d.n - start), acc);
    block_reduce_store<NACC, WARPS>(acc, s_red, out);
    if (tid >= NACC && tid < PYLO_STAT_STRIDE) out[tid] = 0.f;
    if (rank == 0 && tid < PYLO_STAT_STRIDE) d.closed[tid] = 0.f;
    return;
  }
  cluster_arrive();   // waited for before the first look into another CTA
  const int X = d.X, Y = d.Y, share = (X + parts - 1) / parts, row0 = rank * share, rows = max(0, min(share, X - row0)), cnt = rows * Y;
  const int64_t start = (int64_t)row0 * Y;
  const bool fast = d.mode == PYLO_MODE_FAST2D, r_is_a = d.r_is_a != 0;
  float *s_g = sf, *s_p = s_g + shape.slice, *s_m0 = s_p + shape.slice, *s_m1 = s_m0 + shape.slice, *s_m2 = s_m1 + shape.slice;
  float *s_v = s_m2 + shape.slice, *s_rs = s_v + shape.slice, *s_fa = s_rs + shape.rows, *s_col = s_fa + 3 * shape.rows, *s_fb = s_col + shape.cols, *s_sum = s_fb + 3 * shape.cols;
  float *m0p = d.m + start, *m1p = m0p + d.m_stride, *m2p = m1p + d.m_stride, *vp = d.v + start;
  auto copy = [&](auto vec) {
    constexpr bool V = decltype(vec)::value;
    sf_copy<V>(s_g, d.g + start, cnt);
    asm volatile("cp.async.commit_group;" ::: "memory");
    sf_copy<V>(s_p, d.p + start, cnt);
    sf_copy<V>(s_m0, m0p, cnt);
    sf_copy<V>(s_m1, m1p, cnt);
    sf_copy<V>(s_m2, m2p, cnt);
    sf_copy<V>(s_v, vp, cnt);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (fast) copy(std::true_type{});
  else copy(std::false_type{});

  const int cols = (Y + parts - 1) / parts, col0 = min(Y, rank * cols), col1 = min(Y, col0 + cols);   // this CTA's columns to finish
  float old_a[3] = {0.f, 0.f, 0.f}, old_b[3] = {0.f, 0.f, 0.f};   // of its first row and column: asked for long before they are needed
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (tid < rows) old_a[k] = d.fac_a[(int64_t)k * X + row0 + tid];
    if (col0 + tid < col1) old_b[k] = d.fac_b[(int64_t)k * Y + col0 + tid];
  }

  // ---- A: row sums, and column sums over this CTA's rows
  auto square = [](float g) { return g * g + 1e-30f; };
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  if (!plain_grad(gs, prm)) {
    for (int i = tid; i < cnt; i += SF_NT) s_g[i] = xform_grad(s_g[i], gs, prm.clip_val, prm.nan_to_num);
    __syncthreads();
  }
  {
    const int w = Y > 16 ? 32 : (Y > 8 ? 16 : (Y > 4 ? 8 : 4));   // lanes per row
    for (int r0 = 0; r0 < rows; r0 += SF_NT / w) {                // the same trip count for all threads
      const int r = r0 + tid / w;
      float s = 0.f;
      if (r < rows) {
        const float* const at = s_g + r * Y;
#pragma unroll 8
        for (int y = tid & (w - 1); y < Y; y += w) s += square(at[y]);
      }
      for (int o = w >> 1; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, w);
      if (r < rows && (tid & (w - 1)) == 0) s_rs[r] = s;
    }
    int W = 32;   // threads along the columns; the others take further rows
    while (W < Y && W < SF_NT) W *= 2;
    if (W == SF_NT) {
      for (int y = tid; y < Y; y += SF_NT) {
        float s = 0.f;
#pragma unroll 8
        for (int r = 0; r < rows; ++r) s += square(s_g[r * Y + y]);
        s_col[y] = s;
      }
    } else {
      const int y = tid & (W - 1);
      float s = 0.f;
      if (y < Y) {
#pragma unroll 8
        for (int r = tid / W; r < rows; r += SF_NT / W) s += square(s_g[r * Y + y]);
      }
      s_scr[tid] = s;
      __syncthreads();
      if (tid < Y) {
        for (int q = tid + W; q < SF_NT; q += W) s += s_scr[q];
        s_col[tid] = s;
      }
    }
  }
  // ---- A2: see k_factor_update.  "a" vectors have an entry per row, "b" vectors one per column.  What goes to global memory
  // goes there behind the second barrier: a barrier waits for the stores before it.
  cluster_wait();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this CTA's column sums are there
  float sum[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) sum[j] = 0.f;
  auto add = [&](bool is_r, int k, float v) {
    const float q = rsqrtf(v + 1e-8f);
    if (is_r) { sum[k] += v; sum[3 + k] = fmaf(v, v, sum[3 + k]); sum[6 + k] = fmaf(q, q, sum[6 + k]); }
    else { sum[9 + k] = fmaf(v, v, sum[9 + k]); sum[12 + k] = fmaf(q, q, sum[12 + k]); }
  };
  __syncthreads();
  for (int i = tid; i < rows; i += SF_NT) {
    const float mean = s_rs[i] / (float)Y;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = lerp_torch(i == tid ? old_a[k] : d.fac_a[(int64_t)k * X + row0 + i], mean, prm.w_f[k]);
      s_fa[k * shape.rows + i] = v;
      add(r_is_a, k, v);
    }
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int y = col0 + tid; y < col1; y += SF_NT) {
    float s = 0.f;
#pragma unroll 16
    for (int q = 0; q < parts; ++q) s += cluster_load(&s_col[y], q);
    const float mean = s / (float)X;
    s_sum[y - col0] = s;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = lerp_torch(y == col0 + tid ? old_b[k] : d.fac_b[(int64_t)k * Y + y], mean, prm.w_f[k]);
      s_fb[k * shape.cols + y] = v;
      add(!r_is_a, k, v);
    }
  }
  const int busy = min(WARPS, (max(rows, col1 - col0) + 31) / 32);   // warps that have added anything up
  if (tid < 32 * busy) {
    const float v = warp_fold<0, 16>(sum);
    if (lane < NS) s_warp[tid >> 5][lane] = v;
  }
  __syncthreads();
  if (tid < NS * 16) {   // entry j for CTA q
    const int j = tid / 16, q = tid % 16;
    float v = 0.f;
    for (int w = 0; w < busy; ++w) v += s_warp[w][j];
    if (q < parts) cluster_store(&s_cta[rank][j], q, v);
  }
  for (int e = tid; e < 3 * (col1 - col0) * (parts - 1); e += SF_NT) {   // the accumulators of this CTA's columns, for the others
    const int c = e % (col1 - col0), kq = e / (col1 - col0), k = kq % 3, q = kq / 3;
    float* const at = &s_fb[k * shape.cols + col0 + c];
    cluster_store(at, q + (q >= rank), *at);
  }
  cluster_sync();   // nobody looks into another CTA any more
  if (tid < NS) {
    float v = 0.f;
#pragma unroll 16
    for (int q = 0; q < parts; ++q) v += s_cta[q][tid];
    s_tot[tid] = v;
  }
  __syncthreads();
  const bool whole = d.rcm_pre == 3;   // the row factor's mean is over the vector, or over an entry's three decays
  auto factors = [&](bool is_r, int64_t L, float* at, int stride, float* fac, float* f_out, bool store, float (&f)[3]) {
    const float v[3] = {at[0], at[stride], at[2 * stride]};
    const float own = is_r ? (v[0] + v[1] + v[2]) / 3.0f : 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f[k] = is_r ? safe_rsqrt(v[k] / ((whole ? s_tot[k] / (float)L : own) + 1e-9f)) : safe_rsqrt(v[k]);
      at[k * stride] = f[k];
      if (store) { fac[k * L] = v[k]; f_out[k * L] = f[k]; }
    }
  };
  for (int i = tid; i < rows; i += SF_NT) {
    float f[3];
    factors(r_is_a, X, s_fa + i, shape.rows, d.fac_a + row0 + i, d.f_a + row0 + i, true, f);
    d.sum_a[row0 + i] = s_rs[i];
    if (d.fx) st4(d.fx + 4 * (int64_t)(row0 + i), make_float4(f[0], f[1], f[2], 0.f));
  }
  for (int y = tid; y < Y; y += SF_NT) {   // every CTA all columns
    float f[3];
    const bool mine = y >= col0 && y < col1;
    factors(!r_is_a, Y, s_fb + y, shape.cols, d.fac_b + y, d.f_b + y, mine, f);
    if (mine) d.sum_b[y] = s_sum[y - col0];
  }
  if (rank == 0 && tid < PYLO_STAT_STRIDE) {   // closed forms, see k_factor_update
    const float mult_r = (float)(r_is_a ? Y : X), mult_c = (float)(r_is_a ? X : Y);
    float v = 0.f;
    if (tid >= F::R && tid < F::R + 3) v = s_tot[3 + tid - F::R] * mult_r;
    else if (tid >= F::RR && tid < F::RR + 3) v = s_tot[6 + tid - F::RR] * mult_r;
    else if (tid >= F::C && tid < F::C + 3) v = s_tot[9 + tid - F::C] * mult_c;
    else if (tid >= F::RC && tid < F::RC + 3) v = s_tot[12 + tid - F::RC] * mult_c;
    d.closed[tid] = v;
  }
  // ---- B: state and sums of squares, as in k_state_moments
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const bool near = fabsf(prm.w_m[0]) < 0.5f && fabsf(prm.w_m[1]) < 0.5f && fabsf(prm.w_m[2]) < 0.5f && fabsf(prm.w_v) < 0.5f;
  if (fast && near) {
    // Bound by issue slots (a tensor has sixteen SMs at most): four elements of a row at once, two in each packed instruction.
    uint64_t acc2[NACC];
#pragma unroll
    for (int j = 0; j < NACC; ++j) acc2[j] = 0ull;
    const uint64_t w0 = pack2(prm.w_m[0], prm.w_m[0]), w1 = pack2(prm.w_m[1], prm.w_m[1]), w2 = pack2(prm.w_m[2], prm.w_m[2]);
    const uint64_t wv = pack2(prm.w_v, prm.w_v), epsv = pack2(prm.eps_v, prm.eps_v), minus = pack2(-1.f, -1.f);
    auto lerp2 = [&](uint64_t from, uint64_t to, uint64_t w) { return fma2(w, fma2(from, minus, to), from); };   // lerp_torch, |w| < 0.5
    auto square2 = [&](int j, uint64_t f) { acc2[j] = fma2(f, f, acc2[j]); };
    int r = tid * 4 / Y, y = tid * 4 - r * Y;
    const int dr = SF_NT * 4 / Y, dy = SF_NT * 4 - dr * Y;
    for (int i = tid * 4; i < cnt; i += SF_NT * 4) {
      const uint64_t fa[3] = {pack2(s_fa[r], s_fa[r]), pack2(s_fa[shape.rows + r], s_fa[shape.rows + r]), pack2(s_fa[2 * shape.rows + r], s_fa[2 * shape.rows + r])};
      auto four = [](const float* at) { return *reinterpret_cast<const ulonglong2*>(at); };
      const ulonglong2 g4 = four(s_g + i), p4 = four(s_p + i), b0 = four(s_fb + y), b1 = four(s_fb + shape.cols + y), b2 = four(s_fb + 2 * shape.cols + y);
      ulonglong2 m04 = four(s_m0 + i), m14 = four(s_m1 + i), m24 = four(s_m2 + i), v4 = four(s_v + i);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        auto half = [&](auto& q) -> auto& { return h ? q.y : q.x; };
        const uint64_t g = half(g4), p = half(p4);
        auto &m0 = half(m04), &m1 = half(m14), &m2 = half(m24), &v = half(v4);
        if constexpr (FAM == PYLO_FAM_VELO) {
          constexpr int B = F::NF;
          acc2[B] = add2(acc2[B], m0); acc2[B + 1] = add2(acc2[B + 1], m1); acc2[B + 2] = add2(acc2[B + 2], m2); acc2[B + 6] = add2(acc2[B + 6], v);
          square2(B + 3, m0); square2(B + 4, m1); square2(B + 5, m2); square2(B + 7, v);
        }
        m0 = lerp2(m0, g, w0);
        m1 = lerp2(m1, g, w1);
        m2 = lerp2(m2, g, w2);
        v = lerp2(v, fma2(g, g, epsv), wv);
        float va, vb;
        unpack2(v, va, vb);
        const uint64_t rs = pack2(rsqrtf(va + prm.eps_feat), rsqrtf(vb + prm.eps_feat));
        const uint64_t k0 = mul2(fa[0], half(b0)), k1 = mul2(fa[1], half(b1)), k2 = mul2(fa[2], half(b2));
        if constexpr (FAM == PYLO_FAM_ADAFAC) {   // the order of elem_features
          square2(0, g); square2(1, p); square2(2, m0); square2(3, m1); square2(4, m2); square2(5, v);
          square2(6, mul2(m0, rs)); square2(7, mul2(m1, rs)); square2(8, mul2(m2, rs)); square2(9, rs);
          square2(10, mul2(k0, g)); square2(11, mul2(k1, g)); square2(12, mul2(k2, g));
          square2(25, mul2(k0, m0)); square2(26, mul2(k1, m1)); square2(27, mul2(k2, m2));
        } else {
          float ga, gb;
          unpack2(g, ga, gb);
          square2(0, g); square2(1, pack2(fminf(fmaxf(ga, -0.1f), 0.1f), fminf(fmaxf(gb, -0.1f), 0.1f)));
          square2(2, p); square2(3, m0); square2(4, m1); square2(5, m2); square2(6, v);
          square2(7, mul2(m0, rs)); square2(8, mul2(m1, rs)); square2(9, mul2(m2, rs)); square2(10, rs);
          square2(11, mul2(k0, g)); square2(12, mul2(k1, g)); square2(13, mul2(k2, g)); square2(14, mul2(g, rs));
          square2(27, mul2(k0, m0)); square2(28, mul2(k1, m1)); square2(29, mul2(k2, m2));
        }
      }
      *reinterpret_cast<ulonglong2*>(m0p + i) = m04;
      *reinterpret_cast<ulonglong2*>(m1p + i) = m14;
      *reinterpret_cast<ulonglong2*>(m2p + i) = m24;
      *reinterpret_cast<ulonglong2*>(vp + i) = v4;
      r += dr;
      y += dy;
      if (y >= Y) { y -= Y; ++r; }
    }
#pragma unroll
    for (int j = 0; j < NACC; ++j) {
      float a, b;
      unpack2(acc2[j], a, b);
      acc[j] = a + b;
    }
  } else {
    int r = tid / Y, y = tid - r * Y;
    const int dr = SF_NT / Y, dy = SF_NT - dr * Y;
    for (int i = tid; i < cnt; i += SF_NT) {
      const float g = s_g[i];
      float m0 = s_m0[i], m1 = s_m1[i], m2 = s_m2[i], v = s_v[i];
      velo_stats<FAM>(acc, m0, m1, m2, v);
      m0 = lerp_torch(m0, g, prm.w_m[0]);
      m1 = lerp_torch(m1, g, prm.w_m[1]);
      m2 = lerp_torch(m2, g, prm.w_m[2]);
      v = lerp_torch(v, g * g + prm.eps_v, prm.w_v);
      m0p[i] = m0; m1p[i] = m1; m2p[i] = m2; vp[i] = v;
      float f[F::NF];
      elem_features<FAM>(f, g, s_p[i], m0, m1, m2, v, rsqrtf(v + prm.eps_feat), s_fa[r] * s_fb[y], s_fa[shape.rows + r] * s_fb[shape.cols + y],
                         s_fa[2 * shape.rows + r] * s_fb[2 * shape.cols + y]);
      accumulate<FAM, false>(acc, f);
      r += dr;
      y += dy;
      if (y >= Y) { y -= Y; ++r; }
    }
  }
  block_reduce_store<NACC, WARPS>(acc, s_red, out);
  if (tid >= NACC && tid < PYLO_STAT_STRIDE) out[tid] = 0.f;
}
