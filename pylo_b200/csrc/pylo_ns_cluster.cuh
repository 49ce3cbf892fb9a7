// The whole Newton-Schulz chain of a matrix of up to 128 rows (its shorter side) in one launch: a cluster of CTAs keeps the
// matrix in shared memory and registers for all rounds (included by pylo_kernels.cu after pylo_ns_f16.cuh, whose operands, their
// scales and their three products of fp16 planes it shares).
//
// A small matrix pays for latency only.  As a chain of launches (k_gemm_f16x2*) every product of 128 x 784 takes 8 to 9 us to
// fetch its operands, multiply for less than one and write the result for the next launch, fifteen times in a row.  Here
// CTA q of the cluster owns up to 192 columns of x: their fp32 values in registers, their two planes in shared memory, where
// they are operand A and B (K-major) of a = x x^T and operand B (MN-major) of b x.  Per round:
//   * every CTA multiplies its columns with themselves; the cluster adds the partial sums up, CTA q the q-th part of a's columns
//     in rank order, and hands the sums to everyone: two exchanges through distributed shared memory;
//   * every CTA makes b = c1 a + c2 a a by itself (a third exchange would cost more than its 24 products of 64 cycles), and
//     x' = c0 x + b x of its columns, on registers.
// What bounds it: latency again, but of shared memory.  A round of 128 x 784 takes 12.5 us: 7.5 for three series of products of
// 0.8 us with their operands' conversion, 5 for the exchanges.  The chain takes 64 us (155 as launches), 128 x 128 37 (122), 48
// matrices of 128 x 128 to 128 x 512 77 (227).
#pragma once

#define NC_THREADS 512
#define NC_COLS 192              // columns of a CTA at most (COLS of the kernel: 128 where no matrix of the launch needs more)
#define NC_SIDE 128              // rows at most
#define NC_XBOX(cb, rb) (((cb) * 2 + (rb)) * NF_BOX)   // 64 x 64 boxes of a plane: two of rows side by side, then on to the next 64 columns

template <int COLS>
struct NcSmem {
  unsigned char x[2][NC_XBOX(COLS / 64, 0)];   // planes of this CTA's columns
  unsigned char m[2][NC_XBOX(NC_SIDE / 64, 0)];   // planes of a, then of b
  float part[NC_SIDE * NC_SIDE];                  // [column][row]: this CTA's share of a, then the sums
  float red[40];
  float sumsq[16];                                // of the CTAs' columns
  int sent[16];                                   // by the cluster's CTAs, at the end: 2 x rounds of copies, + 1 after a wait that ran out
  uint64_t bar, got[2], free;
  uint32_t tmem_base;
  volatile int abort;
};

// parts: CTAs that share a matrix; 0: one CTA runs it in plain fp32 (ns_small_body).  An item's CTAs start with a cluster.
struct nc_item { const float* x; float* out; int rows, cols, batch, parts, cta0; float c0, c1, c2, eps; };
struct nc_group { nc_item p[NF_GROUP]; int n, iters; };

__device__ __forceinline__ void nc_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// 16 neighbouring values of a row, times scale, into both planes (K-major boxes, 128-byte swizzle)
__device__ __forceinline__ void nc_put16(unsigned char* hi_plane, unsigned char* lo_plane, int row, int col, const float* v, float scale) {
  const int at = NC_XBOX(col >> 6, row >> 6) + (row & 63) * 128;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    __align__(16) __half2 hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {   // two at a time: single conversions to fp16 run at a fraction of the rate
      const float a = v[8 * h + 2 * j] * scale, b = v[8 * h + 2 * j + 1] * scale;
      hi[j] = __floats2half2_rn(a, b);
      const float2 back = __half22float2(hi[j]);
      lo[j] = __floats2half2_rn(a - back.x, b - back.y);
    }
    const int piece = at + (((((col & 63) >> 3) + h) ^ (row & 7)) << 4);
    *reinterpret_cast<uint4*>(hi_plane + piece) = *reinterpret_cast<const uint4*>(hi);
    *reinterpret_cast<uint4*>(lo_plane + piece) = *reinterpret_cast<const uint4*>(lo);
  }
}

template <int COLS>
__global__ void __launch_bounds__(NC_THREADS, 1) k_ns_cluster(const __grid_constant__ nc_group grp, int* __restrict__ status) {
  extern __shared__ unsigned char nc_raw[];
  using Smem = NcSmem<COLS>;
  Smem& sm = *reinterpret_cast<Smem*>(nc_raw + ((1024 - (smem_addr(nc_raw) & 1023)) & 1023));   // at the same place in every CTA
  constexpr float S = 4096.f;   // of all planes, see ns_chain
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int k = 0;
  while (k + 1 < grp.n && (int)blockIdx.x >= grp.p[k + 1].cta0) ++k;
  const nc_item& it = grp.p[k];
  const int parts = max(1, it.parts), cta = blockIdx.x - it.cta0, matrix = cta / parts, rank = cta % parts;
  const uint32_t first = cluster_rank() - rank;   // the matrix's CTAs are `first` to `first` + parts - 1 of the cluster
  if (tid == 0) {
    mbar_init(&sm.bar, 1);
    mbar_init(&sm.got[0], 1);
    mbar_init(&sm.got[1], 1);
    mbar_init(&sm.free, max(1, parts - 1));
    sm.abort = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  cluster_arrive();   // waited for below: then every CTA of the cluster runs and its barriers are there
  if (warp == 1) { tc_alloc(&sm.tmem_base, 512); tc_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);   // two accumulators of COLS columns
  const bool tall = it.rows > it.cols;
  const int r = tall ? it.cols : it.rows, c = tall ? it.rows : it.cols;
  const int nr = (r + 31) & ~31, cs = ((c + parts - 1) / parts + 15) & ~15, k0 = rank * cs;
  const long long base = (long long)matrix * r * c;
  // this thread: row `row` of x, of a and of b; of x the 16 columns from 16 (group + 4 q), of a and b the 32 from 32 group
  const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane;
  const bool rows_here = quarter * 32 < nr, mine = rows_here && 32 * group < nr;   // the same for the whole warp
  const uint32_t t_row = tmem + ((uint32_t)(quarter * 32) << 16);
  pdl_begin();
  const bool busy = matrix < it.batch;              // the others fill the item's last cluster up
  const bool shared = busy && it.parts > 0;
  float xr[COLS / 64][16], acc = 0.f;
#pragma unroll
  for (int q = 0; q < COLS / 64; ++q) {
    const int col = 16 * (group + 4 * q), kk = k0 + col;
#pragma unroll
    for (int j = 0; j < 16; ++j) xr[q][j] = 0.f;
    if (shared && row < r && col < cs) {
      if (tall) {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (kk + j < c) xr[q][j] = it.x[base + (long long)(kk + j) * r + row];
      } else {
        const float* p = it.x + base + (long long)row * c + kk;
        if ((c & 3) == 0) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (kk + j < c) { const float4 v = ld4(p + j); xr[q][j] = v.x; xr[q][j + 1] = v.y; xr[q][j + 2] = v.z; xr[q][j + 3] = v.w; }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) if (kk + j < c) xr[q][j] = p[j];
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) acc = fmaf(xr[q][j], xr[q][j], acc);
    }
  }
  if (shared) acc = block_sum(acc, sm.red);
  else if (busy)
    ns_small_body<NC_THREADS>(it.x + base, it.out + base, it.rows, it.cols, grp.iters, it.c0, it.c1, it.c2, it.eps, reinterpret_cast<float*>(&sm), sm.red);
  cluster_wait();
  // A wait that runs out is one answer for the warp (`dead`), which waits for nothing from then on.  The first warp, which issues
  // the CTA's products and copies and speaks to the other CTAs, does none of that any more either: so every barrier has had
  // exactly as many arrivals and bytes as `products` and the CTAs' `sent` say, and what is still in flight can be waited for.
  uint32_t parity = 0, exchanged = 0, freed = 0;
  int products = 0, sent = 0;
  bool dead = false;
  auto wait = [&](uint64_t* bar, uint32_t phase) {
    if (!dead) dead = !__all_sync(0xffffffffu, ns_wait(bar, phase, &sm.abort));
  };
  // Told to the others: this CTA has read what they sent.  wait_free: all of them have said so.
  auto say_free = [&]() {
    if (warp == 0 && !dead && lane < parts && lane != rank)
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(nf_at_rank(&sm.free, first + lane)) : "memory");
  };
  auto wait_free = [&]() {
    wait(&sm.free, freed);
    __syncwarp();
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    freed ^= 1;
  };
  if (shared) {
  double tot = (double)acc;
  if (parts > 1) {
    if (warp == 0 && lane < parts)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(nf_at_rank(&sm.sumsq[rank], first + lane)), "f"(acc) : "memory");
    __syncthreads();   // this CTA's own is there
    say_free();
    wait_free();
    tot = 0.0;
    for (int p = 0; p < parts; ++p) tot += (double)sm.sumsq[p];
  }
  const float f = 1.0f / (sqrtf((float)tot) + it.eps);
#pragma unroll
  for (int q = 0; q < COLS / 64; ++q)
#pragma unroll
    for (int j = 0; j < 16; ++j) xr[q][j] *= f;

  const float c0 = it.c0, c1 = it.c1, c2 = it.c2;
  const int per = nr / parts, block = per * NC_SIDE;   // columns of a that a CTA adds up (nr is a multiple of 32, parts 1, 2, 4, 8 or 16), in floats
  auto put_x = [&]() {
#pragma unroll
    for (int q = 0; q < COLS / 64; ++q) {
      const int col = 16 * (group + 4 * q);
      if (rows_here && col < cs) nc_put16(sm.x[0], sm.x[1], row, col, xr[q], S);
    }
  };
  // Three products per K step of 16 (lo hi, hi lo, hi hi), of the first half of the contraction into one accumulator, of the
  // second into the other: the tensor core truncates when it accumulates, sums16 adds the two with round-to-nearest (error
  // of the chain on 128 x 784 1.9e-6, with one accumulator 3.3e-6, as of the chain of launches).  b_mn: operand B's contraction index is its slow one.
  auto multiply = [&](const unsigned char* a_hi, const unsigned char* a_lo, const unsigned char* b_hi, const unsigned char* b_lo, int n, int ksteps, bool b_mn) {
    fence_async_smem();   // the operands were written through the generic proxy
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && !dead) {
      ++products;
      if (elect_one()) {
        tc_fence_after();
        const uint32_t ah = smem_addr(a_hi), al = smem_addr(a_lo), bh = smem_addr(b_hi), bl = smem_addr(b_lo);
        const uint32_t idesc = nf_idesc(NC_SIDE, n, 0, b_mn);
        auto series = [&](uint32_t pa, uint32_t pb, int half, int k0, int k1, bool first) {
          for (int ks = k0; ks < k1; ++ks) {
            const uint32_t oa = NC_XBOX(ks >> 2, 0) + (ks & 3) * 32, ob = b_mn ? (ks >> 2) * NF_BOX + (ks & 3) * 2048 : oa;
            uint64_t db = nf_desc(pb + ob, 0);
            if (b_mn) db = (db & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(NC_XBOX(1, 0) >> 4) << 16);   // its boxes of 64 columns
            nf_mma<false>(tmem + half * COLS, nf_desc(pa + oa, 0), db, idesc, first && ks == k0 ? 0u : 1u);
          }
        };
        const int mid = (ksteps + 1) / 2;
        for (int half = 0; half < 2; ++half) {
          const int from = half ? mid : 0, to = half ? ksteps : mid;
          series(al, bh, half, from, to, true);
          series(ah, bl, half, from, to, false);
          series(ah, bh, half, from, to, false);
        }
        tc_commit(&sm.bar);
      }
      __syncwarp();
    }
    wait(&sm.bar, parity);
    parity ^= 1;
    __syncwarp();
    tc_fence_after();
  };

  // 16 columns of this thread's row of a product of `ksteps` steps, eight at a time (registers)
  auto sums16 = [&](int col, bool two, auto&& use) {
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      uint32_t v[8], w[8];
      nc_ld8(t_row + col + h, v);
      if (two) nc_ld8(t_row + COLS + col + h, w);
      else {
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = 0u;
      }
      tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j) use(h + j, __uint_as_float(v[j]) + __uint_as_float(w[j]));
    }
  };
  // An exchange: piece p of `src` (pieces `step` floats apart) to place `rank` of `dst` in the p-th CTA, by bulk copies that arrive at
  // barrier `which` there; over when the other CTAs' pieces are here.  (Reads through distributed shared memory between cluster
  // barriers: two microseconds more per round.)
  auto send = [&](int which, const float* src, int step, float* dst) {
    asm volatile("fence.proxy.async;" ::: "memory");   // the pieces were written through the generic proxy
    __syncthreads();
    if (warp == 0 && !dead) {
      ++sent;
      if (lane == 0) nf_expect(&sm.got[which], (parts - 1) * block * 4);
      if (lane < parts && lane != rank)
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(nf_at_rank(dst + rank * block, first + lane)), "r"(smem_addr(src + lane * step)), "r"(block * 4), "r"(nf_at_rank(&sm.got[which], first + lane)) : "memory");
      __syncwarp();
    }
    wait(&sm.got[which], exchanged);
    __syncwarp();
  };

  // this thread's 32 columns of its row of a, then of b
  float av[32];
  auto put_m = [&]() {
    if (mine) {
      nc_put16(sm.m[0], sm.m[1], row, 32 * group, av, S);
      nc_put16(sm.m[0], sm.m[1], row, 32 * group + 16, av + 16, S);
    }
  };

  put_x();
  for (int round = 0; round < grp.iters; ++round) {
    // ---- a = x x^T
    multiply(sm.x[0], sm.x[1], sm.x[0], sm.x[1], nr, cs / 16, false);
    if (mine) {
#pragma unroll
      for (int h = 0; h < 32; h += 16) sums16(32 * group + h, cs > 16, [&](int j, float v) { av[h + j] = v * (1.0f / (S * S)); });
    }
    if (parts > 1) {
      if (round > 0) wait_free();   // the others are done with what this round's copies write to
      if (mine) {
#pragma unroll
        for (int j = 0; j < 32; ++j) sm.part[(32 * group + j) * NC_SIDE + row] = av[j];
      }
      send(0, sm.part, block, reinterpret_cast<float*>(sm.m));
      for (int e = tid; e < block / 4; e += NC_THREADS) {
        float4* const own = reinterpret_cast<float4*>(sm.part + rank * block) + e;
        const float4* const got = reinterpret_cast<const float4*>(sm.m) + e;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = 0; p < parts; ++p) {
          const float4 v = p == rank ? *own : got[p * (block / 4)];
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        *own = s;
      }
      send(1, sm.part + rank * block, 0, sm.part);
      exchanged ^= 1;
      if (mine) {
#pragma unroll
        for (int j = 0; j < 32; ++j) av[j] = sm.part[(32 * group + j) * NC_SIDE + row];
      }
    }
    // ---- b = c1 a + c2 a a
    put_m();
    if (c2 != 0.f) {
      multiply(sm.m[0], sm.m[1], sm.m[0], sm.m[1], nr, nr / 16, false);
      if (mine) {
#pragma unroll
        for (int h = 0; h < 32; h += 16) sums16(32 * group + h, true, [&](int j, float v) { av[h + j] = fmaf(c2 / (S * S), v, c1 * av[h + j]); });
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) av[j] *= c1;
    }
    put_m();
    // ---- x' = c0 x + b x
    multiply(sm.m[0], sm.m[1], sm.x[0], sm.x[1], cs, nr / 16, true);
    if (parts > 1 && round + 1 < grp.iters) say_free();   // a's sums are read, and so is b: the next round's copies may come
#pragma unroll
    for (int q = 0; q < COLS / 64; ++q) {
      const int col = 16 * (group + 4 * q);
      if (rows_here && col < cs) sums16(col, true, [&](int j, float v) { xr[q][j] = fmaf(v, 1.0f / (S * S), c0 * xr[q][j]); });
    }
    if (round + 1 < grp.iters) put_x();
  }
#pragma unroll
  for (int q = 0; q < COLS / 64; ++q) {
    const int col = 16 * (group + 4 * q), kk = k0 + col;
    if (row < r && col < cs) {
      if (tall) {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (kk + j < c) it.out[base + (long long)(kk + j) * r + row] = xr[q][j];
      } else {
        float* p = it.out + base + (long long)row * c + kk;
        if ((c & 3) == 0) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (kk + j < c) st4(p + j, make_float4(xr[q][j], xr[q][j + 1], xr[q][j + 2], xr[q][j + 3]));
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) if (kk + j < c) p[j] = xr[q][j];
        }
      }
    }
  }
  }
  // After a wait that ran out nothing may be on its way when a CTA leaves: neither this CTA's products, nor copies into its shared
  // memory, nor copies out of another's.  All CTAs say what they have sent; behind the barrier, where nobody sends any more, the
  // failed ones take in what is theirs, and all of them stay until that is done.  A copy belongs to the phase of `got` that this
  // CTA announced last, or to the next one, which it has not announced: another CTA is at most one round of copies ahead,
  // and then only if the last announced phase is complete.
  if (warp == 0 && lane < (int)cluster_size()) cluster_store(&sm.sent[cluster_rank()], lane, 2 * sent + (dead ? 1 : 0));
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // no CTA leaves while another may write to its shared memory
  if (__any_sync(0xffffffffu, lane < (int)cluster_size() && (sm.sent[lane] & 1))) {   // the same in all CTAs of the cluster
    if (warp == 0 && dead) {
      if (products) pipe_wait(&sm.bar, (uint32_t)(products - 1) & 1);
      const int bytes = ((r + 31) & ~31) / parts * NC_SIDE * 4;
      for (int which = 0; which < 2 && parts > 1; ++which) {
        const int own = (sent + 1 - which) / 2;
        const int theirs = lane < parts && lane != rank ? ((sm.sent[first + lane] >> 1) + 1 - which) / 2 : own;
        const int missing = __popc(__ballot_sync(0xffffffffu, theirs < own)), ahead = __popc(__ballot_sync(0xffffffffu, theirs > own));
        if (missing && lane == 0)   // these never come
          asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.got[which])), "r"(missing * bytes) : "memory");
        if (own) pipe_wait(&sm.got[which], (uint32_t)(own - 1) & 1);
        if (ahead && lane == 0) nf_expect(&sm.got[which], ahead * bytes);
        if (ahead) pipe_wait(&sm.got[which], (uint32_t)own & 1);
      }
    }
    cluster_sync();
  }
  if (tid == 0 && sm.abort && status) atomicOr(status, 4);
  if (warp == 1) tc_dealloc(tmem, 512);
}
