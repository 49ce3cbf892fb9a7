// The Newton-Schulz chain of the CELO2 family on fp16 tensor-core products of split operands (included by pylo_kernels.cu
// after pylo_ns_gemm.cuh, whose helpers it uses).
//
//   C[b] = alpha * A[b] B[b]^T + beta * D[b]
//
// Every matrix of the iteration (CELO2_naive.py:59-73: a = x x^T, b = c1 a + c2 a a, x = c0 x + b x) is bounded by a small
// number in norm, because x starts with norm 1, so a matrix can be kept as TWO fp16 PLANES, hi = fp16(s v) and
// lo = fp16(s v - hi) with one power of two s: 11 + 11 significant bits, the same as a TF32 high and low part, and nothing
// below 2^-25 / s is lost.  Three products per K step (lo hi, hi lo, hi hi) give the fp32 product, as with TF32, at twice the
// rate of the tensor core, and because the producing kernel's epilogue writes the planes, operands reach shared memory by
// TMA as they are: no loader warps, no split in the main loop (the loaders' split and its shared-memory traffic were what
// bound the TF32 kernel, 60 % of its tensor rate).
//
// fp16 operands may also be read "MN-major" (the contraction index is the slow one), so neither x^T nor a transposed
// input or output is ever made: for a wide x (rows <= columns) a = x x^T, x' = b x; for a tall one a = x^T x, x' = x b.
// The products x x^T and a a are symmetric: only tiles that reach the diagonal or lie above it are computed, and the
// epilogue stores every element at its mirror place too.
//
// The same product of several stacks of matrices (a model has one stack per shape) goes into one launch: the tiles of all of
// them are dealt over the SMs together, and a model of small matrices pays for one chain of launches, not one per shape.
//
// One persistent CTA per SM, eighteen warps: one lane issues the TMA copies, one lane the products (K steps of 16), sixteen
// warps run the epilogue (its instructions wait for one another; eight warps were too few to hide that under a product with a
// short K: chain on 12 x 768 x 3072 1317 us with eight, 1229 with sixteen; 4 x 768 x 3072 656 and 547).  The tensor core truncates when it accumulates, so the contraction is cut into
// chunks of 256 that start from zero, alternating between two accumulators of 256 columns; the epilogue warps add the
// chunks up with round-to-nearest in registers (64 per thread) while the next chunk is multiplied.  Results leave through
// shared memory, 16 columns at a time, so that a warp's loads and stores cover whole sectors of four rows (straight from
// the accumulator layout, a row per lane, they touch 32 lines each and bound every product with K < 1000).
//
// What binds it: the tensor pipe (a pair: 12 products of 128 cycles per 64 KB stage), tile quantisation, and below K = 1000 a
// tile's way out.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#define NF_BM 128
#define NF_BK 64
#define NF_EPI_WARPS 16
#define NF_THREADS ((NF_EPI_WARPS + 2) * 32)
#define NF_CHUNK_BLOCKS 4       // K blocks per accumulation chunk (256 terms)
#define NF_BOX 8192             // bytes of one TMA box: 64 x 64 fp16
#define NF_GROUP 8              // products of one launch at most

// PAIR: two CTAs on two SMs share a tile of 256 x 256 (cta_group::2): each holds its own 128 rows of A and one half of B's
// columns, and the tensor cores of both read both halves.  Per product and SM a third less operand data crosses from L2 than
// for a tile of 128 x 256 (64 instead of 96 KB per 64 terms; at that rate L2 is what binds), and a third stage fits.
template <int BN, bool PAIR>
struct NfSmem {   // per stage: A hi, A lo (128 x 64 each), B hi, B lo (BN x 64 each, of a pair one half)
  static constexpr int STAGES = 3;   // of 64 KB
  static constexpr int BROWS = PAIR ? BN / 2 : BN;
  unsigned char st[STAGES][2 * (NF_BM / 64) * NF_BOX + 2 * (BROWS / 64) * NF_BOX];
  float out[NF_EPI_WARPS][32 * 16];   // per epilogue warp: 32 rows x 16 columns on their way out
  uint64_t full[STAGES], empty[STAGES], acc_ready[2], acc_free[2], parts;
  uint32_t tmem_base;
  volatile int abort;
};

struct nf_args {
  float* C;               // fp32 result [batch][M][ldc], or NULL
  const float* D;         // [batch][M][ldd], or NULL
  const float* d_scale;   // [batch]: beta is multiplied by it; or NULL
  __half* P;              // planes of the result, [2][batch][M][ldp], or NULL
  long long sC, sD, sP;   // batch strides in elements
  long long planeP;       // distance between the two planes
  int M, N, K, ldc, ldd, ldp, batch;
  float alpha, beta, scale;   // scale: of the planes written
  int a_mn, b_mn;         // operand stored with the contraction index as rows
  int symmetric;
  int per, tile0;         // tiles per matrix, and of the products before this one in the launch
};
struct nf_problem { CUtensorMap A, B; nf_args g; };
struct nf_group { nf_problem p[NF_GROUP]; int n, tiles; };

__device__ __forceinline__ void nf_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void nf_tma(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int b, int plane) {
  if constexpr (PAIR)   // the barrier may be the other CTA's
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(b), "r"(plane) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(b), "r"(plane) : "memory");
}
// the address of another CTA's copy of a shared variable
__device__ __forceinline__ uint32_t nf_at_rank(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void nf_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// four columns (quad 0..3) of a row of a warp's 32 x 16 stage; neighbouring rows' quads are spread over the banks
__device__ __forceinline__ float* nf_out(float* stage, int row, int quad) { return stage + row * 16 + 4 * (quad ^ ((row >> 1) & 3)); }
template <bool PAIR>
__device__ __forceinline__ void nf_commit(uint64_t* bar) {
  if constexpr (PAIR)   // arrives at the barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)), "h"((uint16_t)3) : "memory");
  else
    tc_commit(bar);
}
// descriptor of a 128-byte-swizzled operand of 64 x 64 boxes.  K-major: rows of 64 k, 8-row groups 1024 bytes apart (boxes
// follow one another).  MN-major: rows are k, a row holds 64 mn; 8-k groups 1024 bytes apart, 64-mn boxes NF_BOX apart.
__device__ __forceinline__ uint64_t nf_desc(uint32_t saddr, int mn) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)(mn ? NF_BOX >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
template <bool PAIR>
__device__ __forceinline__ void nf_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// fp32 accumulate, fp16 x fp16, M = 128 or (a pair) 256
__device__ __forceinline__ uint32_t nf_idesc(uint32_t m, uint32_t n, int a_mn, int b_mn) {
  return (1u << 4) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// tiles of one matrix of BM x BN; symmetric: those whose columns are not all below the diagonal of their rows
template <int BM, int BN>
__host__ __device__ inline int nf_tiles_per_matrix(int M, int N, int symmetric) {
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  if (!symmetric) return tiles_m * tiles_n;
  int n = 0;
  for (int tm = 0; tm < tiles_m; ++tm) n += tiles_n - tm * BM / BN;
  return n;
}
template <int BM, int BN>
__device__ __forceinline__ void nf_tile_coords(int r, int M, int N, int symmetric, int& tm, int& tn) {
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  if (!symmetric) { tm = r / tiles_n; tn = r % tiles_n; return; }
  for (tm = 0; tm < tiles_m; ++tm) {
    const int first = tm * BM / BN, cnt = tiles_n - first;
    if (r < cnt) { tn = first + r; return; }
    r -= cnt;
  }
  tm = 0; tn = 0;
}

// SPLIT: the CTAs of a cluster share one tile, each with its part of the contraction; the first adds their sums up through
// distributed shared memory, in rank order, and carries on alone.  One tile per cluster.
template <int BN, bool PAIR, bool SPLIT>
__device__ __forceinline__ void nf_gemm_body(const nf_group& grp, int* __restrict__ status) {
  extern __shared__ unsigned char nf_raw[];
  using Smem = NfSmem<BN, PAIR>;
  constexpr int STAGES = Smem::STAGES, TILE_M = PAIR ? 2 * NF_BM : NF_BM;
  Smem& sm = *reinterpret_cast<Smem*>(nf_raw + ((1024 - (smem_addr(nf_raw) & 1023)) & 1023));   // at the same place in both CTAs of a pair
  constexpr int A_PLANE = (NF_BM / 64) * NF_BOX, B_PLANE = (Smem::BROWS / 64) * NF_BOX, STAGE = 2 * A_PLANE + 2 * B_PLANE;
  // the warp index as a broadcast from lane 0: the role branches are warp-uniform and the issuing branch keeps its
  // descriptors in uniform registers
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int rank = PAIR ? (int)cluster_rank() : 0;
  const int part = SPLIT ? (int)cluster_rank() : 0, parts = SPLIT ? (int)cluster_size() : 1;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&sm.acc_ready[s], 1); mbar_init(&sm.acc_free[s], (PAIR ? 2 : 1) * NF_EPI_WARPS); }
    if constexpr (SPLIT) mbar_init(&sm.parts, (parts - 1) * NF_EPI_WARPS);
    sm.abort = 0;
  }
  if (tid < 2 * grp.n) {   // the tensor maps' first use would wait for them
    const nf_problem& q = grp.p[tid >> 1];
    asm volatile("prefetch.tensormap [%0];" ::"l"((tid & 1) ? &q.B : &q.A) : "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)), "r"(512) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tc_alloc(&sm.tmem_base, 512);
      tc_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR || SPLIT) cluster_sync();   // the other CTAs' barriers exist
  tc_fence_after();
  pdl_begin();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);   // two accumulators of 256 columns
  const int n_tiles = grp.tiles, ctas = PAIR ? 2 : parts, first_tile = blockIdx.x / ctas, tile_step = gridDim.x / ctas;
  // the product a tile belongs to, and its place there
  auto locate = [&](int tile, int& b, int& tm, int& tn) -> const nf_problem& {
    int k = 0;
    while (k + 1 < grp.n && tile >= grp.p[k + 1].g.tile0) ++k;
    const nf_args& g = grp.p[k].g;
    const int r = tile - g.tile0;
    b = r / g.per;
    nf_tile_coords<TILE_M, BN>(r - b * g.per, g.M, g.N, g.symmetric, tm, tn);
    return grp.p[k];
  };

  // the K blocks of a tile that are this CTA's
  auto blocks = [&](const nf_args& g, int& kb0, int& kb1) {
    const int n_kb = (g.K + NF_BK - 1) / NF_BK, per = SPLIT ? (n_kb + parts - 1) / parts : n_kb;
    kb0 = SPLIT ? min(part * per, n_kb) : 0;
    kb1 = SPLIT ? min(kb0 + per, n_kb) : n_kb;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    if (elect_one()) {
      asm volatile("fence.proxy.async;" ::: "memory");   // what earlier kernels stored is read through the async proxy
      long long kbc = 0;
      bool dead = false;
      for (int tile = first_tile; tile < n_tiles && !dead && !sm.abort; tile += tile_step) {
        int b, tm, tn;
        const nf_problem& q = locate(tile, b, tm, tn);
        const int a_mn = q.g.a_mn, b_mn = q.g.b_mn;
        int kb0, kb1;
        blocks(q.g, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb, ++kbc) {
          const int s = (int)(kbc % STAGES);
          const long long use = kbc / STAGES;
          if (use > 0 && !ns_wait(&sm.empty[s], (uint32_t)((use - 1) & 1), &sm.abort)) { dead = true; break; }
          // boxes that reach beyond the matrix are filled with zeros and count in full; of a pair the first CTA's barrier
          // takes the bytes of both
          if (rank == 0) nf_expect(&sm.full[s], (PAIR ? 2 : 1) * STAGE);
          const uint32_t bar = PAIR ? nf_at_rank(&sm.full[s], 0) : smem_addr(&sm.full[s]);
          uint32_t dst = smem_addr(sm.st[s]);
          const int k = kb * NF_BK;
          for (int plane = 0; plane < 2; ++plane)
#pragma unroll
            for (int u = 0; u < NF_BM / 64; ++u, dst += NF_BOX) {
              const int mn = tm * TILE_M + rank * NF_BM + 64 * u;
              nf_tma<PAIR>(dst, &q.A, bar, a_mn ? mn : k, a_mn ? k : mn, b, plane);
            }
          for (int plane = 0; plane < 2; ++plane)
#pragma unroll
            for (int u = 0; u < Smem::BROWS / 64; ++u, dst += NF_BOX) {
              const int mn = tn * BN + rank * Smem::BROWS + 64 * u;
              nf_tma<PAIR>(dst, &q.B, bar, b_mn ? mn : k, b_mn ? k : mn, b, plane);
            }
        }
      }
      // the CTA must not end while a copy into its shared memory is in flight: normally the issuing lane has waited for
      // every stage; after an abort wait (bounded) for the stages filled last
      if (rank == 0 && (dead || sm.abort)) {
        for (long long f = kbc > STAGES ? kbc - STAGES : 0; f < kbc; ++f) {
          const uint32_t a = smem_addr(&sm.full[f % STAGES]);
          for (int it = 0; it < NS_SPIN_LIMIT; ++it) {
            uint32_t ok;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(a), "r"((uint32_t)((f / STAGES) & 1)) : "memory");
            if (ok) break;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products (of a pair the first CTA issues them)
    if (rank == 0 && elect_one()) {
      long long kbc = 0, cc = 0;
      bool dead = false;
      for (int tile = first_tile; tile < n_tiles && !dead && !sm.abort; tile += tile_step) {
        int b, tm, tn;
        const nf_problem& q = locate(tile, b, tm, tn);
        const int a_mn = q.g.a_mn, b_mn = q.g.b_mn;
        int kb0, kb1;
        blocks(q.g, kb0, kb1);
        const uint32_t idesc = nf_idesc(TILE_M, BN, a_mn, b_mn);
        const uint64_t a_step = (a_mn ? 2048 : 32) >> 4, b_step = (b_mn ? 2048 : 32) >> 4;   // 16 terms further along K
        for (int kb = kb0; kb < kb1; ++kb, ++kbc) {
          const int in_chunk = (kb - kb0) % NF_CHUNK_BLOCKS;
          const uint32_t acc = tmem + (uint32_t)(cc & 1) * 256;
          if (in_chunk == 0 && cc >= 2) {   // this accumulator's previous chunk must have been added up
            if (!ns_wait(&sm.acc_free[cc & 1], (uint32_t)(((cc >> 1) - 1) & 1), &sm.abort)) { dead = true; break; }
            tc_fence_after();
          }
          const int s = (int)(kbc % STAGES);
          if (!ns_wait(&sm.full[s], (uint32_t)((kbc / STAGES) & 1), &sm.abort)) { dead = true; break; }
          tc_fence_after();
          const uint32_t base = smem_addr(sm.st[s]);
          const uint64_t ah = nf_desc(base, a_mn), al = nf_desc(base + A_PLANE, a_mn);
          const uint64_t bh = nf_desc(base + 2 * A_PLANE, b_mn), bl = nf_desc(base + 2 * A_PLANE + B_PLANE, b_mn);
#pragma unroll
          for (int ks = 0; ks < NF_BK / 16; ++ks) nf_mma<PAIR>(acc, al + ks * a_step, bh + ks * b_step, idesc, (in_chunk > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
          for (int ks = 0; ks < NF_BK / 16; ++ks) nf_mma<PAIR>(acc, ah + ks * a_step, bl + ks * b_step, idesc, 1u);
#pragma unroll
          for (int ks = 0; ks < NF_BK / 16; ++ks) nf_mma<PAIR>(acc, ah + ks * a_step, bh + ks * b_step, idesc, 1u);
          nf_commit<PAIR>(&sm.empty[s]);
          if (in_chunk == NF_CHUNK_BLOCKS - 1 || kb == kb1 - 1) { nf_commit<PAIR>(&sm.acc_ready[cc & 1]); ++cc; }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue: a thread adds up a quarter of a row of the tile
    constexpr int COLS = BN * 4 / NF_EPI_WARPS;   // columns per thread
    const int quarter = warp & 3, col0 = ((warp - 2) >> 2) * COLS;
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    float* const stage = sm.out[warp - 2];
    const int sr = lane >> 2, sc = (lane & 3) * 4;   // on the way out: row sr + 8 i, columns sc .. sc + 3 of 16
    long long cc = 0;
    bool dead = false;
    for (int tile = first_tile; tile < n_tiles && !dead && !sm.abort; tile += tile_step) {
      int b, tm, tn;
      const nf_args& g = locate(tile, b, tm, tn).g;
      int kb0, kb1;
      blocks(g, kb0, kb1);
      const int n_chunks = (kb1 - kb0 + NF_CHUNK_BLOCKS - 1) / NF_CHUNK_BLOCKS;
      const int M = g.M, N = g.N, ldc = g.ldc, ldd = g.ldd, ldp = g.ldp, sym = g.symmetric;
      const int m0 = tm * TILE_M + rank * NF_BM + quarter * 32;
      const float alpha = g.alpha, scale = g.scale;
      float run[COLS];
      if (g.D && part == 0) {
        // beta D / alpha is what the sum starts from: read while the first products run.  alpha is a power of two where D is
        // large (x'), so nothing is rounded that would not be rounded at the end.
        const float f = (g.d_scale ? g.beta * g.d_scale[b] : g.beta) / alpha;
        const float* const D = g.D + (long long)b * g.sD;
        const bool dvec = (ldd & 3) == 0;
        // all of this thread's pieces are requested before the first is turned (they wait in the registers of the sum): four
        // loads in flight at a time kept the 12 products of 768 x 3072 with an addition at 209 us with eight epilogue warps, all
        // of them took 164 (147 with the present sixteen)
#pragma unroll
        for (int q = 0; q < COLS / 16; ++q) {
          const int n = tn * BN + col0 + 16 * q + sc;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int m = m0 + sr + 8 * i;
            float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m < M && n < N && (!sym || n + 3 >= m)) {
              const float* drow = D + (long long)m * ldd + n;
              if (dvec && n + 3 < ldd) d = ld4(drow);
              else {
                d.x = drow[0];
                if (n + 1 < N) d.y = drow[1];
                if (n + 2 < N) d.z = drow[2];
                if (n + 3 < N) d.w = drow[3];
              }
            }
            run[16 * q + 4 * i] = d.x; run[16 * q + 4 * i + 1] = d.y; run[16 * q + 4 * i + 2] = d.z; run[16 * q + 4 * i + 3] = d.w;
          }
        }
#pragma unroll
        for (int q = 0; q < COLS / 16; ++q) {   // from rows of four lanes to a row per lane
#pragma unroll
          for (int i = 0; i < 4; ++i)
            st4(nf_out(stage, sr + 8 * i, lane & 3), make_float4(run[16 * q + 4 * i], run[16 * q + 4 * i + 1], run[16 * q + 4 * i + 2], run[16 * q + 4 * i + 3]));
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const float4 d = ld4(nf_out(stage, lane, h));
            run[16 * q + 4 * h] = f * d.x; run[16 * q + 4 * h + 1] = f * d.y; run[16 * q + 4 * h + 2] = f * d.z; run[16 * q + 4 * h + 3] = f * d.w;
          }
          __syncwarp();
        }
      } else {
#pragma unroll
        for (int j = 0; j < COLS; ++j) run[j] = 0.f;
      }
      for (int c = 0; c < n_chunks; ++c, ++cc) {
        if (!ns_wait(&sm.acc_ready[cc & 1], (uint32_t)((cc >> 1) & 1), &sm.abort)) { dead = true; break; }
        tc_fence_after();
        const uint32_t t_acc = t_lane + (uint32_t)(cc & 1) * 256;
#pragma unroll
        for (int q = 0; q < COLS / 16; ++q) {
          uint32_t v[16];
          nf_ld16(t_acc + 16 * q, v);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) run[16 * q + j] += __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (PAIR) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(nf_at_rank(&sm.acc_free[cc & 1], 0)) : "memory");
          else ns_arrive(&sm.acc_free[cc & 1]);
        }
      }
      if (dead) break;
      if constexpr (SPLIT) {
        // the stages are free: this CTA's products are done.  A thread's sums, four floats of a warp's lanes side by side
        float4* const box = reinterpret_cast<float4*>(sm.st) + (warp - 2) * (COLS / 4) * 32 + lane;
        if (part > 0) {
#pragma unroll
          for (int h = 0; h < COLS / 4; ++h) box[32 * h] = make_float4(run[4 * h], run[4 * h + 1], run[4 * h + 2], run[4 * h + 3]);
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(nf_at_rank(&sm.parts, 0)) : "memory");
          continue;
        }
        if (!ns_wait(&sm.parts, 0, &sm.abort)) break;
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        for (int r = 1; r < parts; ++r) {
          const uint32_t src = nf_at_rank(box, r);
#pragma unroll
          for (int h = 0; h < COLS / 4; ++h) {
            float4 v;
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(src + 512 * h) : "memory");
            run[4 * h] += v.x; run[4 * h + 1] += v.y; run[4 * h + 2] += v.z; run[4 * h + 3] += v.w;
          }
        }
      }
      float* const C = g.C ? g.C + (long long)b * g.sC : nullptr;
      __half* const P = g.P ? g.P + (long long)b * g.sP : nullptr;
      const long long planeP = g.planeP;
      const bool cvec = (ldc & 3) == 0;
#pragma unroll
      for (int q = 0; q < COLS / 16; ++q) {
        const int n0 = tn * BN + col0 + 16 * q;
        if (n0 < N && m0 < M && (!sym || n0 + 15 >= m0)) {   // the same for the whole warp
#pragma unroll
          for (int h = 0; h < 4; ++h)
            st4(nf_out(stage, lane, h), make_float4(alpha * run[16 * q + 4 * h], alpha * run[16 * q + 4 * h + 1],
                                                                 alpha * run[16 * q + 4 * h + 2], alpha * run[16 * q + 4 * h + 3]));
          __syncwarp();
          const int n = n0 + sc;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = sr + 8 * i, m = m0 + rr;
            if (m < M && n < N && (!sym || n + 3 >= m)) {
              float4 o = ld4(nf_out(stage, rr, lane & 3));
              float v[4] = {o.x, o.y, o.z, o.w};
              if (C) {
                float* crow = C + (long long)m * ldc + n;
                if (cvec && n + 3 < ldc) st4(crow, make_float4(v[0], v[1], v[2], v[3]));
                else {
#pragma unroll
                  for (int j = 0; j < 4; ++j) if (n + j < N) crow[j] = v[j];
                }
              }
              if (P) {
                __half hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float s = v[j] * scale;
                  hi[j] = __float2half_rn(s);
                  lo[j] = __float2half_rn(s - __half2float(hi[j]));
                }
                __half* prow = P + (long long)m * ldp + n;
                if (!sym || n >= m) {   // ldp is a multiple of 8: a piece is inside the (padded) row
                  *reinterpret_cast<uint2*>(prow) = *reinterpret_cast<const uint2*>(hi);
                  *reinterpret_cast<uint2*>(prow + planeP) = *reinterpret_cast<const uint2*>(lo);
                } else {                // the piece with the diagonal: the part left of it belongs to the mirror
#pragma unroll
                  for (int j = 0; j < 4; ++j) if (n + j >= m && n + j < N) { prow[j] = hi[j]; prow[planeP + j] = lo[j]; }
                }
              }
            }
          }
          __syncwarp();
          if (sym && P) {
            // the mirror image, from the accumulators: the lanes of a warp write neighbours of row n0 + j
            const int m = m0 + lane;
            if (m < M) {
              __half* pcol = P + m;
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (n0 + j > m && n0 + j < N) {
                  const float s = alpha * run[16 * q + j] * scale;
                  const __half hi = __float2half_rn(s);
                  pcol[(long long)(n0 + j) * ldp] = hi;
                  pcol[planeP + (long long)(n0 + j) * ldp] = __float2half_rn(s - __half2float(hi));
                }
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR || SPLIT) cluster_sync();   // no CTA leaves while another may read its shared memory
  if (tid == 0 && sm.abort && status) atomicOr(status, 4);
  if (warp == 1) {
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    else tc_dealloc(tmem, 512);
  }
}

// 256 x 256 on pairs of SMs where that fills the GPU, else 128 x 128 on one SM
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NF_THREADS, 1) k_gemm_f16x2_pair(const __grid_constant__ nf_group grp, int* __restrict__ status) {
  nf_gemm_body<256, true, false>(grp, status);
}
__global__ void __launch_bounds__(NF_THREADS, 1) k_gemm_f16x2(const __grid_constant__ nf_group grp, int* __restrict__ status) {
  nf_gemm_body<128, false, false>(grp, status);
}
// few tiles with a long contraction: launched in clusters of 2, 4 or 8
__global__ void __launch_bounds__(NF_THREADS, 1) k_gemm_f16x2_split(const __grid_constant__ nf_group grp, int* __restrict__ status) {
  nf_gemm_body<128, false, true>(grp, status);
}

// ------------------------------------------------------------------------------------------------
// Start of the chain: x / (||x||_F + eps), as planes.  Slices of NF_SLICE elements of a matrix: partial sums of squares,
// then every slice's CTA adds its matrix's partials up in the same fixed order.
// ------------------------------------------------------------------------------------------------
#define NF_SLICE 8192
struct nf_prep {
  const float* x;      // [batch][n]
  float* part;         // [batch][slices]
  float* inv;          // [batch]: 1 / (norm + eps)
  __half* P;           // planes [2][batch][rows][ldp]
  long long n, sP, planeP;
  int cols, ldp, slices, cta0;   // cta0: CTAs of the items before this one
  float eps, scale;
};
struct nf_prep_group { nf_prep p[NF_GROUP]; int n; };
__device__ __forceinline__ const nf_prep& nf_locate(const nf_prep_group& grp, int& b, int& slice) {
  int k = 0;
  while (k + 1 < grp.n && (int)blockIdx.x >= grp.p[k + 1].cta0) ++k;
  const int r = blockIdx.x - grp.p[k].cta0;
  b = r / grp.p[k].slices;
  slice = r - b * grp.p[k].slices;
  return grp.p[k];
}
__global__ void __launch_bounds__(NT) k_ns_sumsq(const __grid_constant__ nf_prep_group grp) {
  pdl_begin();
  __shared__ float s_red[40];
  int b, slice;
  const nf_prep& q = nf_locate(grp, b, slice);
  const float* p = q.x + b * q.n + (long long)slice * NF_SLICE;
  const long long rem = q.n - (long long)slice * NF_SLICE;
  const int left = (int)(rem < NF_SLICE ? rem : NF_SLICE);
  float acc = 0.f;
  const int c4 = ((uintptr_t)p & 15) == 0 ? (left & ~3) : 0;
#pragma unroll 4
  for (int i = threadIdx.x * 4; i < c4; i += NT * 4) {
    const float4 v = ldg4(p + i);
    acc += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  for (int i = c4 + threadIdx.x; i < left; i += NT) acc += p[i] * p[i];
  acc = block_sum(acc, s_red);
  if (threadIdx.x == 0) q.part[(long long)b * q.slices + slice] = acc;
}

// planes of scale * x * inv; a CTA takes the elements of one slice
__global__ void __launch_bounds__(NT) k_ns_split(const __grid_constant__ nf_prep_group grp) {
  pdl_begin();
  __shared__ double s_d[NWARP];
  __shared__ float s_inv;
  int b, slice;
  const nf_prep& q = nf_locate(grp, b, slice);
  double acc = 0.0;
  for (int i = threadIdx.x; i < q.slices; i += NT) acc += (double)q.part[(long long)b * q.slices + i];
  acc = warp_sum_d(acc);
  if ((threadIdx.x & 31) == 0) s_d[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < NWARP; ++w) t += s_d[w];
    s_inv = 1.0f / (sqrtf((float)t) + q.eps);
    if (slice == 0) q.inv[b] = s_inv;
  }
  __syncthreads();
  const float f = s_inv, scale = q.scale;
  const int cols = q.cols, ldp = q.ldp;
  const long long n = q.n, planeP = q.planeP, first = (long long)slice * NF_SLICE, last = n < first + NF_SLICE ? n : first + NF_SLICE;
  const float* __restrict__ xb = q.x + b * n;
  __half* __restrict__ pb = q.P + b * q.sP;
  if ((cols & 3) == 0 && ((uintptr_t)xb & 15) == 0) {
    for (long long i = first + threadIdx.x * 4; i < last; i += NT * 4) {
      const float4 v4 = ldg4(xb + i);
      const long long row = i / cols;
      const long long at = row * ldp + (i - row * cols);
      const float v[4] = {v4.x * f * scale, v4.y * f * scale, v4.z * f * scale, v4.w * f * scale};
      __half hi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { hi[j] = __float2half_rn(v[j]); lo[j] = __float2half_rn(v[j] - __half2float(hi[j])); }
      *reinterpret_cast<uint2*>(pb + at) = *reinterpret_cast<const uint2*>(hi);
      *reinterpret_cast<uint2*>(pb + planeP + at) = *reinterpret_cast<const uint2*>(lo);
    }
  } else {
    for (long long i = first + threadIdx.x; i < last; i += NT) {
      const long long row = i / cols;
      const long long at = row * ldp + (i - row * cols);
      const float v = xb[i] * f * scale;
      const __half hi = __float2half_rn(v);
      pb[at] = hi;
      pb[planeP + at] = __float2half_rn(v - __half2float(hi));
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Matrices whose whole chain is a few million FMAs at most: one CTA per matrix, everything in shared memory, plain fp32.
// A tile of the tensor-core kernel would be mostly padding (a 16 x 16 slice of a ViT patch embedding fills 1/64 of it), and
// fifteen launches would cost more than the arithmetic.
// ------------------------------------------------------------------------------------------------
// One matrix by a CTA of THREADS threads.  smem: ns_small_floats(rows, cols) floats of shared memory, s_red: 33.
template <int THREADS>
__device__ __forceinline__ void ns_small_body(const float* __restrict__ src, float* __restrict__ dst, int rows, int cols, int iters,
                                              float c0, float c1, float c2, float eps, float* smem, float* s_red) {
  const bool tall = rows > cols;
  const int r = tall ? cols : rows, c = tall ? rows : cols, n = rows * cols, pitch = c + 1, pa = r + 1;
  float* X = smem;
  float* Y = X + r * pitch;
  float* A = Y + r * pitch;
  float* B = A + r * pa;
  const int tid = threadIdx.x;
  float acc = 0.f;
  for (int i = tid; i < n; i += THREADS) {
    const float v = src[i];
    acc = fmaf(v, v, acc);
    const int a = i / cols, b = i - a * cols;
    X[tall ? b * pitch + a : a * pitch + b] = v;
  }
  const float f = 1.0f / (sqrtf(block_sum(acc, s_red)) + eps);
  for (int i = tid; i < r * pitch; i += THREADS) if (i % pitch < c) X[i] *= f;
  // lanes per entry of a (r x r): as many as keep all threads busy
  int L = 1;
  while (L < 32 && r * r * L * 2 <= THREADS) L *= 2;
  __syncthreads();
  for (int it = 0; it < iters; ++it) {
    for (int p0 = 0; p0 < r * r; p0 += THREADS / L) {       // the same trip count for all threads
      const int p = p0 + tid / L, i = p / r, j = p - i * r;
      float s = 0.f;
      if (p < r * r)
        for (int k = tid % L; k < c; k += L) s = fmaf(X[i * pitch + k], X[j * pitch + k], s);
      for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, L);
      if (p < r * r && tid % L == 0) A[i * pa + j] = s;
    }
    __syncthreads();
    for (int p = tid; p < r * r; p += THREADS) {
      const int i = p / r, j = p - i * r;
      float s = 0.f;
      for (int k = 0; k < r; ++k) s = fmaf(A[i * pa + k], A[k * pa + j], s);
      B[i * pa + j] = fmaf(c2, s, c1 * A[i * pa + j]);
    }
    __syncthreads();
    for (int p = tid; p < r * c; p += THREADS) {
      const int i = p / c, k = p - i * c;
      float s = c0 * X[i * pitch + k];
      for (int j = 0; j < r; ++j) s = fmaf(B[i * pa + j], X[j * pitch + k], s);
      Y[i * pitch + k] = s;
    }
    __syncthreads();
    float* t = X; X = Y; Y = t;
  }
  for (int i = tid; i < n; i += THREADS) {
    const int a = i / cols, b = i - a * cols;
    dst[i] = X[tall ? b * pitch + a : a * pitch + b];
  }
}
__global__ void __launch_bounds__(NT) k_ns_small(const float* __restrict__ x, float* __restrict__ out, int rows, int cols, int iters,
                                                 float c0, float c1, float c2, float eps) {
  pdl_begin();
  extern __shared__ __align__(16) float ns_s[];
  __shared__ float s_red[40];
  const long long at = (long long)blockIdx.x * rows * cols;
  ns_small_body<NT>(x + at, out + at, rows, cols, iters, c0, c1, c2, eps, ns_s, s_red);
}
