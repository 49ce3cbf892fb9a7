/*
 * pylo_b200 - C ABI of the B200 (sm_100a) learned-optimizer step kernels.
 *
 * One shared library, plain C linkage, raw device pointers and sizes, a CUDA
 * stream passed as void*.  Every entry point returns an int:
 *   0            ok
 *   < 0          an argument was rejected on the host before anything was launched
 *   > 0          a cudaError_t reported by the launch
 * No entry point allocates, frees, synchronises or throws, unless its comment
 * says otherwise.  The caller owns all memory.  Descriptor, tile and item arrays
 * are DEVICE pointers; pylo_step_params and pylo_velo_rnn are HOST pointers whose
 * contents are copied into the launch.  Calls are re-entrant as long
 * as two calls in flight do not share workspace.
 *
 * The three pybind functions of the reference that this library replaces:
 *   cuda_lo.learned_optimizer_kernel      pylo/csrc/learned_optimizer.cu:303-404
 *   celo2_cuda_kernel.celo2_kernel        pylo/csrc/celo2_kernel.cu:284-357
 *   velo_cuda_kernel.velo_kernel_simple   pylo/csrc/velo_kernel.cu:370-462
 * together with the torch-op state update the reference's Python classes run
 * before calling them (pylo/optim/AdafacLO_cuda.py:322-373,
 * pylo/optim/CELO2_cuda.py:205-232, pylo/optim/velo_cuda.py:502-546).
 *
 * The work is described by two tables in DEVICE memory that the host builds
 * once per parameter set: an array of pylo_tensor_desc (one per parameter
 * tensor) and arrays of tiles that cut the tensors into units of work.  One
 * optimizer step is a fixed sequence of launches over those tables
 * (see pylo_b200_* below, in call order).
 */
#ifndef PYLO_B200_H
#define PYLO_B200_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define PYLO_B200_ABI_VERSION 19

/* optimizer families (which feature set / network geometry a launch uses) */
#define PYLO_FAM_ADAFAC 0 /* AdafacLO_CUDA, ELO_CUDA: 28+11 features, 39-32-32-2 */
#define PYLO_FAM_CELO2 1  /* CELO2_CUDA, ELO_CELO2_CUDA: 30 features, 30-8-8-3, writes step_out */
#define PYLO_FAM_VELO 2   /* VeLO_CUDA: 30 features, 30-4-4-3, per-tensor weights */

/* how a tensor is traversed */
#define PYLO_MODE_FAST2D 0  /* contiguous [X,Y], Y % 4 == 0, 16-byte aligned: float4 path */
#define PYLO_MODE_GENERIC 1 /* any contiguous [O,X,M,Y,I] view, scalar loads */
#define PYLO_MODE_KERNEL 3  /* contiguous [X,Y,I] with I <= 32 positions (convolution weights; O = M = 1), Y * I % 4 == 0, 16-byte aligned: a
                               matrix of Y * I columns whose "a" vectors have an entry per row and position; for pylo_b200_apply as GENERIC */
#define PYLO_MODE_VEC1D 2   /* fewer than two dims: accumulators are full size ("vector_like") */

#define PYLO_STAT_STRIDE 40  /* floats per tile partial / per tensor sums: 30 feature slots + 8 VeLO statistics */
#define PYLO_TILE_ELEMS 16384 /* elements per element-wise tile (at most) */
#define PYLO_A_COLS 1024      /* columns per row/column-sum tile */
#define PYLO_WFOLD_STRIDE 4800 /* ADAFAC: floats of desc.wfold, the folded network and the tensor cores' operands (the others: see workspace_layout) */
#define PYLO_SMALL_FLOATS 52224 /* shared memory of pylo_b200_small_front, in floats */
#define PYLO_MAX_PEERS 7       /* other GPUs of one box */

/*
 * One unit of element-wise work: a whole parameter tensor, or one matrix slice of a tensor
 * with more than two dims when the normalisers are taken per slice (CELO2 family,
 * CELO2_naive.py:328-329).  A slice points into its tensor's buffers (idx0, m_stride) and
 * shares its factor vectors.  The tensor is viewed as a contiguous 5-D array
 * [O, X, M, Y, I]; X and Y are its two factored axes in memory order and O, M,
 * I the products of the other axes.  "a" vectors drop the Y axis (length
 * O*X*M*I, indexed by x for a 2-D tensor), "b" vectors drop the X axis (length
 * O*M*Y*I, indexed by y).  r_is_a says whether the reference's row accumulator
 * (exp_avg_sq_r / fac_r / fac_vec_row, which drops axis dr) is the "a" one.
 */
typedef struct pylo_tensor_desc {
  const float* g; /* gradient [n] */
  float* p;       /* parameter [n] */
  float* m;       /* momentum [3][n] */
  float* v;       /* second moment [n] */
  float* fac_a;   /* factored accumulator state, [3][La] (VEC1D: the row one, [3][n]) */
  float* fac_b;   /* factored accumulator state, [3][Lb] (VEC1D: the column one or NULL) */
  float* f_a;     /* workspace [3][La]: rsqrt factor in "a" orientation */
  float* f_b;     /* workspace [3][Lb] */
  float* fx;      /* workspace [La][4]: f_a interleaved per index (FAST2D, KERNEL, and GENERIC matrices with tables, see workspace_layout; else NULL) */
  float* sum_a;   /* workspace [La]: sum over Y of g'^2 + 1e-30 */
  float* sum_b;   /* workspace [Lb]: sum over X */
  float* part_a;  /* workspace [X][n_cb]  row-sum partials (tensors in atiles; else NULL); KERNEL: [La][2 n_cb] */
  float* part_b;  /* workspace [n_strips][Lb] column-sum partials */
  float* h_a;     /* workspace [La][H] (ADAFAC) or [La][H][2] (CELO2, VELO): first-layer term of the "a" features (+ bias); h_a, h_b: NULL
                     where apply_adafac_tc is the only sweep over the tensor, which reads no tables */
  float* h_b;     /* workspace [H][Lb]: first-layer term of the "b" features */
  float* closed;  /* workspace [PYLO_STAT_STRIDE]: closed-form sums of squares of vector features */
  float* sums;    /* workspace [48]: per-tensor sums (30 feature slots, 8 VeLO statistics, their 8 low-order parts) */
  float* wfold;   /* workspace: network with normalisers folded in; ADAFAC: [PYLO_WFOLD_STRIDE], the tensor cores' operands behind it */
  float* tile_part; /* workspace [n_tiles][PYLO_STAT_STRIDE] */
  float* out;     /* CELO2: raw step output [n]; else NULL */
  const float* w; /* network weights for this tensor, family layout (see pylo_b200_prep_apply) */
  const float* lr_mult; /* VeLO: device scalar multiplying lr for this tensor, else NULL */
  float* p_peer[PYLO_MAX_PEERS]; /* the same parameter inside the other ranks' peer-mapped buffers (first n_peer
                                    entries valid): kernels that write p store the new value there as well, which
                                    replaces the all-gather of updated parameters.  n_peer < 0: p_peer[0] is a
                                    multicast address mapping the parameter in every rank's buffer, and the kernels
                                    issue one multimem store to it instead */
  int64_t n;        /* elements of this unit */
  int64_t m_stride; /* distance in floats between the three momentum planes (n for a whole tensor) */
  int64_t idx0;     /* offset of this unit's first element inside the [O,X,M,Y,I] view (0 for a whole tensor) */
  int64_t La, Lb;   /* lengths of the "a" and "b" vectors (0 for VEC1D) */
  int32_t O, X, M, Y, I;
  int32_t mode;
  int32_t r_is_a;
  int32_t rcm_pre, rcm_A, rcm_post; /* row_col_mean: the row accumulator viewed [pre][A][post], mean over A */
  int32_t rb, n_strips, n_cb;       /* phase-A tiling: rows per strip, strips, column blocks (tensors in atiles) */
  int32_t tile0, n_tiles;           /* this tensor's range in the element-wise tile list */
  int32_t vec_elementwise;          /* 1: this unit is a slice of a tensor (its normalisers cover the slice only),
                                       so the vector-only features are accumulated per element, not in closed form */
  float lr;                         /* learning rate of the tensor's group */
  float wd;                         /* weight decay (family meaning) */
  float step;                       /* AdafacLO/ELO: 0-based step for the time features */
  float clip_norm;                  /* >0: scale g by clip_norm / max(global norm, clip_norm) */
  float exp_mult, step_mult;
  int32_t n_peer;                   /* number of valid p_peer entries (0: single GPU, or parameters gathered by NCCL) */
  int32_t pad_;
} pylo_tensor_desc;

/* a unit of element-wise work: elements [start, start + elems) of tensor `tensor`.  elems <= 0 means PYLO_TILE_ELEMS; a
 * host with little work cuts it into smaller tiles (multiples of 4) so that they fill the GPU.  A tensor's tiles in the
 * list given to pylo_b200_state_moments all have one size, and desc.tile0 / n_tiles / tile_part go with that list. */
typedef struct pylo_tile {
  int64_t start;
  int32_t tensor;
  int32_t elems;
} pylo_tile;

/* a unit of row/column-sum work: rows [row0, row0+rb) x columns [col0, col0+PYLO_A_COLS) */
typedef struct pylo_atile {
  int32_t tensor;
  int32_t strip;
  int32_t cb;
  int32_t pad_;
} pylo_atile;

/* per-launch constants shared by all tensors */
typedef struct pylo_step_params {
  int32_t family;
  int32_t nan_to_num;     /* ELO: torch.nan_to_num on the (scaled) gradient */
  int32_t wd_mode;        /* 0 none in kernel; 1 AdafacLO (after update, on new p); 2 ELO (on old p); 3 VeLO (lr_eff) */
  float step_delta;       /* added to every desc.step: lets the host advance the step count without re-uploading the table */
  float w_m[3];           /* 1 - beta_m[k], computed in fp32 as the reference does */
  float w_v;              /* 1 - beta_rms */
  float w_f[3];           /* 1 - beta_fac[k] */
  float eps_v;            /* added to g^2 before the second-moment EMA (1e-30 AdafacLO/ELO, 0 otherwise) */
  float eps_feat;         /* inside rsqrt(v + eps): 1e-6 AdafacLO/ELO/VeLO, 1e-8 CELO2 */
  float eps_norm;         /* inside rsqrt(S/n + eps): 1e-5 AdafacLO/ELO/VeLO, 1e-9 CELO2 */
  float clip_val;         /* element-wise clamp of the gradient; +inf for none */
  int32_t no_tables;      /* prep_apply: 0 = make the per-row (desc.h_a) and per-column (desc.h_b) first-layer tables, and for ADAFAC
                             what apply_adafac_tc reads; 1 = neither; 2 = only what apply_adafac_tc reads (ADAFAC); 3 = the tables only.
                             apply_adafac_tc: 4 = small_front has made the networks; the features' scales come from the tile partials */
  const float* gnorm_sq;  /* device scalar: sum of squares of all gradients, or NULL */
  int32_t sum_tiles;      /* prep_apply: 1 = add the tile partials up itself (finalize_moments was not called) */
  int32_t bulk_copies;    /* state_moments: 1 = FAST2D tiles come through a ring of bulk copies, for large models that consist
                             of them; 0 = all tiles are read into registers */
  int* status;            /* device int: state_moments ORs 8 in if a bounded wait for its own copies ran out (the step is
                             then incomplete); the apply kernels that write parameters (ADAFAC, VELO) write none while it
                             is not zero; may be NULL */
  int* host_status;       /* a word of pinned host memory that both events are written to; may be NULL */
  const float* w_host;    /* HOST pointer to the network of desc.w, where it is the same for all units, or NULL.  CELO2: apply_packed
                             then takes it as an argument of its launch instead of reading the folded one of every unit;
                             ADAFAC: apply_adafac_tc its output layer */
  float* step_squares;    /* CELO2: apply_packed leaves the sum of squares of item k's raw steps in step_squares[k] (what celo2_post_sums
                             would make, in other pieces); may be NULL */
} pylo_step_params;

int pylo_b200_abi_version(void);
int pylo_b200_sizeof_desc(void);
int pylo_b200_sizeof_params(void);

/* Workspace sizing, for hosts that fill pylo_tensor_desc themselves.  The reference needs no counterpart: its
 * only scratch is the second_moment[28|30] tensor its Python classes allocate per call
 * (AdafacLO_cuda.py:376-380, CELO2_cuda.py:287-291, velo_cuda.py:731-735).
 *
 * pylo_b200_workspace_layout fills, for one tensor of the given family, traversal mode and geometry, the size
 * in floats of every workspace sub-buffer that pylo_tensor_desc points at (0 where the mode does not use it),
 * and the phase-A tiling (rb, n_strips, n_cb) and the number of element-wise tiles that go into the descriptor.  A GENERIC tensor
 * that is a plain matrix (O = M = I = 1) may be given with its X and Y (a KERNEL one is, with its X and its Y * I columns): its sums then go into the items of FAST2D tensors (atiles),
 * and for CELO2 and VELO it has the tables of pylo_b200_apply_packed's ragged items.
 * A unit of element-wise work that is a slice of a tensor (vec_elementwise = 1) owns only the last three
 * sub-buffers (sums, wfold, tile_part), sized with n = the slice's elements, plus a zero-filled `closed`; the
 * others belong to its tensor.  Every sub-buffer must start on a 256-byte boundary and the whole workspace
 * must be zero before the first step.
 * pylo_b200_workspace_bytes adds the sizes up, each rounded up to 256 bytes: tensor_part != 0 counts f_a .. closed,
 * unit_part != 0 counts sums, wfold, tile_part.  Host-only; nothing is launched. */
typedef struct pylo_ws_layout {
  int64_t f_a, f_b, sum_a, sum_b, fx, part_a, part_b, h_a, h_b, closed; /* per tensor */
  int64_t sums, wfold, tile_part;                                         /* per unit of element-wise work */
  int32_t rb, n_strips, n_cb, n_tiles;
} pylo_ws_layout;
int pylo_b200_workspace_layout(int family, int mode, int64_t n, int64_t La, int64_t Lb, int32_t X, int32_t Y,
                               pylo_ws_layout* out);
int64_t pylo_b200_workspace_bytes(const pylo_ws_layout* layout, int tensor_part, int unit_part);

/* Sum of squares of every gradient (CELO2_cuda.py:180-188, ELO_cuda.py:150-158).
 * items: one per tensor with a gradient (all of them, AdamW-routed ones included);
 * tiles: element-wise tiles over the items; scratch: [n_tiles] floats; out: device scalar. */
typedef struct pylo_gvec {
  const float* g;
  int64_t n;
} pylo_gvec;
int pylo_b200_grad_sumsq(const pylo_gvec* items, const pylo_tile* tiles, int n_tiles,
                         float* scratch, float* out, void* stream);

/* The same sum of squares for callers that cannot provide scratch memory (no counterpart in the
 * reference: it never needs scratch because it reduces with atomics).
 *
 * Who needs it: a host that cannot allocate device memory for us - for example a binding from another
 * language that links nothing but this library, or an optimizer hook that is forbidden to call
 * cudaMalloc inside the step because cudaMalloc stalls the whole device.  This entry point calls no
 * cudaMalloc / cudaFree and no allocating library routine; the per-tile partial sums go to a fixed
 * array inside the library (PYLO_STATIC_SCRATCH_TILES floats = 256 KiB, resident on every GPU that
 * loads the library until the process ends).
 *
 * Limits and rules:
 *  - n_tiles <= PYLO_STATIC_SCRATCH_TILES (2^16 tiles = 2^30 gradient elements); more is refused with
 *    PYLO_ERR_STATIC_SCRATCH_TOO_SMALL and nothing is launched.
 *  - The first call on each device looks up the array's device address (with that device current).
 *    Make that first call during set-up, before any stream capture begins.
 *  - All calls share the one array, and it keeps whatever the previous call left in it.  That is
 *    harmless here (each call overwrites every slot it later reads, so nothing needs zeroing), but two
 *    calls that overlap on the GPU - different streams, or different host threads - race on it and
 *    give wrong sums.  Serialise them.
 * items, tiles, out, stream: as for pylo_b200_grad_sumsq. */
#define PYLO_STATIC_SCRATCH_TILES 65536
#define PYLO_ERR_STATIC_SCRATCH_TOO_SMALL (-4)
int pylo_b200_grad_sumsq_static(const pylo_gvec* items, const pylo_tile* tiles, int n_tiles, float* out,
                                void* stream);

/* Phase A: row and column sums of g'^2 + 1e-30 (the reductions inside
 * grad_sqr.mean(dim=dr / dc), AdafacLO_cuda.py:333-340, CELO2_cuda.py:218-224, velo_cuda.py:531-541).
 * atiles cover the FAST2D tensors, GENERIC matrices laid out like them (the first n_ragged) and KERNEL tensors (the next n_kernel):
 * a strip x 1024-column block each; they leave per-strip column partials, which pylo_b200_factor_update adds up.  gitems cover the GENERIC tensors: items with pad_ = 1 take 256 of the Lb columns
 * (cb) over the rows of a strip (desc.rb of the X rows), items with pad_ = 0 take cb of the La / I
 * blocks that have I row sums each, from block strip * cb on. */
int pylo_b200_rowcol_sums(const pylo_tensor_desc* descs, const pylo_atile* atiles, int n_atiles, int n_ragged, int n_kernel,
                          const pylo_atile* gitems, int n_gitems, const pylo_step_params* prm, void* stream);

/* Phase A2, one cluster of CTAs per tensor: the sums over strips and column blocks of phase A's partials, EMA of the factored accumulators, row_col_mean,
 * row/column rsqrt factors (AdafacLO_cuda.py:342-345, CELO2_cuda.py:229-231, velo_cuda.py:716-729)
 * and the closed-form feature moments of the twelve vector-only features.  mats: DEVICE list of the n_tensors tensors to take (VEC1D ones
 * have nothing to do, as long as their `closed` is zero), or NULL for the first n_tensors.  threads: 1024 or 512 per CTA, which decides
 * the order of the sums; 512 is faster for more tensors than run at once (eight CTAs each). */
int pylo_b200_factor_update(const pylo_tensor_desc* descs, const int32_t* mats, int n_tensors, int threads, const pylo_step_params* prm,
                            void* stream);

/* Phase B: momentum / second-moment EMA in place and per-tile sums of squares of
 * every element-wise feature (AdafacLO_cuda.py:341,370-373; lo_kernel learned_optimizer.cu:100-190;
 * celo2_moment_kernel celo2_kernel.cu:130-199; velo_compute_moments_kernel velo_kernel.cu:170-256).
 * For VeLO it also accumulates the statistics of the state before the update that
 * lstm_features_for_tensor needs (velo_cuda.py:213-252). */
int pylo_b200_state_moments(const pylo_tensor_desc* descs, const pylo_tile* tiles, int n_tiles,
                            int reverse, const pylo_step_params* prm, void* stream);

/* Phases A, A2 and B of a small model in one launch, a cluster of 1, 2, 4, 8 or 16 CTAs per tensor.  Every tensor is VEC1D, or a
 * contiguous matrix (O = M = I = 1) whose row_col_mean is over the whole vector (rcm_pre = 3) or over the decays (rcm_pre = 1,
 * rcm_A = 3); the units are the tensors.  slice: the most elements of a CTA's ceil(X / cluster) rows, up to 8192 (of a vector:
 * any); rows, cols: the most such rows and columns; 6 slice + 4 rows + 5 cols, each rounded up to 4, fit PYLO_SMALL_FLOATS.
 * Every tensor leaves `cluster` rows of tile_part, so desc.n_tiles has to be that.  networks (ADAFAC): further clusters that make the
 * networks apply_adafac_tc reads, which then (no_tables = 4) adds up the partials itself; prep_apply is not needed. */
int pylo_b200_small_front(const pylo_tensor_desc* descs, int n_tensors, int cluster, int slice, int rows, int cols, int networks,
                          const pylo_step_params* prm, void* stream);

/* Phase B2, one CTA per tensor: fixed-order reduction of the tile partials into desc.sums. */
int pylo_b200_finalize_moments(const pylo_tensor_desc* descs, int n_tensors, void* stream);

/* Phase P: fold the normalisers rsqrt(S_j/n + eps) and, for
 * AdafacLO/ELO, the time features tanh(t/tau - 1) (learned_optimizer.cu:27-32,245-248) into the
 * first layer, and tabulate the first-layer contribution of the vector-only features.  items: tensor = unit, strip =
 * index of the unit's item.  Item 0 of every unit writes the folded network; with tables, an item also makes
 * 2048 / H entries of a table: items 0 .. ceil(X / (2048/H)) - 1 the per-row one, the following ceil(Y / (2048/H)) the
 * per-column one (FAST2D units; the others have item 0 only).
 * desc.w layouts: ADAFAC  w_in[32][39] b_in[32] w_h[32][32] b_h[32] w_out[2][32] b_out[2] (out-major);
 *                 CELO2   w_in[30][8]  b_in[8]  w_h[8][8]   b_h[8]  w_out[8][3]  b_out[3] (in-major);
 *                 VELO    w_in[4][30]  b_in[4]  w_h[4][4]   b_h[4]  w_out[3][4]  b_out[3] (out-major). */
int pylo_b200_prep_apply(const pylo_tensor_desc* descs, const pylo_atile* items, int n_items, const pylo_step_params* prm,
                         void* stream);

/* Phase C: rebuild the features, run the network, write the parameter (ADAFAC, VELO) or the raw
 * step (CELO2) (lo_kernel_apply learned_optimizer.cu:194-301, celo2_apply_kernel celo2_kernel.cu:204-282,
 * velo_apply_kernel velo_kernel.cu:260-368). */
int pylo_b200_apply(const pylo_tensor_desc* descs, const pylo_tile* tiles, int n_tiles, int reverse,
                    const pylo_step_params* prm, void* stream);

/* Phase C for the FAST2D tensors of the ADAFAC family (same arithmetic as pylo_b200_apply, organised for
 * the FMA-bound 39-32-32-2 network: a thread keeps one column, packed fp32x2 FMAs).  ctiles: one entry per
 * tile with strip = row-tile index, cb = column-tile index, pad_ = columns per CTA (32, 64, 128 or 256) | (n_sub << 16); a work item
 * covers n_sub sub-tiles of 32 rows in one column block.  With this kernel in use pylo_b200_apply gets only the non-FAST2D tiles.
 * With one of the FAST2D kernels in use pylo_b200_apply handles the GENERIC and VEC1D units only. */
int pylo_b200_apply_adafac_cols(const pylo_tensor_desc* descs, const pylo_atile* ctiles, int n_ctiles,
                                const pylo_step_params* prm, void* stream);

/* Phase C for the tensors of the ADAFAC family on the tensor cores (no reference counterpart: the
 * reference evaluates the network with scalar FMAs, lo_kernel_apply learned_optimizer.cu:236-284).  Same outputs
 * as pylo_b200_apply_adafac_cols; it reads no first-layer tables, but the operands that pylo_b200_prep_apply makes
 * with no_tables = 2 or 0.  The two hidden layers run as tcgen05 products of
 * operands split into a high and a low fp16 plane (hi x hi + hi x lo + lo x hi), features scaled by one power of two and every hidden unit
 * by one of its own, which keeps a 32-term dot product within ~3e-7 of the sum of its terms' magnitudes, whatever the units' scales, with a
 * floor under a feature's magnitude: 2^-(25 + q) of its root mean square over the unit, 2^q sqrt(n) <= 2^15 and q <= 6 (2^-27 at 16 M
 * elements).  A feature that is not a number or infinite makes the element's hidden activations zero, where the scalar path may
 * give an infinity.  ttiles: strip = row-strip index, cb = block of 128 columns, pad_ = rows per work item (one
 * warpgroup of a CTA takes a whole item).  Units that are neither FAST2D nor KERNEL: pad_ = 0x10000 | tiles per work item, strip = item
 * index, cb = 0; an item is that many runs of 128 consecutive elements; generic != 0 says that the list may hold such
 * items, or items on KERNEL units; no_tables = 4 is refused without it.  status: device int; the kernel ORs 1 into it if a wait on the tensor
 * core ran out (the parameters it could not finish then keep their old values), and a launch that finds it
 * non-zero stores nothing; may be NULL.  host_status: a word of pinned (device-accessible) host memory that both events
 * are also written to, so that the host can look without asking the device; may be NULL. */
int pylo_b200_apply_adafac_tc(const pylo_tensor_desc* descs, const pylo_atile* ttiles, int n_ttiles, int generic,
                              const pylo_step_params* prm, int* status, int* host_status, void* stream);

/* Phase C for the FAST2D tensors of the CELO2 and VELO families (same arithmetic as pylo_b200_apply, done on
 * pairs of adjacent elements with packed fp32x2 instructions).  ctiles: strip = row-tile index, cb = column-tile
 * index, pad_ = threads per row (8 .. 256, a thread owns 4 columns) | rows per thread << 16 (0: 16); a tile has
 * rows * (256 / threads) rows and 4 * threads columns.  ragged != 0: the items are on GENERIC matrices with tables (any Y, any
 * alignment).  For these families pylo_b200_prep_apply stores desc.h_a as (v, v) pairs, [X][H][2], and
 * for every family desc.h_b transposed, [H][Y].  tiles: other tensors' for
 * pylo_b200_apply, done in the same launch for VELO and in one after it for CELO2. */
int pylo_b200_apply_packed(const pylo_tensor_desc* descs, const pylo_atile* ctiles, int n_ctiles, int ragged,
                           const pylo_tile* tiles, int n_tiles, const pylo_step_params* prm, void* stream);

/* Batched fp32-faithful matrix product on the tensor cores, for the Newton-Schulz orthogonalisation of the CELO2
 * family (orthogonalize_via_newton_schulz, CELO2_naive.py:59-73, called at CELO2_cuda.py:332-335; the reference runs
 * it as torch.matmul):
 *     C[b][m][n] = alpha * sum_k A[b][m][k] * B[b][n][k] + beta * D[b][m][n]        b < batch
 * A is [M][K] with row pitch lda, B is [N][K] with row pitch ldb (both with K contiguous), C and D are [M][N].
 * One round of the iteration is three calls: a = x x^T (A = B = x), b = c1 a + c2 a a (A = B = D = a, a being
 * symmetric) and x' = c0 x + b x (A = b, B = x^T, D = x).  Every operand element is split into a TF32 high and low
 * part inside the kernel and three tcgen05 products (lo x hi, hi x lo, hi x hi) are accumulated in fp32.
 * Requirements (else -1): K, N and all pitches and batch strides multiples of 4, all pointers 16-byte aligned,
 * D (may be NULL) different from C.  g is a HOST pointer.  status: device int, bit 2 is ORed in if a bounded wait
 * inside the kernel ran out (the output is then incomplete); may be NULL. */
typedef struct pylo_gemm_desc {
  const float* A;
  const float* B;
  float* C;
  const float* D;
  int64_t strideA, strideB, strideC, strideD; /* distance in floats between consecutive matrices of the batch */
  int32_t M, N, K, lda, ldb, ldc, ldd, batch;
  float alpha, beta;
  int32_t symmetric; /* != 0: M == N and the result is symmetric (x x^T, a a): only the tiles that touch the diagonal or
                        lie above it are computed; complete C with pylo_b200_transpose(mirror = 1) afterwards */
  int32_t pad_;
} pylo_gemm_desc;
int pylo_b200_gemm_tn_3xtf32(const pylo_gemm_desc* g, int* status, void* stream);

/* Batched transposes for the Newton-Schulz chain.  mirror == 0: dst[b][j][i] = src[b][i][j] for [rows][cols]
 * matrices (src != dst).  mirror != 0: in place on square matrices (src == dst): everything below the diagonal
 * becomes the mirror image of what is above it. */
int pylo_b200_transpose(const float* src, float* dst, int rows, int cols, int ld_src, int ld_dst, int64_t stride_src,
                        int64_t stride_dst, int batch, int mirror, void* stream);

/* The whole Newton-Schulz chain of n stacks of equally shaped matrices (CELO2_naive.py:59-73), the products of up to eight
 * stacks side by side in one launch:
 *     x /= ||x||_F + eps;  iters times  { a = x x^T;  b = c1 a + c2 a a;  x = c0 x + b x }   (a tall x from the right side)
 * x and out are [batch][rows][cols], contiguous, different; x is left as it is.  Operands are kept as two fp16 planes of one
 * power-of-two scale (22 significant bits, as many as a TF32 high and low part), which is sound while every |x| of the chain
 * stays below 10: the caller checks its coefficients.  Matrices of a few thousand elements run in plain fp32 instead,
 * those of up to 128 rows (their shorter side) and 3072 columns in one launch, a cluster of CTAs each, without a workspace, or
 * in the launches of larger stacks of the same call.
 * work: pylo_b200_newton_schulz_workspaces(...) bytes of device memory (may be NULL where that is 0), 256-byte aligned;
 * pylo_b200_newton_schulz_workspace(...), what a stack needs at least, does too.
 * descs is a HOST array; all stacks run the same number of iterations.  status: device int, bit 2 is ORed in if a bounded wait ran out; may be NULL.  Returns -5 where the
 * driver offers no tensor maps. */
typedef struct pylo_ns_desc {
  const float* x;
  float* out;
  void* work;
  int64_t work_bytes;
  int32_t rows, cols, batch, iters;
  float c0, c1, c2, eps;
} pylo_ns_desc;
int64_t pylo_b200_newton_schulz_workspace(int rows, int cols, int batch, int iters);
/* The bytes for every stack of one call, which may be more than what the stack needs at least: a few matrices of up to 128 rows run
 * fastest in the launches of larger ones beside them.  x, out and work of the descs are not looked at. */
int pylo_b200_newton_schulz_workspaces(const pylo_ns_desc* descs, int n, int64_t* bytes);
int pylo_b200_newton_schulz(const pylo_ns_desc* descs, int n, int* status, void* stream);
/* how many kernels that call launches (x and out are not looked at) */
int pylo_b200_newton_schulz_launches(const pylo_ns_desc* descs, int n);

/* CELO2 tail (CELO2_cuda.py:336-339): step * rsqrt(mean(step^2 over the last two axes) + 1e-9) * rmsmult,
 * then p -= lr * (step + wd * p).  Items are matrices (the last two axes of a tensor). */
typedef struct pylo_post_item {
  const float* step; /* [n] orthogonalised (or raw) step */
  float* p;          /* [n] */
  float* part;       /* workspace [n_tiles] */
  int64_t n;
  int32_t tile0, n_tiles;
  float lr, wd, rmsmult, pad_;
} pylo_post_item;
int pylo_b200_celo2_post_sums(const pylo_post_item* items, const pylo_tile* tiles, int n_tiles, void* stream);
/* status, host_status: as in pylo_step_params: no parameter is written while *status is not zero (the words that were given to
 * state_moments and newton_schulz); may be NULL */
int pylo_b200_celo2_post_apply(const pylo_post_item* items, const pylo_tile* tiles, int n_tiles, const int* status, int* host_status,
                               void* stream);

/* AdamW branch for 1-D / embedding tensors.
 * independent != 0: CELO2_cuda.py:234-253 (own exp_avg/exp_avg_sq, betas b1,b2, bias correction with step t);
 * independent == 0: ELO_CELO2_cuda.py:244-253 (updates shared mom[3]/rms with prm, steps from mom[0], rms).
 * bc1 > 0: bc1 and bc2 replace the items' own (all tensors are at the same step, no table to upload). */
typedef struct pylo_adam_item {
  const float* g;
  float* p;
  float* m; /* independent: exp_avg [n]; shared: mom [3][n] */
  float* v; /* independent: exp_avg_sq [n]; shared: rms [n] */
  int64_t n;
  float lr, wd, bc1, bc2; /* lr = adam_lr_mult*lr; bc = 1 - beta^t */
  float clip_norm, pad_[3];
} pylo_adam_item;
int pylo_b200_adamw(const pylo_adam_item* items, const pylo_tile* tiles, int n_tiles, int independent,
                    float beta1, float one_minus_beta1, float beta2, float one_minus_beta2, float eps,
                    float bc1, float bc2, const pylo_step_params* prm, void* stream);
/* celo2_post_apply and adamw in one launch, for small models (up to PYLO_TAIL_ONE_LAUNCH tiles of both). */
#define PYLO_TAIL_ONE_LAUNCH 592
int pylo_b200_celo2_tail(const pylo_post_item* post, const pylo_tile* post_tiles, int n_post, const int* status, int* host_status,
                         const pylo_adam_item* items, const pylo_tile* tiles, int n_tiles, int independent, float beta1, float one_minus_beta1,
                         float beta2, float one_minus_beta2, float eps, float bc1, float bc2, const pylo_step_params* prm, void* stream);

/* VeLO front end.  velo_tensor_features: desc.sums -> the [T][30] LSTM input rows, row T-1-t for
 * tensor t (velo_cuda.py:213-252,419-422); loss features and fraction features are passed in.
 * When the tensors are sharded over ranks, descs holds this rank's n_local tensors, layer_of[i] is the
 * position of local tensor i among all n_total tensors (NULL: identity), rank_onehot is [n_local][5]; the
 * caller zeroes x_in first and sums it over the ranks afterwards.
 * velo_rnn: mix layers, LSTM cell, control and step-size heads, bank mixing (VeLO_RNN.py:110-135,
 * VeLO_MLP.py:92-126).  Outputs: weights [T][160] (row per tensor, tensor order), lr_mult [T]. */
typedef struct pylo_velo_rnn {
  const float *mix2_w, *mix2_b, *fmix_w, *fmix_b; /* [H][30], [H] */
  const float *lstm_w, *lstm_b;                   /* [4H][2H], [4H] */
  const float *ctrl_w, *ctrl_b;                   /* [B][H], [B] */
  const float *step_w, *step_b;                   /* [H], [1] */
  const float* bank;                              /* [B][159] */
  float *h, *c;                                   /* [T][H] LSTM state, updated in place */
  float *x_in;                                    /* [T][30] */
  const int *status;                              /* device int: while it is not zero, h, c and the loss buffer are left as
                                                     they are (tensor_features' input was incomplete); may be NULL */
  float *xmix;                                    /* workspace [T][H] */
  float *gates;                                   /* workspace [2][T][4H] */
  float *controls;                                /* workspace [T][B] */
  float *weights;                                 /* out [T][160] */
  float *lr_mult;                                 /* out [T] */
  int32_t T, H, B;
  int32_t mixed;                                  /* 1: pylo_b200_velo_inputs has made xmix */
} pylo_velo_rnn;
/* The loss buffer (BufferLossAccumulators, velo_cuda.py:170-211): means[10], iteration, running_min[10], decays[10], and
 * the step's loss, a device scalar or (loss == NULL) value. */
typedef struct pylo_velo_loss {
  float* means;
  int32_t* iteration;
  float* running_min;
  const float* decays;
  const float* loss;
  float value;
  int32_t pad_;
} pylo_velo_loss;
/* velo_tensor_features also does finalize_moments for its tensors (leave that call out).  fraction: step / num_steps, of
 * which the nine time features are made (velo_cuda.py:155-162); lossbuf is a HOST pointer: the launch uses the features the buffer has after this step's loss, and velo_rnn, which must
 * follow with the same lossbuf, advances it (NULL there: it is left as it is). */
int pylo_b200_velo_tensor_features(const pylo_tensor_desc* descs, int n_local, const int32_t* layer_of,
                                   int n_total, const float* rank_onehot, float fraction,
                                   const pylo_velo_loss* lossbuf, float* x_in, void* stream);
int pylo_b200_velo_rnn(const pylo_velo_rnn* rnn, const pylo_velo_loss* lossbuf, void* stream);
/* velo_tensor_features and the first layer of velo_rnn in one launch, for all (up to 16) tensors of a model (made for up to 16 tiles each: every
 * CTA adds them all up; the same sums to the last bit up to 20), and H a multiple of 128 up to 512; velo_rnn with mixed = 1 comes next. */
int pylo_b200_velo_inputs(const pylo_tensor_desc* descs, const int32_t* layer_of, const float* rank_onehot, float fraction,
                          const pylo_velo_loss* lossbuf, const pylo_velo_rnn* rnn, void* stream);
/* The loss buffer's update and features alone, for a host with a front end of its own: writes loss9[9]. */
int pylo_b200_velo_loss_features(float* means, int32_t* iteration, float* running_min, const float* decays,
                                 const float* loss, float* loss9, void* stream);

/* All tables of one optimizer's tensors, and a step's phases over them in one call: PYLO_STEP_FRONT is rowcol_sums,
 * factor_update, state_moments (tiles in reverse), finalize_moments; PYLO_STEP_BACK is prep_apply and the apply kernels
 * (PYLO_STEP_APPLY_REST: the launch, if there is one of its own, of what is not FAST2D).  A host that times the phases gives
 * them one by one.  plan and prm are HOST pointers.  ctiles: items of pylo_b200_apply_adafac_tc where tensor_cores is set (the n_ctiles_gen
 * on units that are not FAST2D first), else of apply_adafac_cols / apply_packed, with the other units in tiles_slow. */
#define PYLO_STEP_SUMS 1
#define PYLO_STEP_FACTORS 2
#define PYLO_STEP_STATE 4
#define PYLO_STEP_MOMENTS 8
#define PYLO_STEP_PREP 16
#define PYLO_STEP_APPLY 32
#define PYLO_STEP_APPLY_REST 64
#define PYLO_STEP_FRONT (PYLO_STEP_SUMS | PYLO_STEP_FACTORS | PYLO_STEP_STATE | PYLO_STEP_MOMENTS)
#define PYLO_STEP_BACK (PYLO_STEP_PREP | PYLO_STEP_APPLY | PYLO_STEP_APPLY_REST)
#define PYLO_ROWCOL_ONE_LAUNCH 2368 /* items of rowcol_sums on FAST2D tensors up to which the GENERIC tensors' items join their launch */
#define PYLO_ROWCOL_KERNEL_APART 2960 /* the same where there are KERNEL items, with which the GENERIC tensors' go in either case: one or two \
                                       convolution weights beside matrices of 300 M elements (9216 items) 320 us joined, 261 apart; 85 M \
                                       (3168) 111 / 105; 31 M (3840) 60 / 60; 25 M (3072) 66 / 65; 21 M (2560) 47.5 / 49.8 */
#define PYLO_TC_ONE_LAUNCH 4736 /* items on FAST2D units below which one launch of apply_adafac_tc takes both kinds of items: \
                                  the variant that takes both is 2 % slower on FAST2D items (ViT-B/16 2700 / 2751 us per \
                                  step, two Llama-3-8B blocks 12640 / 12925), a launch more costs about 10 us (convolutions \
                                  of 11 M parameters with a 0.5 M classifier 308.6 / 302.7) */
typedef struct pylo_step_plan {
  const pylo_tensor_desc *tdesc, *desc; /* per tensor, per unit */
  const pylo_atile *atiles, *gitems, *pitems, *ctiles;
  const pylo_tile *tiles, *tiles_slow;
  const pylo_atile* rtiles; /* CELO2, VELO: items of apply_packed on matrices with tables whose rows are not aligned */
  const int32_t* mats;      /* the n_mats tensors that are not VEC1D, or NULL: the first n_mats */
  int *status, *host_status;
  int32_t n_tensors, n_units, n_atiles, n_gitems, n_pitems, n_ctiles, n_ctiles_gen, n_tiles, n_tiles_slow, tensor_cores;
  int32_t sum_tiles; /* 1: leave finalize_moments out and let prep_apply add up the tile partials, for units of up to
                        about 200 tiles (VELO, of any size: velo_tensor_features does it) */
  int32_t n_ragged, n_rtiles; /* of atiles, the first that are not on FAST2D tensors; of rtiles */
  int32_t small_cluster, small_slice, small_rows, small_cols; /* small_cluster > 0: SUMS, FACTORS and STATE, asked for together,
                        are one launch of pylo_b200_small_front */
  int32_t n_kernel; /* of atiles, those behind the first n_ragged that are on KERNEL tensors */
  int32_t n_mats;
  int32_t small_networks; /* clusters of small_front that make the networks; > 0: no prep_apply (ADAFAC with tensor_cores) */
  int32_t factor_threads; /* of factor_update */
  int32_t pad_;
} pylo_step_plan;
int pylo_b200_step(const pylo_step_plan* plan, const pylo_step_params* prm, int phases, void* stream);
/* Host only: adds 1 to n step counters (HOST pointers to doubles); first: the old value of the first, equal: whether all
 * old values were the same. */
int pylo_b200_advance_steps(double* const* steps, int n, double* first, int* equal);

#ifdef __cplusplus
}
#endif
#endif /* PYLO_B200_H */
