"""Host-side planning for the multi-tensor step: descriptor tables, tile lists, workspace.

The optimizer classes describe every tensor on the learned-optimizer path with
a :class:`LoTensor`; :class:`LoPlan` turns the list into the device-resident
tables the C ABI works on (include/pylo_b200.h) and issues the fixed launch
sequence of one step.  Nothing here touches tensor values on the host.
"""

from __future__ import annotations

import ctypes as C
from collections import Counter
from dataclasses import dataclass
from typing import List, NamedTuple, Optional, Sequence, Tuple

import numpy as np
import torch

from . import _lib as L


#: Tiles of a unit up to which phase P adds their partials up itself instead of a launch before it.  Every item of phase P
#: repeats its unit's sum (six rows at a time, a chain that grows with the tiles), the launch costs a fixed time.  AdafacLO and
#: CELO2, one to five units, us per step without and with the launch: 98 tiles 36.0 / 37.4, 112: 41.4 / 42.3, 160: 46.1 / 47.3,
#: 192: 45.5 / 47.2 and 75.3 / 75.7; 224: 48.3 / 48.0, 256: 43.1 / 42.4, 512: 58.8 / 56.4.  Ten to forty units of up to 112
#: tiles: 1.6 us less to 1.4 more.  Models of 14 to 216 units of 36 to 192 tiles (12 M to 290 M elements, steps of up to 9 ms;
#: the two phases alone): 3.3 us less to 0.4 more, and up to 2.1 more where over 2900 items read 300 K rows of partials again.
SUM_TILES_MOST = 192


#: CTAs of the launch that takes phases A to B of a small model, a cluster per tensor, that run at once (one per SM).
SMALL_CTAS = L.SM_COUNT


def _prod(xs) -> int:
    out = 1
    for x in xs:
        out *= int(x)
    return out


@dataclass
class LoTensor:
    """One tensor on the learned-optimizer path (all tensors fp32, contiguous, on one CUDA device)."""

    p: torch.Tensor
    m: torch.Tensor                     # (3,) + shape
    v: torch.Tensor                     # shape or (1,) + shape
    fac_r: Optional[torch.Tensor]       # [3] + shape[dr -> 1]; fewer than 2 dims: (3,) + shape
    fac_c: Optional[torch.Tensor]       # [3] + shape[dc -> 1]; fewer than 2 dims: (3,) + shape or None
    fdims: Optional[Tuple[int, int]]    # (dc, dr) or None for fewer than 2 dims
    rcm_axis: int = 0                   # axis of fac_r over which row_col_mean is taken
    lr: float = 1e-3
    wd: float = 0.0
    clip_norm: float = 0.0
    exp_mult: float = 0.0
    step_mult: float = 1.0
    out: Optional[torch.Tensor] = None  # CELO2 raw step
    w: Optional[torch.Tensor] = None    # network weights in family layout
    lr_mult: Optional[torch.Tensor] = None
    slice_last2: bool = False           # normalise features per matrix (last two axes) instead of per tensor
    peer_ptrs: Optional[Sequence[int]] = None  # device addresses of this parameter in the other ranks' buffers
    peer_multicast: bool = False  # peer_ptrs holds ONE multicast address that maps the parameter on every rank


def geometry(shape: Sequence[int], fdims):
    """(O, X, M, Y, I, r_is_a) of a contiguous tensor whose factored axes are fdims = (dc, dr)."""
    dc, dr = fdims
    ax, ay = (dc, dr) if dc < dr else (dr, dc)
    O = _prod(shape[:ax])
    X = int(shape[ax])
    M = _prod(shape[ax + 1:ay])
    Y = int(shape[ay])
    I = _prod(shape[ay + 1:])
    return O, X, M, Y, I, int(dr == ay)


#: how much of its blocks of 128 columns a convolution weight has to fill for the tensor-core sweep to take it as a matrix (a block's
#: empty lanes cost what full ones do), and from which size on: small ones are all latency, and fewer launches as matrices.  AdafacLO, 60 tensors of 50 K
#: elements, (n, c, 3, 3), us per step as matrices / the general way: c = 8 (0.56 full) 220 / 195, 16 (0.56) 200 / 188, 20 (0.70) 166 / 183,
#: 32 (0.75) 156 / 180, 24 (0.84) 149 / 176, 64 (0.90) 138 / 175; (n, 20, 2, 2) (0.63) 210 / 188; of 17 K elements 101 / 94, 96 / 91, 85 / 86;
#: 32 of (64, 16, 3, 3) 44 / 52
KERNEL_FULL, KERNEL_FULL_FROM = 2 / 3, 32768


def fill_geometry(d, shape: Sequence[int], fdims, rcm_axis: int, sliced: bool = False, tensors=(), full: float = 0.0):
    """The descriptor fields of a tensor of this shape that say how it is walked through; ``sliced``: its features are
    normalised per matrix, ``tensors``: what has to be aligned for the fast mode, ``full``: see KERNEL_FULL.  Returns its (O, X, M, Y, I) and whether the mode
    is FAST2D, or None for fewer than 2 dims."""
    d["n"] = n = _prod(shape)
    if fdims is None:
        d["mode"] = L.MODE_VEC1D
        d["O"] = d["X"] = d["M"] = d["I"] = 1
        d["Y"] = min(n, 2**31 - 1)
        d["r_is_a"] = 1
        d["rcm_pre"] = d["rcm_A"] = d["rcm_post"] = 1
        return None
    O, X, M, Y, I, r_is_a = geometry(shape, fdims)
    d["O"], d["X"], d["M"], d["Y"], d["I"], d["r_is_a"] = O, X, M, Y, I, r_is_a
    d["La"], d["Lb"] = n // Y, n // X
    rshape = [3] + list(shape)   # of the row accumulator
    rshape[1 + fdims[1]] = 1
    d["rcm_pre"], d["rcm_A"], d["rcm_post"] = _prod(rshape[:rcm_axis]), rshape[rcm_axis], _prod(rshape[rcm_axis + 1:])
    vec = O == 1 and M == 1 and Y * I % 4 == 0 and n < 2**31 and not sliced and _aligned16(*tensors)
    fast = vec and I == 1
    # convolution weights of at least half a block of 128 columns: matrices whose row vectors have an entry per position (5 M parameters
    # of 3x3 convolutions, AdafacLO, us per step 275 -> 228: state 60 -> 46, network 160 -> 128; 205 with the sums in one launch)
    kernel = vec and 1 < I <= 32 and Y * I >= 64 and (n < KERNEL_FULL_FROM or Y * I >= full * 128 * -(-Y * I // 128))
    d["mode"] = L.MODE_FAST2D if fast else L.MODE_KERNEL if kernel else L.MODE_GENERIC
    return O, X, M, Y, I, fast


def _aligned16(*tensors) -> bool:
    return all(t is None or t.data_ptr() % 16 == 0 for t in tensors)


def make_tiles(sizes: Sequence[int], elems: int = L.TILE_ELEMS) -> Tuple[np.ndarray, List[Tuple[int, int]]]:
    """Element-wise tiles of ``elems`` elements over items of the given sizes; returns (tiles, [(tile0, n_tiles)] per item)."""
    counts = (np.asarray(sizes, dtype=np.int64) + elems - 1) // elems
    first = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    tiles = np.zeros(int(first[-1]), dtype=L.TILE_DTYPE)
    owner = np.repeat(np.arange(len(counts)), counts)
    tiles["tensor"] = owner
    tiles["start"] = (np.arange(len(tiles), dtype=np.int64) - first[owner]) * elems
    tiles["elems"] = elems
    return tiles, list(zip(first[:-1].tolist(), counts.tolist()))


def equal_tiles(sizes: Sequence[int], k: int) -> Tuple[np.ndarray, List[Tuple[int, int]]]:
    """:func:`make_tiles` with exactly ``k`` tiles per item (the last ones may be empty), of a multiple of four elements."""
    elems = -(-np.asarray(sizes, dtype=np.int64) // (4 * k)) * 4
    tiles = np.zeros(len(sizes) * k, dtype=L.TILE_DTYPE)
    tiles["tensor"], tiles["elems"] = np.repeat(np.arange(len(sizes)), k), np.repeat(elems, k)
    tiles["start"] = (elems[:, None] * np.arange(k)).reshape(-1)
    return tiles, [(k * i, k) for i in range(len(sizes))]


def plain_matrices(d: np.ndarray) -> np.ndarray:
    """Which descriptors are of contiguous matrices whose row_col_mean is over a whole vector or over the decays."""
    Lr = np.where(d["r_is_a"] != 0, d["La"], d["Lb"])
    whole = (d["rcm_pre"] == 3) & (d["rcm_A"] == Lr) & (d["rcm_post"] == 1)
    decays = (d["rcm_pre"] == 1) & (d["rcm_A"] == 3) & (d["rcm_post"] == Lr)
    return (d["O"] == 1) & (d["M"] == 1) & (d["I"] == 1) & (whole | decays)


def tile_elems(total: int, least: int, tiles_wanted: int) -> int:
    """Elements per tile for ``total`` elements of work: the largest power of two up to ``L.TILE_ELEMS`` that still gives
    ``tiles_wanted`` tiles (enough CTAs to fill the GPU), and never less than ``least`` (one pass of a CTA)."""
    e = L.TILE_ELEMS
    while e > least and total < e * tiles_wanted:
        e //= 2
    return e


_TILES = np.arange(L.TILE_ELEMS, 0, -1024, dtype=np.int64)   # what a tile of the state sweep may have: multiples of a CTA's pass


def state_tile(sizes: Sequence[int], alike: bool = False, slow: int = 0) -> int:
    """Elements per tile of the state sweep over units of these sizes: the multiple of 1024 (one pass of a CTA) with which the CTAs that
    run at once, two per SM, have least to do in their turns, where that saves a tenth over the power of two that gives four CTAs per
    SM a tile.  A tile's start and its block reduction cost about three passes.

    Units that are read element by element across inner axes take longer and, as a model's first tensors, come last: ``slow`` is the
    largest such unit, and in one turn a tile that is no more than a part of it costs as much again.  Two turns
    are the best number only where all units go the same way (``alike``).  us per step in one turn / two / three: VeLO on ViTs, 3.9 M 157 / 146 / 139,
    2.9 M 133 / 125 / 119; AdafacLO on convolutions, 4.7 M - / 174 / 163, 2.7 M 121 / 129 / 124.  Alike: VeLO on transformers, 5.3 M
    - / 146 / 152, 4.8 M - / 132 / 138, AdafacLO on 8.6 M - / 287 / 293, CELO2 on perceptrons of 4.5 M 162 / 162 / 163.  Over 202 models of
    all kinds from 0.4 to 50 M a step takes 0.87 to 1.02 of what it took with whole turns for all kinds alike (saving a sixth, a pass for the
    start, never two turns), 0.90 to 1.02 of what it takes with the power of two, and 0.6 % more than with the best tile; over 60 further
    ones 0.86 to 1.04 and 0.92 to 1.03."""
    at_once, total = 2 * L.SM_COUNT, sum(sizes)
    plain = tile_elems(total, 1024, 4 * L.SM_COUNT)
    if not 0 < total <= 16 * at_once * L.TILE_ELEMS:   # more turns than a better last one would show in
        return plain
    n, e = np.asarray(sizes, dtype=np.int64), _TILES[:, None]
    turns = -(-(-(-n // e)).sum(1) // at_once)
    cost = turns * (_TILES + 3072)
    if len(n) >= at_once:   # whole turns of units that are less than half a tile, CELO2's matrices: they cost what is in them
        short = 2 * n < e
        cost += (short * n).sum(1) // at_once - short.sum(1) // at_once * _TILES
    if slow:
        cost += (turns == 1) * (slow > _TILES) * _TILES
    if not alike:
        cost += (turns == 2) * (_TILES != plain) * cost[0]
    best = int(cost.argmin())
    return int(_TILES[best]) if cost[best] < 0.9 * cost[L.TILE_ELEMS // 1024 - plain // 1024] else plain


def atile_grid(tensor: int, n_strips: int, n_cb: int, tag: int = 0) -> np.ndarray:
    """Work items (tensor, strip, cb, tag) for every strip and column block."""
    a = np.empty((n_strips, n_cb, 4), dtype=np.int32)
    a[..., 0], a[..., 3] = tensor, tag
    a[..., 1] = np.arange(n_strips)[:, None]
    a[..., 2] = np.arange(n_cb)
    return a.reshape(-1, 4)


def atile_list(parts: List[np.ndarray]) -> np.ndarray:
    flat = np.concatenate(parts) if parts else np.empty((0, 4), dtype=np.int32)
    return np.ascontiguousarray(flat).view(L.ATILE_DTYPE).reshape(-1)


class DeviceTable:
    """A numpy structured array mirrored in device memory.  The first upload is an ordinary copy (most tables never see
    another); later ones go through two pinned staging buffers and do not wait."""

    def __init__(self, host: np.ndarray, device):
        self.host = host
        self.nbytes = max(host.nbytes, 16)
        self.dev = torch.empty(self.nbytes, dtype=torch.uint8, device=device)
        self._stage = None
        self._events = [None, None]
        self._turn = 0
        self._last = None
        self.upload()

    @property
    def ptr(self) -> int:
        return self.dev.data_ptr()

    def upload(self):
        """Copy the host array to the device unless it still holds exactly these bytes."""
        raw = self.host.view(np.uint8).reshape(-1) if self.host.nbytes else None
        if raw is not None and self._last is not None and np.array_equal(raw, self._last):
            return
        first, self._last = self._last is None, None if raw is None else raw.copy()
        if raw is None:
            return
        if first:
            self.dev.copy_(torch.from_numpy(raw))
            return
        if self._stage is None:
            self._stage = [torch.empty(self.nbytes, dtype=torch.uint8).pin_memory() for _ in range(2)]
        i = self._turn
        self._turn ^= 1
        if self._events[i] is not None:
            self._events[i].synchronize()
        self._stage[i].numpy()[: self.host.nbytes] = raw
        self.dev.copy_(self._stage[i], non_blocking=True)
        ev = torch.cuda.Event()
        ev.record()
        self._events[i] = ev


class FixedTable:
    """A table that stays as it is: its place is in one device buffer with the plan's others, copied there once (seven copies of a
    few hundred bytes each took a tenth of the time to build a small model's plan)."""

    def __init__(self, host: np.ndarray):
        self.host, self.ptr = host, 0

    @staticmethod
    def place(tables: Sequence["FixedTable"], device) -> torch.Tensor:
        ends = np.cumsum([(max(t.host.nbytes, 16) + 255) // 256 * 256 for t in tables])
        raw = np.zeros(int(ends[-1]), dtype=np.uint8)
        buffer = torch.empty(len(raw), dtype=torch.uint8, device=device)
        for t, at in zip(tables, [0] + ends[:-1].tolist()):
            raw[at:at + t.host.nbytes] = t.host.view(np.uint8).reshape(-1)
            t.ptr = buffer.data_ptr() + at
        buffer.copy_(torch.from_numpy(raw))
        return buffer


def apply_tile_shape(family: int, X: int, Y: int, least: int = 8):
    """(rows per work item, columns per work item, tag for ``pylo_atile.pad_``) of a FAST2D tensor's apply sweep on the CUDA
    cores.

    * AdafacLO family: n_sub sub-tiles of 32 rows in one block of 32..256 columns, as long as possible while the tensor
      still yields >= 8 items per SM; tag = columns | n_sub << 16;
    * CELO2 / VeLO: four columns per thread, 16 rows per thread (see :func:`packed_rows`), tag = threads per row (at least
      ``least``).
    """
    if family == L.FAM_ADAFAC:
        cw = min((256, 128, 64, 32), key=lambda c: ((Y + c - 1) // c * c - Y, -c))
        ncol = (Y + cw - 1) // cw
        n_sub = next((k for k in (8, 4, 2) if ((X + 32 * k - 1) // (32 * k)) * ncol >= 1184), 1)
        return 32 * n_sub, cw, cw | (n_sub << 16)
    tpr = min([c for c in (256, 128, 64, 32, 16, 8) if c >= least], key=lambda c: ((Y + 4 * c - 1) // (4 * c) * 4 * c - Y, -c))
    return 16 * (256 // tpr), 4 * tpr, tpr


def tensor_core_rows(shapes: Sequence[Tuple[int, int]]) -> int:
    """Rows of an item of the tensor-core sweep (rows x 128 columns, taken by one warpgroup) over tensors of these (rows,
    columns): the height that makes the busiest worker's share shortest, over all tensors together; an item's set-up costs
    about one and a half rows.  86 M ViT-B/16 parameters: 64 rows instead of 8, sweep 2050 -> 1750 us."""
    xs = np.array([X for X, _ in shapes], dtype=np.int64)
    cols = np.array([-(-Y // 128) for _, Y in shapes], dtype=np.int64)
    share = lambda R: -(-int((-(-xs // R) * cols).sum()) // L.TC_WORKERS) * (R + 1.5)
    return min((64, 32, 16, 8, 4, 2, 1), key=share)


def packed_rows(tiles: Sequence[Tuple[int, int, int, int]]) -> int:
    """Rows per thread of the packed sweep (CELO2, VeLO) over tensors of these (rows, columns, rows and columns of a tile at 16
    rows per thread): 64 (a tile's start costs about a row's time), fewer while the model does not give every SM its two
    CTAs several tiles each."""
    n_items = lambda k: sum(-(-X // (rt * k // 16)) * -(-Y // w) for X, Y, rt, w in tiles)
    return next((k for k in (64, 32, 16, 8, 4) if n_items(k) >= (16 if k > 16 else 4) * L.SM_COUNT), 2)


def ragged_rows(family: int, tiles: Sequence[Tuple[int, int, int, int]]) -> int:
    """Rows per thread of the packed sweep over matrices whose rows are not aligned: the number that makes the longest share of a
    CTA shortest; a tile's start counts as a row (VeLO over 3.4 M parameters, us per step with 4, 8, 16, 32 rows: 128.3, 128.8,
    134.9, 171.2, over 33 M 576.9, 551.2, 550.1, 557.2; CELO2 over 3.4 M 141.1, 134.7, 144.1, 144.6)."""
    ctas = L.SM_COUNT * (2 if family == L.FAM_VELO else 1)
    n_items = lambda k: sum(-(-X // (rt * k // 16)) * -(-Y // w) for X, Y, rt, w in tiles)
    return min((64, 32, 16, 8, 4), key=lambda k: -(-n_items(k) // ctas) * (k + 1))


def apply_items(family: int, tensor_cores: bool, fast, slow, least: int = 8, kernel=()) -> np.ndarray:
    """Work list of the tiled apply sweep: ``fast`` = [(unit, rows, columns)] of the FAST2D units, ``slow`` = [(unit,
    elements)] of the others, which only the tensor-core kernel takes (as runs of 128 elements, first in the list), ``kernel`` =
    [(unit, rows, columns)] of the KERNEL ones, which it takes as matrices of all positions' columns (next in the list)."""
    if tensor_cores:
        kernel = list(kernel)
        slow = [(u, -(-n // 128), 128) for u, n in slow]
        rows = lambda parts: tensor_core_rows([(X, Y) for _, X, Y in parts])
        gen = both = rows(slow + kernel + fast)
        if sum(-(-X // both) * -(-Y // 128) for _, X, Y in fast) >= L.TC_ONE_LAUNCH and slow + kernel:
            # A large model's slow units have a launch of their own, which is over when its longest item is: their height follows
            # from them alone.  At the FAST2D units' 64 rows a ViT-B/16's patch embedding was 72 items of 64 tiles for 592
            # workers, and the SMs that had them came late to the FAST2D launch (133 us by itself, now 21)
            gen, both = rows(slow + kernel), rows(fast)
        parts = [(u, X, Y, gen, 128, L.TC_GEN_ITEM | gen) for u, X, Y in slow] + [(u, X, Y, gen, 128, gen) for u, X, Y in kernel] + [(u, X, Y, both, 128, both) for u, X, Y in fast]
    else:
        parts = [(u, X, Y) + apply_tile_shape(family, X, Y, least) for u, X, Y in fast]
        if family != L.FAM_ADAFAC:
            shapes = [(X, Y, rt, w) for _, X, Y, rt, w, _ in parts]
            k = packed_rows(shapes) if least == 8 else ragged_rows(family, shapes)
            parts = [(u, X, Y, rt * k // 16, w, tag | k << 16) for u, X, Y, rt, w, tag in parts]
    return atile_list([atile_grid(u, -(-X // rt), -(-Y // w), tag) for u, X, Y, rt, w, tag in parts])


def small_front(mats: Sequence[Tuple[int, int]], vectors: Sequence[int]):
    """(CTAs per tensor, elements, rows and columns of the largest share) with which ``pylo_b200_small_front`` takes tensors of
    these (rows, columns) and these vectors, or None: as many CTAs a tensor as all run at once, or as few as hold it where two
    turns do.

    us per step, three launches / one: six tensors (118 K elements, 16 CTAs each) 33.9 / 28.5, fourteen (26 K) with 8 CTAs
    30.7 / 23.7 (with 16, two turns: 29.2), 28 (462 K, 8 CTAs, two turns) 48.3 / 46.6, 124 (533 K, 2 CTAs, two turns) 83.7 /
    63.0, eight of odd sizes (325 K, 16 CTAs) 56.8 / 43.1; three turns: 76 (1.3 M, 16 CTAs) 98 / 137."""
    T = len(mats) + len(vectors)

    def share(cl):
        rows = max([-(-X // cl) for X, _ in mats], default=0)
        cols = max([Y for _, Y in mats], default=0)
        most = max([-(-X // cl) * Y for X, Y in mats], default=0)
        floats = 6 * (-(-most // 4) * 4) + 4 * (-(-rows // 4) * 4) + 5 * (-(-cols // 4) * 4)
        fits = most <= L.SMALL_SLICE and floats <= L.SMALL_FLOATS and max(vectors, default=0) <= cl * L.SMALL_SLICE
        return (cl, most, rows, cols) if fits else None

    found = next((q for q in map(share, [cl for cl in (16, 8, 4, 2, 1) if T * cl <= SMALL_CTAS]) if q), None)
    return found or next((q for q in map(share, [cl for cl in (1, 2, 4, 8, 16) if T * cl <= 2 * SMALL_CTAS]) if q), None)


def small_networks(n_tensors: int, cluster: int) -> bool:
    """Whether one more cluster of this size makes the networks of the tensor-core sweep: where each of its CTAs has two at most (they
    take 3 us each, the tensors' own work 11; the 101 vectors of a ViT-B/16 in clusters of two CTAs: 170 us), and it costs no
    further turn: a cluster lies in one of eight groups of at least 18 SMs."""
    at_once = 8 * (18 // cluster)
    return n_tensors <= 2 * cluster and -(-(n_tensors + 1) // at_once) == -(-n_tensors // at_once)


class SumOrder(NamedTuple):
    """How the sums over a tensor are made.  All of it decides in which order a tensor's terms are added up."""

    small: Optional[Tuple[int, int, int, int]]   # see small_front
    elems: int          # elements of a tile where that does not cut the tensors
    sum_tiles: bool     # no launch for phase B2: of small units phase P adds the tile partials up, for VeLO the LSTM's input kernel does
    bulk_copies: bool   # the state sweep reads through a ring of bulk copies
    factor_threads: int = 1024   # per CTA of the factor phase

    def tiles(self, sizes):
        return equal_tiles(sizes, self.small[0]) if self.small else make_tiles(sizes, self.elems)


def sum_order(family: int, d: np.ndarray, sizes: Sequence[int], modes: np.ndarray, sliced: bool) -> SumOrder:
    """The rule, for tensors with these descriptors and their units of these sizes and modes.

    Tiles: see :func:`state_tile`.

    The state sweep's ring of bulk copies leaves little L1 cache to the units that are not FAST2D and keeps the launches around it
    apart, so it has to have enough to do: from 64 M elements on (VeLO on 100 M: 1615 -> 1580 us per step, on 17 M: 341 -> 351;
    AdafacLO on 25 M: 837 -> 851, on 86 M even), nearly all of them FAST2D.

    The factor phase has a cluster of eight CTAs per tensor with factors: half as many threads each where not all run at once."""
    total, small = int(sum(sizes)), None
    if not sliced and total <= 2 * SMALL_CTAS * L.SMALL_SLICE:
        vectors = d["mode"] == L.MODE_VEC1D
        if (vectors | plain_matrices(d)).all():
            small = small_front(list(zip(d["X"][~vectors].tolist(), d["Y"][~vectors].tolist())), d["n"][vectors].tolist())
    elems = L.TILE_ELEMS
    if small is None:
        across = modes == L.MODE_GENERIC   # inner axes between an element and the next of its row
        if across.any() and not sliced:
            across &= ~plain_matrices(d)
        slow = max([sizes[u] for u in np.flatnonzero(across)], default=0)
        elems = state_tile(sizes, not slow and not (modes == L.MODE_KERNEL).any(), slow)
    most = small[0] if small else -(-max(sizes, default=0) // elems)
    fast = int(sum(n for n, m in zip(sizes, modes.tolist()) if m == L.MODE_FAST2D))
    together = int((d["mode"] != L.MODE_VEC1D).sum()) * L.FACTOR_CLUSTER <= L.SM_COUNT
    return SumOrder(small, elems, family == L.FAM_VELO or most <= SUM_TILES_MOST, fast >= L.BULK_COPY_ELEMS and 8 * fast >= 7 * total,
                    1024 if together else 512)


def model_shapes(params) -> Optional[Sequence[Tuple[int, ...]]]:
    """The shapes of all tensors of the model that these parameters are a rank's share of (the sharded steps of
    :mod:`pylo_b200.zero` note them), or None where there is no such note or it does not fit them."""
    noted = [getattr(p, "_pylo_model_shapes", None) for p in params]
    first = noted[0] if noted else None
    return first if first is not None and all(q is first or q == first for q in noted) and share_of(params, first) else None


def share_of(params, shapes) -> bool:
    """Whether these parameters can be some of a model's tensors of these shapes."""
    return not Counter(tuple(p.shape) for p in params) - Counter(shapes)


class LoPlan:
    """Descriptor tables, tile lists and workspace for the tensors of one optimizer instance.

    Two tables: one descriptor per tensor (phases A and A2 work on whole tensors) and one per
    unit of element-wise work (phases B to C).  A unit is a tensor, or one matrix slice of a
    tensor flagged ``slice_last2``; when nothing is sliced the two tables are one.
    """

    H = {L.FAM_ADAFAC: 32, L.FAM_CELO2: 8, L.FAM_VELO: 4}

    def __init__(self, family: int, tensors: List[LoTensor], device, tensor_cores=False, model=None):
        """``model``: (shape, factored axes, rcm_axis) of all tensors of the model, in any order, of which ``tensors`` are a rank's
        share; their step is then the one that a plan over the whole model makes, to the last bit."""
        self.family = family
        # whether the AdafacLO family's FAST2D tensors take the tensor-core apply kernel
        self.tensor_cores = bool(tensor_cores) and family == L.FAM_ADAFAC
        self.tensors = tensors
        self.device = torch.device(device)
        T = len(tensors)
        H = self.H[family]
        full = KERNEL_FULL if self.tensor_cores else 0.0
        tdesc = np.zeros(T, dtype=L.DESC_DTYPE)
        ws_items = []  # (table, row, field, count)
        atiles, ratiles, katiles, gitems = [], [], [], []
        ws_bytes = 0  # the library's own count of the workspace, checked against the layout below
        for i, t in enumerate(tensors):
            shape = tuple(t.p.shape)
            n = t.p.numel()
            if n == 0:
                raise ValueError("empty parameter tensors are not supported on the learned-optimizer path")
            for name in ("p", "m", "v", "fac_r", "fac_c", "out"):
                x = getattr(t, name)
                if x is not None and not (x.is_cuda and x.dtype == torch.float32 and x.is_contiguous()):
                    raise ValueError(f"{name} of tensor {i} must be a contiguous fp32 CUDA tensor")
            d = tdesc[i]
            d["m_stride"], d["idx0"] = n, 0
            sliced = t.slice_last2 and len(shape) > 2
            sides = fill_geometry(d, shape, t.fdims, t.rcm_axis, sliced, (t.p, t.m, t.v, t.out), full)
            d["lr"], d["wd"], d["clip_norm"] = t.lr, t.wd, t.clip_norm
            d["exp_mult"], d["step_mult"] = t.exp_mult, t.step_mult
            d["p"], d["m"], d["v"] = t.p.data_ptr(), t.m.data_ptr(), t.v.data_ptr()
            d["out"] = t.out.data_ptr() if t.out is not None else 0
            d["w"] = t.w.data_ptr() if t.w is not None else 0
            d["lr_mult"] = t.lr_mult.data_ptr() if t.lr_mult is not None else 0
            if t.peer_ptrs:
                if len(t.peer_ptrs) > L.MAX_PEERS:
                    raise ValueError(f"at most {L.MAX_PEERS} peers (8 GPUs of one box)")
                d["p_peer"][: len(t.peer_ptrs)] = list(t.peer_ptrs)
                d["n_peer"] = -1 if t.peer_multicast else len(t.peer_ptrs)
            if t.fdims is None:
                ws = L.workspace_layout(family, L.MODE_VEC1D, n)
                d["fac_a"] = t.fac_r.data_ptr()
                d["fac_b"] = t.fac_c.data_ptr() if t.fac_c is not None else 0
            else:
                O, X, M, Y, I, fast = sides
                La, Lb = n // Y, n // X
                fac_a, fac_b = (t.fac_r, t.fac_c) if t.fdims[1] > t.fdims[0] else (t.fac_c, t.fac_r)
                d["fac_a"], d["fac_b"] = fac_a.data_ptr(), fac_b.data_ptr()
                # matrices whose rows are not aligned go the way of the others with single accesses, where a warp finds its 32
                # columns twice: 3.4 M VeLO parameters in rows of 1433 and 1001, sums 25.8 -> 13.5 us, apply sweep 68 -> 33
                ragged = not fast and not sliced and O == M == I == 1 and Y >= 64
                # sub-buffer sizes and the phase-A tiling come from the library (pylo_b200_workspace_layout), so that
                # this table and a table built by any other host of the C ABI agree
                kernel = int(d["mode"]) == L.MODE_KERNEL
                in_atiles = fast or ragged or kernel
                ws = L.workspace_layout(family, int(d["mode"]), n, La, Lb, X if in_atiles else 0, Lb if in_atiles else 0)
                if self.tensor_cores:   # the tensor-core sweep reads no tables
                    ws.h_a = ws.h_b = 0
                ws_items += [("t", i, f, getattr(ws, f)) for f in ("f_a", "f_b", "sum_a", "sum_b")]
                d["rb"], d["n_strips"], d["n_cb"] = ws.rb, ws.n_strips, ws.n_cb
                if in_atiles:
                    ws_items += [("t", i, f, getattr(ws, f)) for f in ("fx", "part_a", "part_b", "h_a", "h_b") if getattr(ws, f)]
                    (ratiles if ragged else katiles if kernel else atiles).append(atile_grid(i, ws.n_strips, ws.n_cb))
                else:
                    ws_items.append(("t", i, "part_b", ws.part_b))
                    gitems.append(atile_grid(i, ws.n_strips, (Lb + 255) // 256, 1))
                    per = max(1, 4096 // (Y * I))  # blocks of Y*I elements per row-sum item: about 4 K elements
                    rows = atile_grid(i, (La // I + per - 1) // per, 1)
                    rows[:, 2] = per
                    gitems.append(rows)
            ws_items.append(("t", i, "closed", L.STAT_STRIDE))
            ws_bytes += L.lib.pylo_b200_workspace_bytes(C.byref(ws), 1, 0)

        # units of element-wise work
        self.sliced = any(t.slice_last2 and t.p.dim() > 2 for t in tensors)
        unit_owner = []  # (tensor index, element offset)
        for i, t in enumerate(tensors):
            if t.slice_last2 and t.p.dim() > 2:
                mat = t.p.shape[-1] * t.p.shape[-2]
                unit_owner += [(i, k * mat) for k in range(t.p.numel() // mat)]
            else:
                unit_owner.append((i, 0))
        U = len(unit_owner)
        if self.sliced:
            udesc = np.zeros(U, dtype=L.DESC_DTYPE)
            for u, (i, off) in enumerate(unit_owner):
                udesc[u] = tdesc[i]
                t = tensors[i]
                if t.slice_last2 and t.p.dim() > 2:
                    mat = t.p.shape[-1] * t.p.shape[-2]
                    udesc["n"][u], udesc["idx0"][u], udesc["vec_elementwise"][u] = mat, off, 1
                    for f in ("p", "m", "v", "out"):
                        if udesc[f][u]:
                            udesc[f][u] += 4 * off
                    ws_items.append(("u", u, "closed", L.STAT_STRIDE))  # stays zero: no closed forms for a slice
                    ws_bytes += (L.STAT_STRIDE + 63) // 64 * 256
        else:
            udesc = tdesc
        sizes = [int(udesc["n"][u]) for u in range(U)]
        if model is None:
            order = sum_order(family, tdesc, sizes, udesc["mode"], self.sliced)
        else:
            whole = np.zeros(len(model), dtype=L.DESC_DTYPE)
            for d, (shape, fdims, rcm_axis) in zip(whole, model):
                fill_geometry(d, shape, fdims, rcm_axis, full=full)   # the other ranks' buffers are aligned
            order = sum_order(family, whole, whole["n"].tolist(), whole["mode"], False)
        self.small = order.small   # as many tiles a tensor as CTAs take its rows
        tiles, ranges = order.tiles(sizes)
        for u, (t0, k) in enumerate(ranges):
            udesc["tile0"][u], udesc["n_tiles"][u] = t0, k
            ws = L.workspace_layout(family, L.MODE_VEC1D, sizes[u])  # the per-unit part depends on the element count only
            ws.n_tiles, ws.tile_part = k, k * L.STAT_STRIDE
            ws_items += [("u", u, f, getattr(ws, f)) for f in ("sums", "wfold", "tile_part")]
            ws_bytes += L.lib.pylo_b200_workspace_bytes(C.byref(ws), 0, 1)
        # workspace: every sub-buffer starts on a 256-byte boundary
        off = 0
        placed = []
        for table, row, fld, count in ws_items:
            placed.append((table, row, fld, off))
            off += (count + 63) // 64 * 64
        if off * 4 != ws_bytes:
            raise AssertionError(f"workspace layout ({off * 4} bytes) disagrees with pylo_b200_workspace_bytes ({ws_bytes})")
        self.workspace = torch.zeros(max(off, 64), dtype=torch.float32, device=self.device)
        base = self.workspace.data_ptr()
        for table, row, fld, o in placed:
            (tdesc if table == "t" else udesc)[fld][row] = base + 4 * o
        if self.sliced:  # units inherit their tensor's factor workspace
            for u, (i, _) in enumerate(unit_owner):
                for f in ("f_a", "f_b", "fx", "sum_a", "sum_b", "part_a", "part_b", "h_a", "h_b"):
                    udesc[f][u] = tdesc[f][i]
                if not udesc["vec_elementwise"][u]:
                    udesc["closed"][u] = tdesc["closed"][i]
        self.unit_owner = unit_owner
        self.tdesc = DeviceTable(tdesc, self.device)
        self.desc = DeviceTable(udesc, self.device) if self.sliced else self.tdesc
        self.tiles = FixedTable(tiles)
        self.n_tiles = len(tiles)
        self.atiles = FixedTable(atile_list(ratiles + katiles + atiles))
        self.n_atiles, self.n_ragged = len(self.atiles.host), len(atile_list(ratiles))
        self.gitems = FixedTable(atile_list(gitems))
        self.n_gitems = len(self.gitems.host)
        self.mats = FixedTable(np.flatnonzero(tdesc["mode"] != L.MODE_VEC1D).astype(np.int32))   # the tensors with factors
        self.n_mats = len(self.mats.host)
        self.n_tensors = T
        self.n_units = U
        self.total_elems = int(sum(sizes))
        self._keepalive = []
        # FAST2D tensors take a tiled apply kernel (see apply_items); everything else the generic one, or, with
        # tensor cores, items of the same kernel
        fast, kernel = [], []
        # phase P: item 0 of every unit folds the network, the further ones (and item 0) make the tables' parts
        pitems = [np.zeros((U, 4), dtype=np.int32)]
        pitems[0][:, 0] = np.arange(U)
        per = L.PREP_TABLE // H
        unit_of = {i: u for u, (i, _) in enumerate(unit_owner)}  # a FAST2D tensor is never sliced: one unit
        ragged = []
        for i in range(T):
            X, Y = int(tdesc["X"][i]), int(tdesc["Y"][i])
            if tdesc["mode"][i] == L.MODE_KERNEL and self.tensor_cores:
                kernel.append((unit_of[i], X, Y * int(tdesc["I"][i])))
            if tdesc["mode"][i] != L.MODE_FAST2D and not tdesc["h_a"][i]:
                continue
            if tdesc["h_a"][i]:   # the tables' parts
                pitems.append(atile_grid(unit_of[i], (X + per - 1) // per + (Y + per - 1) // per, 1)[1:])
            (fast if tdesc["mode"][i] == L.MODE_FAST2D else ragged).append((unit_of[i], X, Y))
        tiled = {u for u, _, _ in fast + ragged + kernel}
        slow_units = [u for u in range(U) if u not in tiled]
        self.ctiles = FixedTable(apply_items(family, self.tensor_cores, fast, [(u, sizes[u]) for u in slow_units], kernel=kernel))
        self.n_ctiles = len(self.ctiles.host)
        self.rtiles = FixedTable(apply_items(family, False, ragged, [], 32))
        self.n_rtiles = len(self.rtiles.host)
        #: how many of them, at the front of the list, are on tensors that are not FAST2D (tensor cores only)
        self.n_ctiles_gen = int((~np.isin(self.ctiles.host["tensor"], [u for u, _, _ in fast])).sum()) if self.tensor_cores else 0
        self.pitems = FixedTable(atile_list(pitems))
        self.n_pitems = len(self.pitems.host)
        #: the kernel that takes the FAST2D tensors' apply sweep (also the key of its timings in phase_times())
        if self.tensor_cores:
            self.apply_kernel = "k_apply_adafac_tc"
        elif family == L.FAM_ADAFAC:
            self.apply_kernel = "k_apply_adafac_cols"
        else:
            self.apply_kernel = "k_apply_packed<CELO2>" if family == L.FAM_CELO2 else "k_apply_packed<VELO>"
        #: device flag that a kernel raises when one of its bounded waits ran out
        self.status = torch.zeros(128, dtype=torch.int32, device=self.device)
        # its twin in pinned host memory, written by the kernel itself: the next step looks at it without asking the device
        self._status_host = torch.zeros(1, dtype=torch.int32).pin_memory()
        self._status_view = self._status_host.numpy()
        # the other units' apply sweep: vectors are short and every element costs a whole network, so the tiles are as
        # small as one element per thread where that is what fills the GPU (five 4096-vectors: 104 us as one tile each)
        slow_units = [] if self.tensor_cores else slow_units
        slow_sizes = [sizes[u] for u in slow_units]
        slow, _ = make_tiles(slow_sizes, tile_elems(sum(slow_sizes), 256, 4 * L.SM_COUNT))
        slow["tensor"] = np.asarray(slow_units, dtype=np.int32)[slow["tensor"]] if len(slow) else slow["tensor"]
        self.tiles_slow = FixedTable(slow)
        self.n_tiles_slow = len(slow)
        self._fixed = FixedTable.place([self.tiles, self.atiles, self.gitems, self.ctiles, self.rtiles, self.pitems, self.tiles_slow, self.mats], self.device)
        self.sum_tiles, self.bulk_copies = order.sum_tiles, int(order.bulk_copies)
        #: everything pylo_b200_step needs for a step over these tensors
        self.step_plan = L.StepPlan(
            tdesc=self.tdesc.ptr, desc=self.desc.ptr, atiles=self.atiles.ptr, gitems=self.gitems.ptr, pitems=self.pitems.ptr,
            ctiles=self.ctiles.ptr, tiles=self.tiles.ptr, tiles_slow=self.tiles_slow.ptr, rtiles=self.rtiles.ptr, mats=self.mats.ptr if T * L.FACTOR_CLUSTER > L.SM_COUNT else 0,
            n_mats=self.n_mats if T * L.FACTOR_CLUSTER > L.SM_COUNT else T,   # few tensors: all of them, which costs nothing
            status=self.status.data_ptr(), host_status=self._status_host.data_ptr(),
            n_tensors=T, n_units=U, n_atiles=self.n_atiles, n_gitems=self.n_gitems, n_pitems=self.n_pitems,
            n_ctiles=self.n_ctiles, n_ctiles_gen=self.n_ctiles_gen, n_tiles=self.n_tiles, n_tiles_slow=self.n_tiles_slow, n_ragged=self.n_ragged, n_rtiles=self.n_rtiles,
            n_kernel=sum(len(a) for a in katiles), factor_threads=order.factor_threads,
            tensor_cores=int(self.tensor_cores), sum_tiles=int(self.sum_tiles))
        if self.small:
            (self.step_plan.small_cluster, self.step_plan.small_slice, self.step_plan.small_rows, self.step_plan.small_cols) = self.small
            self.step_plan.small_networks = int(self.tensor_cores and small_networks(T, self.small[0]))
        self._step_plan_ref = C.byref(self.step_plan)
        self._hyper = None          # what set_hyper last wrote
        self._grad_ptrs = None      # the gradient addresses the table holds
        self._step_base = None      # the step count the table holds for every tensor, where it is one
        self._dirty = True          # the host table is ahead of the device's
        self.step_delta = 0.0
        self._prof = None
        #: launches since construction (or since the caller zeroed it), and what each call of :meth:`run` adds
        self.launch_count = 0
        self._launches = {k: sum(n for ph, _, n in self._phases() if ph & k) for k in (L.STEP_FRONT, L.STEP_BACK, L.STEP_FRONT | L.STEP_BACK)}

    # ------------------------------------------------------------------ per-step refresh
    def set_field(self, name, values):
        """Set a per-tensor field (scalar or one value per tensor) in both tables."""
        self.tdesc.host[name][:] = values
        if self.sliced:
            vals = np.broadcast_to(np.asarray(values), (self.n_tensors,))
            self.desc.host[name][:] = [vals[i] for i, _ in self.unit_owner]

    def set_hyper(self, **fields):
        """Per-tensor fields (scalar or one value per tensor) as :meth:`set_field`, skipped where they are what they were."""
        if fields != self._hyper:
            for name, values in fields.items():
                self.set_field(name, values)
            self._hyper, self._dirty = fields, True

    def refresh(self, grads: Sequence[torch.Tensor], counters=None):
        """Point the descriptors at this step's gradients (and step counts) and upload the tables where that changed them.

        ``counters.advance()``, called once the gradients are accepted, gives the step count: one value for all tensors,
        or one per tensor."""
        ptrs = grad_pointers(grads)
        if ptrs is None or ptrs != self._grad_ptrs:
            self._grad_ptrs = ptrs
            self._keepalive = []
            at = np.zeros(self.n_tensors, dtype=np.uint64)
            for i, g in enumerate(grads):
                if not (g.is_cuda and g.dtype == torch.float32 and g.is_contiguous() and g.data_ptr() % 16 == 0):
                    g = g.detach().to(torch.float32).contiguous().clone()
                    self._keepalive.append(g)
                    self._grad_ptrs = None   # the copy is this step's: look again at the next
                at[i] = g.data_ptr()
            if not np.array_equal(self.tdesc.host["g"], at):
                self.tdesc.host["g"][:] = at
                if self.sliced:
                    self.desc.host["g"][:] = [at[i] + np.uint64(4 * off) for i, off in self.unit_owner]
                self._dirty = True
        self.step_delta = 0.0
        if counters is not None:
            steps = counters.advance()
            # when every tensor advanced by the same amount since the table was last written, leave the
            # table alone and hand the kernels the difference (no upload on the step path)
            one = isinstance(steps, float)
            delta = None
            if one and self._step_base is not None:
                delta = steps - self._step_base
            elif self.tdesc._last is not None:
                diff = np.asarray(steps, dtype=np.float64) - self.tdesc.host["step"].astype(np.float64)
                delta = float(diff[0]) if len(diff) and np.all(diff == diff[0]) else None
            if delta is not None and 0 <= delta < 2**20:
                self.step_delta = delta
            else:
                self.set_field("step", steps)
                self._dirty = True
            self._step_base = steps - self.step_delta if one else None
        if self._dirty:
            self.tdesc.upload()
            if self.sliced:
                self.desc.upload()
            self._dirty = False

    # ------------------------------------------------------------------ launch sequence
    #: the kernel that dominates each timed phase, for reports
    KERNEL_OF = {"rowcol_sums": "k_rowcol_fast", "factor_update": "k_factor_update", "state_moments": "k_state_moments",
                 "finalize_moments": "k_finalize_moments", "prep_apply": "k_prep_apply", "small_front": "k_small_front"}

    def _phases(self):
        """[(phase of pylo_b200_step, name, launches)] in the step's order, without those that launch nothing."""
        split = self.tensor_cores and self.n_ctiles - self.n_ctiles_gen >= L.TC_ONE_LAUNCH   # a launch of its own for what is not FAST2D
        rest = int(split and self.n_ctiles_gen > 0) if self.tensor_cores else int(self.n_tiles_slow > 0) + int(self.n_rtiles > 0)
        main = int(self.n_ctiles > (self.n_ctiles_gen if split else 0))
        other = "k_apply_adafac_tc<true>" if self.tensor_cores else "k_apply"
        apply = [(L.STEP_APPLY, self.apply_kernel if self.n_ctiles > self.n_ctiles_gen else other, main)]
        apply.insert(0 if self.tensor_cores else 1, (L.STEP_APPLY_REST, other, rest))
        if self.family == L.FAM_VELO and (self.n_ctiles or self.n_rtiles):   # the packed sweep takes the other units' tiles along
            apply = [(L.STEP_APPLY | L.STEP_APPLY_REST, self.apply_kernel, int(self.n_ctiles > 0) + int(self.n_rtiles > 0))]
        kernel = self.step_plan.n_kernel
        fast = self.n_atiles - self.n_ragged - kernel
        mixed = kernel > 0 or self.n_gitems > 0
        joined = mixed and 0 < fast <= (L.ROWCOL_KERNEL_APART if kernel else L.ROWCOL_ONE_LAUNCH)   # all kinds of items in one launch
        front = [(L.STEP_SUMS, "rowcol_sums", (self.n_ragged > 0) + int(mixed) + int(fast > 0 and not joined)),
                 (L.STEP_FACTORS, "factor_update", int(self.step_plan.n_mats > 0)),
                 (L.STEP_STATE, "state_moments", 1)]
        if self.small:
            front = [(L.STEP_SUMS | L.STEP_FACTORS | L.STEP_STATE, "small_front", 1)]
        phases = front + [(L.STEP_MOMENTS, "finalize_moments", int(not self.sum_tiles)),
                  (L.STEP_PREP, "prep_apply", int(not self.step_plan.small_networks))] + apply
        return [ph for ph in phases if ph[2]]

    def enable_profile(self, on: bool = True):
        """Record a CUDA-event pair around every phase (read back with :meth:`phase_times`): the launches are those of any
        other step, but each phase then waits for the end of the one before."""
        self._prof = {} if on else None

    def phase_times(self):
        """{phase: [ms, ...]} of the recorded launches; call after a device synchronisation."""
        return {k: [a.elapsed_time(b) for a, b in v] for k, v in (self._prof or {}).items()}

    def run(self, prm: L.StepParams, stream: int, phases: int = L.STEP_FRONT | L.STEP_BACK):
        """The phases of a step (all of them, or only those before or after the caller's own work in between)."""
        prm.step_delta = self.step_delta
        prm.status, prm.host_status = self.step_plan.status, self.step_plan.host_status
        prm.bulk_copies = self.bulk_copies
        self.launch_count += self._launches[phases]
        if self._prof is None:
            L.check(L.lib.pylo_b200_step(self._step_plan_ref, C.byref(prm), phases, stream), "step")
            return
        for phase, name, _ in self._phases():
            if phases & phase:
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                L.check(L.lib.pylo_b200_step(self._step_plan_ref, C.byref(prm), phase, stream), name)
                b.record()
                self._prof.setdefault(name, []).append((a, b))

    def poll_status(self):
        """Raise if a launch of an earlier step has written its status word: every optimizer's step begins with this, for all
        of its plans, before it advances anything of its own."""
        if self._status_view[0] != 0:
            raise L.PyloLibError("a bounded wait inside a kernel timed out in an earlier step: that step is incomplete, the "
                                 "parameters it could not finish kept their old values, and launches write no parameters until "
                                 "clear_status() is called")

    def check_status(self):
        """Synchronise and raise if a kernel reported a wait that ran out.

        Every kernel that writes parameters keeps the old value of those it could not finish, and of all of them where what
        it reads is incomplete, so no invalid parameter was written; but the step is incomplete (the accumulators may have
        advanced in part), and until :meth:`clear_status` no parameter is written at all.  Call this before a checkpoint
        is written."""
        code = int(self.status[0].item())
        if code & 8:
            raise L.PyloLibError("a wait for a kernel's own copies timed out; this step is incomplete")
        if code & 4:
            raise L.PyloLibError("a wait inside a Newton-Schulz kernel timed out; this step is incomplete")
        if code != 0:
            raise L.PyloLibError("apply_adafac_tc: a wait on the tensor core timed out; this step is incomplete "
                                 "(unfinished parameters kept their old values)")

    def clear_status(self):
        """Acknowledge a reported timeout: the next launches write parameters again."""
        self.status.zero_()
        torch.cuda.synchronize(self.device)   # a launch in flight may still write the host's word
        self._status_host.zero_()


class GradNorm:
    """Device-side sum of squares of a list of gradients (the global-norm clip)."""

    def __init__(self, sizes: Sequence[int], device):
        self.out = torch.zeros(1, dtype=torch.float32, device=device)
        self._keepalive = []
        self._grad_ptrs = None
        self.n_tiles = 0
        if len(sizes) == 0:   # a rank that owns no tensor still takes part in the all-reduce of the sum: with zero
            return
        self.items = np.zeros(len(sizes), dtype=L.GVEC_DTYPE)
        self.items["n"] = sizes
        tiles, _ = make_tiles(sizes)
        self.tiles = DeviceTable(tiles, device)
        self.n_tiles = len(tiles)
        self.table = DeviceTable(self.items, device)
        self.scratch = torch.zeros(max(self.n_tiles, 1), dtype=torch.float32, device=device)

    def run(self, grads: Sequence[torch.Tensor], stream: int):
        if self.n_tiles == 0:
            self.out.zero_()
            return self.out
        ptrs = grad_pointers(grads)
        if ptrs is None or ptrs != self._grad_ptrs:
            self._grad_ptrs = ptrs
            self._keepalive = []
            for i, g in enumerate(grads):
                plain = fp32_gradient(g)
                if plain is not g:
                    self._keepalive.append(plain)
                    self._grad_ptrs = None
                self.items["g"][i] = plain.data_ptr()
            self.table.upload()
        L.check(L.lib.pylo_b200_grad_sumsq(self.table.ptr, self.tiles.ptr, self.n_tiles, self.scratch.data_ptr(),
                                           self.out.data_ptr(), stream), "grad_sumsq")
        return self.out


def with_gradients(params):
    """(parameters that have a gradient, their gradients)."""
    grads = [p.grad for p in params]
    if any([g is None for g in grads]):
        params = [p for p, g in zip(params, grads) if g is not None]
        grads = [g for g in grads if g is not None]
    return params, grads


def grad_pointers(grads: Sequence[torch.Tensor]):
    """The gradients' addresses, or None where one of them is not contiguous fp32 and has to be looked at (an fp32 parameter
    may have a gradient of another type: ``p.grad_dtype``).  Looked at on every step: an address says nothing about the type
    of what lies there now."""
    try:
        ptrs = [g.data_ptr() for g in grads]
    except RuntimeError:
        if any(g.is_sparse for g in grads):
            raise RuntimeError("Sparse gradients not supported") from None
        raise
    return ptrs if all([g.dtype is torch.float32 and g.is_contiguous() for g in grads]) else None


def fp32_gradient(g: torch.Tensor) -> torch.Tensor:
    """``g`` as contiguous fp32: itself, or a copy."""
    return g if g.dtype is torch.float32 and g.is_contiguous() else g.detach().to(torch.float32).contiguous()


def current_stream_ptr() -> int:
    """The current stream of the current device (what ``torch.cuda.current_stream().cuda_stream`` says, without the object)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def one_minus(beta: torch.Tensor) -> List[float]:
    """``1 - beta`` evaluated in fp32, as ``1 - tensor`` does in the reference classes."""
    return [float(x) for x in (1 - beta.detach().to("cpu", torch.float32)).tolist()]
