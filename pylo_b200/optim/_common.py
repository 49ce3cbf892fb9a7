"""Pieces shared by the optimizer classes: factored-dims rules, Newton-Schulz, plan caching."""

from __future__ import annotations

import ctypes as C_
import functools
import sys
from typing import List, Optional, Sequence

import numpy as np
import torch
from torch.optim import Optimizer

from .. import _lib as L
from ..plan import DeviceTable, make_tiles


def factored_dims_sorted(shape):
    """(dc, dr): indices of the second-largest and largest axis, ties broken by index
    (AdafacLO_cuda.py:52-73 with min_dim_size_to_factor=1, ELO_cuda.py:46-51)."""
    if len(shape) < 2:
        return None
    order = sorted((s, i) for i, s in enumerate(shape))
    return int(order[-2][1]), int(order[-1][1])


def factored_dims_argsort(shape):
    """(dc, dr) via ``np.argsort`` (CELO2_naive.py:42-47)."""
    if len(shape) < 2:
        return None
    order = np.argsort(shape)
    return int(order[-2]), int(order[-1])


def factored_dims_velo(shape):
    """(dc, dr) with VeLO's tie rule: equal sizes swap unless 4-D with axes (0, 1) (velo_cuda.py:121-131)."""
    if len(shape) < 2:
        return None
    order = np.argsort(shape)
    a, b = int(order[-2]), int(order[-1])
    if shape[a] == shape[b] and not (len(shape) == 4 and a == 0 and b == 1):
        return b, a
    return a, b


def newton_schulz(x: torch.Tensor, coeffs, iters: int = 5, eps: float = 1e-8) -> torch.Tensor:
    """Quintic Newton-Schulz iteration towards the orthogonal factor of ``x`` over its last two axes.

    Same arithmetic, in the same order, as CELO2_naive.py:59-73: work on the wide
    orientation, divide by (Frobenius norm + eps), then ``iters`` times
    ``a = x x^T; b = c1 a + c2 a a; x = c0 x + b x``.  It is a chain of dense fp32
    GEMMs and stays on ``torch.matmul``.
    """
    tall = x.shape[-2] > x.shape[-1]
    if tall:
        x = x.transpose(-2, -1)
    x = x / (torch.linalg.norm(x, dim=(-2, -1), keepdim=True) + eps)
    c0, c1, c2 = coeffs
    for _ in range(iters):
        a = x @ x.transpose(-2, -1)
        b = c1 * a + c2 * (a @ a)
        x = c0 * x + b @ x
    return x.transpose(-2, -1) if tall else x


def _gemm_tn(A, B, C, D, alpha, beta, status, stream, symmetric=False):
    """C[b] = alpha * A[b] @ B[b]^T + beta * D[b] through ``pylo_b200_gemm_tn_3xtf32`` (3-D fp32 tensors whose last axis is
    contiguous).  ``symmetric``: the result is known to be symmetric; only the tiles on and above the diagonal are
    computed and the rest is filled in by mirroring."""
    g = L.GemmDesc()
    g.A, g.B, g.C, g.D = A.data_ptr(), B.data_ptr(), C.data_ptr(), (D.data_ptr() if D is not None else None)
    g.batch, g.M, g.K = A.shape
    g.N = B.shape[1]
    g.lda, g.ldb, g.ldc, g.ldd = A.stride(1), B.stride(1), C.stride(1), (D.stride(1) if D is not None else 0)
    g.strideA, g.strideB, g.strideC = A.stride(0), B.stride(0), C.stride(0)
    g.strideD = D.stride(0) if D is not None else 0
    g.alpha, g.beta = float(alpha), float(beta)
    g.symmetric = int(bool(symmetric))
    L.check(L.lib.pylo_b200_gemm_tn_3xtf32(C_.byref(g), status.data_ptr() if status is not None else None, stream),
            "gemm_tn_3xtf32")
    if symmetric:
        L.check(L.lib.pylo_b200_transpose(C.data_ptr(), C.data_ptr(), g.M, g.N, g.ldc, g.ldc, g.strideC, g.strideC, g.batch, 1,
                                          stream), "transpose(mirror)")


def _transpose(src, dst, stream):
    """dst[b] = src[b]^T for 3-D fp32 tensors whose last axis is contiguous."""
    nb, r, c = src.shape
    L.check(L.lib.pylo_b200_transpose(src.data_ptr(), dst.data_ptr(), r, c, src.stride(1), dst.stride(1), src.stride(0),
                                      dst.stride(0), nb, 0, stream), "transpose")


def newton_schulz_eligible(rows: int, cols: int) -> bool:
    """Whether the TF32 product kernel takes a matrix of this shape: both sides multiples of 4 (rows are moved in 16-byte
    pieces) and the short side at least 64 (half a tile)."""
    r, c = min(rows, cols), max(rows, cols)
    return r % 4 == 0 and c % 4 == 0 and r >= 64


@functools.lru_cache(maxsize=64)
def newton_schulz_bounded(coeffs, iters: int) -> bool:
    """Whether the iteration keeps every matrix small enough for planes of fp16 (|x| < 10, |a|, |b| < 15).

    All of them are polynomials of the singular values, which start in [0, 1]; their largest values are followed through
    the iterations on a fine grid.  The usual coefficients stay below 1.3."""
    c0, c1, c2 = coeffs
    if c2 != 0.0 and abs(c1) > 1e6 * abs(c2):   # the kernel adds c1 a / c2 to a a
        return False
    top = 1.0
    for _ in range(iters):
        s = np.linspace(0.0, top, 4001)
        if top * top > 14.0 or np.abs(c1 * s**2 + c2 * s**4).max() > 14.0:
            return False
        top = float(np.abs(c0 * s + c1 * s**3 + c2 * s**5).max()) * 1.01
        if not top < 9.0:
            return False
    return iters >= 1


def _ns_descs(stacks, iters):
    descs = (L.NsDesc * len(stacks))()
    for d, x in zip(descs, stacks):
        d.rows, d.cols, d.iters = x.shape[-2], x.shape[-1], iters
        d.batch = x.numel() // (d.rows * d.cols)
    return descs


def newton_schulz_native(stacks, outs, works, coeffs, iters, eps, status, stream):
    """One native call for the chains of several stacks of matrices (contiguous, 16-byte aligned): ``outs`` the results,
    ``works`` their workspaces (:func:`newton_schulz_group_buffers`).  Returns the number of launches."""
    descs = _ns_descs(stacks, iters)
    for d, x, out, work in zip(descs, stacks, outs, works):
        d.x, d.out = x.data_ptr(), out.data_ptr()
        d.eps = eps
        d.c0, d.c1, d.c2 = coeffs
        if work is not None:
            d.work, d.work_bytes = work.data_ptr(), work.numel()
    L.check(L.lib.pylo_b200_newton_schulz(descs, len(stacks), status.data_ptr() if status is not None else None, stream), "newton_schulz")
    return int(L.lib.pylo_b200_newton_schulz_launches(descs, len(stacks)))


def newton_schulz_buffers(x: torch.Tensor, iters: int):
    """(result, workspace or None) for one stack of :func:`newton_schulz_native` that is alone in its call."""
    return newton_schulz_group_buffers([x], iters)[0]


def newton_schulz_group_buffers(stacks, iters: int):
    """(result, workspace or None) for every stack of one call of :func:`newton_schulz_native`."""
    need = (C_.c_int64 * len(stacks))()
    L.check(L.lib.pylo_b200_newton_schulz_workspaces(_ns_descs(stacks, iters), len(stacks), need), "newton_schulz_workspaces")
    return [(torch.empty_like(x), torch.empty(n, dtype=torch.uint8, device=x.device) if n else None) for x, n in zip(stacks, need)]


def newton_schulz_tc(x: torch.Tensor, coeffs, iters: int = 5, eps: float = 1e-8, status=None, stream=None) -> torch.Tensor:
    """:func:`newton_schulz` on the tensor cores.

    Same chain as CELO2_naive.py:59-73.  Where the coefficients keep the iterates bounded (the usual ones do), the whole
    chain is one native call (``pylo_b200_newton_schulz``): every matrix is kept as two fp16 planes of one power-of-two
    scale, 22 significant bits, and every product is three tcgen05 products of planes accumulated in fp32.  Else each
    product is a launch of ``pylo_b200_gemm_tn_3xtf32`` on plain fp32 matrices, with x^T kept beside x, for the shapes it
    takes.  Not bit-identical to the fp32 products of ``torch.matmul`` (neither are two builds of cuBLAS); against an fp64
    evaluation both are as close as they are.
    """
    coeffs = tuple(float(v) for v in coeffs)
    if stream is None:
        stream = torch.cuda.current_stream().cuda_stream
    if newton_schulz_bounded(coeffs, iters):
        x = x.contiguous()
        if x.data_ptr() % 16:
            x = x.clone()
        out, work = newton_schulz_buffers(x, iters)
        newton_schulz_native([x], [out], [work], coeffs, iters, eps, status, stream)
        return out
    if not newton_schulz_eligible(*x.shape[-2:]):
        return newton_schulz(x, coeffs, iters, eps)
    shape = x.shape
    x = x.reshape((-1,) + tuple(shape[-2:]))
    tall = x.shape[-2] > x.shape[-1]
    if tall:
        x = x.transpose(-2, -1)
    x = (x / (torch.linalg.norm(x, dim=(-2, -1), keepdim=True) + eps)).contiguous()
    n_b, r, c = x.shape
    c0, c1, c2 = coeffs
    xt = torch.empty((n_b, c, r), dtype=torch.float32, device=x.device)
    a = torch.empty((n_b, r, r), dtype=torch.float32, device=x.device)
    b = torch.empty_like(a)
    x_next = torch.empty_like(x)
    for it in range(iters):
        _transpose(x, xt, stream)
        _gemm_tn(x, x, a, None, 1.0, 0.0, status, stream, symmetric=True)     # a = x x^T
        _gemm_tn(a, a, b, a, c2, c1, status, stream, symmetric=True)          # b = c1 a + c2 a a   (a is symmetric)
        _gemm_tn(b, xt, x_next, x, 1.0, c0, status, stream)                   # x = c0 x + b x
        x, x_next = x_next, x
    if tall:
        x = x.transpose(-2, -1)
    return x.reshape(shape)


def require_cuda_param(p: torch.Tensor, who: str):
    if not p.is_cuda:
        raise RuntimeError(f"{who}: parameters must live on a CUDA device (there is no CPU path)")
    if p.dtype != torch.float32:
        raise RuntimeError(f"{who}: only fp32 parameters are supported, got {p.dtype}")
    if not p.is_contiguous():
        raise RuntimeError(f"{who}: parameters must be contiguous")


def group_floats(group, *names):
    """The values of some of a param group's entries as floats, to be compared with the next step's.

    An entry may be a tensor that a scheduler changes in place: kept as it is, it would always equal itself."""
    return tuple([float(group[name]) for name in names])


def optimizer_step(step):
    """Decorator of an optimizer's ``step``: torch's own wrapper (profiler range, step hooks) and ``no_grad``, but only where
    something can see them.

    The wrapper costs as much as all launches of a small model's step.  The steps of this package run no differentiable
    operation on a parameter, so without hooks and without a profiler a plain call does the same."""
    watched = Optimizer.profile_hook_step(torch.no_grad()(step))
    module = sys.modules[Optimizer.__module__]
    hooks = [getattr(module, name, None) for name in ("_global_optimizer_pre_hooks", "_global_optimizer_post_hooks")]
    profiling = getattr(torch.autograd, "_profiler_enabled", None)

    @functools.wraps(step)
    def run(self, *args, **kwargs):
        own = self.__dict__
        if (profiling is None or profiling() or None in hooks or hooks[0] or hooks[1]
                or own.get("_optimizer_step_pre_hooks", True) or own.get("_optimizer_step_post_hooks", True)):
            return watched(self, *args, **kwargs)
        return step(self, *args, **kwargs)

    run.hooked = True   # tells the base class that the wrapper is there
    return run


class FlatWeights:
    """A small network's weights, one after the other: ``flat`` on the device, which descriptors point to, and on the host what
    launches carry as arguments.

    The host's values are read from ``flat`` here and nowhere else, again after every write to it that autograd's version counter
    sees (not one through ``.data`` or by a foreign kernel), so that a step does not mix old and new ones."""

    def __init__(self, parts, device):
        with torch.inference_mode(False):   # a tensor made in inference mode counts nothing
            self.flat = torch.cat([t.detach().reshape(-1) for t in parts]).to(device).contiguous()
        self._version = None
        self.host()   # now, not in the first step

    def host(self) -> int:
        """Address of the host's copy, good until the next call."""
        version = self.flat._version
        if version != self._version:
            self._values = self.flat.detach().cpu().numpy()
            self._address, self._version = self._values.ctypes.data, version
        return self._address


class StepCounters:
    """The ``step`` entries of some parameters' states, advanced together.

    The usual ones, 0-d fp64 tensors on the CPU, are counted up through their addresses in one native call (one torch
    operation per tensor was most of the host's time on a small model); anything else one by one."""

    def __init__(self, states):
        self.states = states
        self.tensors = [None] * len(states)
        self.first, self.equal = C_.c_double(), C_.c_int()

    def advance(self):
        """Add one to every counter; returns the old values: a float where they are all the same, else a list."""
        if not all([st["step"] is t for st, t in zip(self.states, self.tensors)]):
            self.tensors = [st["step"] for st in self.states]
            plain = all(torch.is_tensor(t) and t.device.type == "cpu" and t.dtype == torch.float64 and t.dim() == 0 for t in self.tensors)
            self.table = (C_.c_void_p * len(self.tensors))(*[t.data_ptr() for t in self.tensors]) if plain else None
        if self.table is not None:
            L.check(L.lib.pylo_b200_advance_steps(self.table, len(self.tensors), C_.byref(self.first), C_.byref(self.equal)), "advance_steps")
            if self.equal.value:
                return self.first.value
            return [float(t) - 1.0 for t in self.tensors]
        old = []
        for st in self.states:
            st["step"] += 1
            old.append(float(st["step"]) - 1.0)
        return old


class ItemPlan:
    """Tile list + item table for the simple element-wise kernels (AdamW, CELO2 tail)."""

    def __init__(self, dtype, sizes: Sequence[int], device, elems: int = L.TILE_ELEMS):
        self.items = np.zeros(len(sizes), dtype=dtype)
        self.items["n"] = sizes
        tiles, ranges = make_tiles(sizes, elems)
        if "tile0" in dtype.names:
            self.items["tile0"], self.items["n_tiles"] = [t0 for t0, _ in ranges], [k for _, k in ranges]
        self.ranges = ranges
        self.tiles = DeviceTable(tiles, device)
        self.n_tiles = len(tiles)
        self.table = DeviceTable(self.items, device)

    def upload(self):
        self.table.upload()
