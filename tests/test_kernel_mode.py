"""Convolution weights as matrices whose row vectors have an entry per position (PYLO_MODE_KERNEL): which tensors go that way, and
the step over them against the oracle and against the general path."""

import numpy as np
import pytest
import torch

import cases
from pylo_b200 import _lib as L
from pylo_b200 import plan

# positions 2, 4, 9, 25, 32; 64 columns and more, a block of 128 or 1024 with remainders; strips of 8 and 32 rows with remainders; row and
# column vectors in either role; a generic tensor, a matrix and a vector in between
SHAPES = [(40, 24, 3, 3), (8, 36, 2), (200, 20, 5, 5), (33, 36, 3, 3), (70, 36, 4, 8), (600, 128, 3, 3), (16, 520, 1, 2), (64, 3, 7, 7),
          (9, 40, 4), (96, 64), (513, 16, 2, 2), (13,)]


def _mode(shape, fdims, sliced=False, tensors=()):
    d = np.zeros(1, dtype=L.DESC_DTYPE)
    plan.fill_geometry(d[0], shape, fdims, 0, sliced, tensors)
    return int(d["mode"][0])


def test_which_tensors_are_taken_as_matrices_of_positions():
    assert _mode((40, 24, 3, 3), (1, 0)) == L.MODE_KERNEL and _mode((40, 24, 3, 3), (0, 1)) == L.MODE_KERNEL
    assert _mode((40, 24, 1, 1), (1, 0)) == L.MODE_FAST2D
    assert _mode((40, 16, 2, 2), (1, 0)) == L.MODE_KERNEL
    assert _mode((40, 15, 2, 2), (1, 0)) == L.MODE_GENERIC          # 60 columns
    assert _mode((40, 25, 3, 3), (1, 0)) == L.MODE_GENERIC          # 225 columns: rows are not aligned
    assert _mode((40, 24, 33), (1, 0)) == L.MODE_GENERIC            # 33 positions
    assert _mode((40, 24, 4, 8), (1, 0)) == L.MODE_KERNEL
    assert _mode((2, 40, 24, 4), (2, 1)) == L.MODE_GENERIC          # an axis before
    assert _mode((64, 3, 7, 7), (3, 0)) == L.MODE_GENERIC           # axes between
    assert _mode((40, 24, 3, 3), (1, 0), sliced=True) == L.MODE_GENERIC
    storage = torch.zeros(40 * 24 * 9 + 1)
    assert _mode((40, 24, 3, 3), (1, 0), tensors=(storage[1:],)) == L.MODE_GENERIC


def test_the_tensor_core_sweep_covers_every_element_of_them_once():
    kernel, fast, slow = [(0, 40, 216), (2, 600, 1152)], [(1, 96, 64)], [(3, 13)]
    items = plan.apply_items(L.FAM_ADAFAC, True, fast, slow, kernel=kernel)
    seen = {u: np.zeros((X, -(-Y // 128)), dtype=int) for u, X, Y in kernel + fast}
    for t, strip, cb, tag in items.tolist():
        if tag < L.TC_GEN_ITEM:
            seen[t][strip * tag:(strip + 1) * tag, cb] += 1
    assert all((a == 1).all() for a in seen.values())
    assert items["tensor"].tolist().index(1) > max(i for i, t in enumerate(items["tensor"].tolist()) if t != 1)   # FAST2D items last


@pytest.mark.gpu
@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"mlp_precision": "fp32"}), ("elo", {}), ("velo", {})])
def test_the_step_matches_the_oracle_and_the_general_path(family, extra, monkeypatch):
    import cuda_util as CU
    from oracle import pylo_oracle as O
    from test_gpu_properties import _make, _nets, _step

    case = dict(shapes=SHAPES, init_seed=71, init_scale=0.1, grad_seed=72, grad_scale=0.3)
    init = [v.clone() for v in cases.init_values(case)]
    general = plan.fill_geometry

    def without(d, *args, **kw):
        out = general(d, *args, **kw)
        d["mode"] = L.MODE_GENERIC if d["mode"] == L.MODE_KERNEL else d["mode"]
        return out

    outs = []
    for route in (general, without):
        monkeypatch.setattr(plan, "fill_geometry", route)
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **extra)
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            _step(opt, family, t)
        outs.append([p.detach().cpu() for p in params])
    ref = [v.clone() for v in init]
    if family == "velo":
        rnn, mlp = _nets(family)
        ora = O.VeLOOracle(O.rnn_weights_from_module(rnn), O.bank_from_module(mlp), SHAPES, lr=1.0, num_steps=100)
    elif family == "elo":
        ora = O.AdafacLOOracle(_nets(family).flat_weights(), lr=1e-2, elo=True, weight_decay=0.1, clip_grad=True)
    else:
        ora = O.AdafacLOOracle(_nets(family).flat_weights(), lr=1e-2)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        ora.step(ref, grads, cases.velo_loss(t)) if family == "velo" else ora.step(ref, grads)
    for out in outs:
        res = CU.compare({2: out}, {2: ref}, init)
        assert res[2][0] < 1e-5 and res[2][1] < 2e-5, res
