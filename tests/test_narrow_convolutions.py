"""Convolution weights whose rows fill little of a block of 128 columns: the tensor-core sweep takes them the general way."""

import numpy as np
import pytest
import torch

import cases
from pylo_b200 import _lib as L
from pylo_b200 import plan


@pytest.mark.parametrize("shape,columns,matrix", [((512, 16, 2, 2), 64, False), ((456, 8, 3, 3), 72, False), ((455, 8, 3, 3), 72, True),
                                                  ((512, 12, 3, 3), 108, True), ((512, 16, 3, 3), 144, False), ((64, 16, 3, 3), 144, True),
                                                  ((512, 20, 3, 3), 180, True), ((512, 32, 2, 2), 128, True), ((512, 33, 2, 2), 132, False),
                                                  ((512, 65, 2, 2), 260, True), ((512, 19, 3, 3), 171, False)])
def test_rows_that_fill_two_thirds_of_their_blocks(shape, columns, matrix):
    d = np.zeros(1, dtype=L.DESC_DTYPE)
    plan.fill_geometry(d[0], shape, (1, 0), 0, full=plan.KERNEL_FULL)
    assert (int(d["mode"][0]) == L.MODE_KERNEL) == (matrix and columns % 4 == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("family,extra,mode", [("adafaclo", {}, L.MODE_GENERIC), ("adafaclo", {"mlp_precision": "fp32"}, L.MODE_KERNEL), ("velo", {}, L.MODE_KERNEL)])
def test_the_step_matches_the_oracle(family, extra, mode):
    import cuda_util as CU
    from oracle import pylo_oracle as O
    from test_gpu_properties import _make, _nets, _step

    shapes = [(270, 16, 3, 3), (457, 8, 3, 3), (70, 32, 3, 3), (40,)]
    case = dict(shapes=shapes, init_seed=91, init_scale=0.1, grad_seed=92, grad_scale=0.3)
    init = [v.clone() for v in cases.init_values(case)]
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    opt = _make(family, params, **extra)
    ref = [v.clone() for v in init]
    if family == "velo":
        rnn, mlp = _nets(family)
        ora = O.VeLOOracle(O.rnn_weights_from_module(rnn), O.bank_from_module(mlp), shapes, lr=1.0, num_steps=100)
    else:
        ora = O.AdafacLOOracle(_nets(family).flat_weights(), lr=1e-2)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        _step(opt, family, t)
        ora.step(ref, grads, cases.velo_loss(t)) if family == "velo" else ora.step(ref, grads)
    made = opt._plan[1]["plan"] if family == "velo" else next(iter(opt._plans.values()))[1]
    assert made.tdesc.host["mode"].tolist() == [mode, mode, L.MODE_KERNEL, L.MODE_VEC1D]
    res = CU.compare({2: [p.detach().cpu() for p in params]}, {2: ref}, init)
    assert res[2][0] < 1e-5 and res[2][1] < 2e-5, res
