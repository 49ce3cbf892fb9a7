"""Large models with a few convolution weights: which launches their sums take, and the steps over them."""

import pytest
import torch

import cases
from pylo_b200 import _lib as L
from pylo_b200 import plan

CONV = [(160, 128, 3), (40, 24, 3, 3), (64, 3, 7, 7)]


def _run(shapes, family, steps=2, **kw):
    from test_gpu_properties import _make, _step

    case = dict(shapes=shapes, init_seed=81, init_scale=0.1, grad_seed=82, grad_scale=0.3)
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    opt = _make(family, params, **kw)
    for t in range(1, steps + 1):
        for p, g in zip(params, cases.grads_at(case, t)):
            p.grad = g.cuda()
        _step(opt, family, t)
    return opt, [p.detach().clone() for p in params]


def _plan_of(opt):
    return opt._plan[1]["plan"] if hasattr(opt, "_plan") else next(iter(opt._plans.values()))[1]


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["adafaclo", "velo"])
def test_large_models_keep_the_lean_sums(family):
    """The variant that takes convolution weights along has fewer CTAs per SM: a large model's matrices have a launch of their own, and
    the same sums (the AdafacLO family's tensors do not depend on one another)."""
    matrices = [(512, 1024)] * 47   # 3008 items
    opt, out = _run(matrices + CONV, family, 1)
    pl = _plan_of(opt)
    n_fast = pl.n_atiles - pl.n_ragged - pl.step_plan.n_kernel
    assert pl.step_plan.n_kernel > 0 and n_fast > L.ROWCOL_KERNEL_APART
    assert {name: n for _, name, n in pl._phases()}["rowcol_sums"] == 2
    few, _ = _run([(512, 1024)] + CONV, family, 1)
    assert {name: n for _, name, n in _plan_of(few)._phases()}["rowcol_sums"] == 1
    if family == "adafaclo":
        _, alone = _run(matrices, family, 1)
        assert all(torch.equal(a, b) for a, b in zip(out, alone))


@pytest.mark.gpu
@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"mlp_precision": "fp32"}), ("velo", {})])
def test_many_tensors_and_the_ring_match_the_oracle(family, extra, monkeypatch):
    """More tensors than the factor phase gives an SM each, column vectors of more than 1024, general means, and positions in a model whose
    state sweep goes through the ring."""
    from oracle import pylo_oracle as O
    import cuda_util as CU
    from test_gpu_properties import _nets

    shapes = [(24, 128, 3, 3), (16, 1100), (513, 64), (33, 36, 3, 3), (13,)] * 5 + [(300, 4100)]
    case = dict(shapes=shapes, init_seed=81, init_scale=0.1, grad_seed=82, grad_scale=0.3)
    init = [v.clone() for v in cases.init_values(case)]
    outs = []
    for ring in (False, True):
        if ring:   # nearly all elements do not have to be FAST2D here
            order = plan.sum_order
            monkeypatch.setattr(plan, "sum_order", lambda *a: order(*a)._replace(bulk_copies=True))
        opt, out = _run(shapes, family, **extra)
        assert _plan_of(opt).bulk_copies == int(ring) and _plan_of(opt).step_plan.n_kernel > 0
        outs.append([p.cpu() for p in out])
    ref = [v.clone() for v in init]
    if family == "velo":
        rnn, mlp = _nets(family)
        ora = O.VeLOOracle(O.rnn_weights_from_module(rnn), O.bank_from_module(mlp), shapes, lr=1.0, num_steps=100)
    else:
        ora = O.AdafacLOOracle(_nets(family).flat_weights(), lr=1e-2)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        ora.step(ref, grads, cases.velo_loss(t)) if family == "velo" else ora.step(ref, grads)
    for out in outs:
        res = CU.compare({2: out}, {2: ref}, init)
        assert res[2][0] < 1e-5 and res[2][1] < 2e-5, res
