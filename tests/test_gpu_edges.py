"""GPU checks at the sizes where the work lists, the generic paths and the Newton-Schulz chain can go wrong: edges of tiles,
remainders, the smallest and the largest of a range; against the CPU oracle or an fp64 evaluation."""

import copy

import pytest
import torch

import cases
import cuda_util as CU
from pylo_b200 import _lib as pylo_lib
from test_gpu_properties import _make, _nets, _step

pytestmark = pytest.mark.gpu

COEFFS = (3.4445, -4.7750, 2.0315)

# inner axes after the factored ones (1 < I <= 32, I > 32), before and between them, rows that are longer than a warp takes
# (4096 on, unaligned), short blocks (Y*I = 4), strips of 8, 16 and 32 rows with remainders, a partial table item
SHAPES = {
    "inner": [(40, 24, 3, 3), (9, 50, 5), (64, 70, 40), (33, 35, 33)],
    "outer": [(3, 40, 5, 24), (2, 3, 37, 41), (30, 3, 4, 4)],
    "long": [(3, 4099), (5, 8193), (600, 7), (1100, 3)],
    "rows": [(513, 64), (512, 68), (9, 1028), (65, 2052), (2049, 36)],
}


def _oracle(family, net, shapes):
    from oracle import pylo_oracle as O

    if family == "adafaclo":
        return O.AdafacLOOracle(net.flat_weights(), lr=1e-2)
    if family == "celo2":
        return O.CELO2Oracle(net.flat_weights(), lr=1e-2, weight_decay=0.1, clip_grad=True, orthogonalize=False)
    rnn, mlp = net
    return O.VeLOOracle(O.rnn_weights_from_module(rnn), O.bank_from_module(mlp), shapes, lr=1.0, num_steps=100)


@pytest.mark.parametrize("which", sorted(SHAPES))
@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"mlp_precision": "fp32"}), ("celo2", {"orthogonalize": False}),
                                          ("velo", {})])
def test_shapes_at_the_edges_match_the_oracle(family, extra, which):
    shapes = SHAPES[which] + [(13,)]
    case = dict(shapes=shapes, init_seed=51, init_scale=0.1, grad_seed=52, grad_scale=0.3)
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    init = [v.clone() for v in cases.init_values(case)]
    ref = [v.clone() for v in init]
    opt, ora = _make(family, params, **extra), _oracle(family, _nets(family), shapes)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        _step(opt, family, t)
        ora.step(ref, grads, cases.velo_loss(t)) if family == "velo" else ora.step(ref, grads)
    res = CU.compare({2: [p.detach().cpu() for p in params]}, {2: ref}, init)
    assert res[2][0] < 1e-5 and res[2][1] < 2e-5, res


@pytest.mark.parametrize("family", ["adafaclo", "celo2", "velo"])
def test_state_sweep_through_the_ring(family, monkeypatch):
    """Large models' state sweep on small ones: tiles shorter than a stage, partial stages, tiles of other kinds in between."""
    shapes = [(513, 64), (7,), (9, 1028), (3, 4), (600, 1040), (65, 7), (300, 4100)]
    runs = []
    for least in (pylo_lib.BULK_COPY_ELEMS, 1):
        monkeypatch.setattr(pylo_lib, "BULK_COPY_ELEMS", least)
        case = dict(shapes=shapes, init_seed=61, init_scale=0.1, grad_seed=62, grad_scale=0.3)
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **({"orthogonalize": False} if family == "celo2" else {}))
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            _step(opt, family, t)
        runs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


# matrices of the shared-memory kernel, of the 128- and 256-wide tiles and of tiles on pairs of SMs, with K tails and odd
# pitches, wide and tall
STACKS = [[(1, 5)], [(64, 64), (3, 16, 16), (10, 128)], [(65, 67), (67, 65), (2, 129, 257)], [(128, 128), (7, 3001), (3001, 7), (100, 260)],
          [(70, 1030), (1020, 70)], [(2, 130, 2111), (40, 90)], [(65, 4100)],   # contractions in two, four and eight parts
          [(2, 1300, 1290), (1290, 2050)], [(1024, 1030), (258, 1024), (2, 200, 392), (33, 1000), (1000, 33), (5, 5), (96, 96), (300, 300), (131, 70), (70, 131)]]


@pytest.mark.parametrize("shapes", STACKS, ids=[str(len(s)) + "x" + str(s[0]) for s in STACKS])
def test_newton_schulz_chains_side_by_side(shapes):
    """Several stacks in one call (also more than one launch takes): every result against fp64."""
    from pylo_b200.optim import _common as K

    gen = torch.Generator(device="cuda").manual_seed(7)
    xs = [torch.randn(s, device="cuda", generator=gen) for s in shapes]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    bufs = [K.newton_schulz_buffers(x, 5) for x in xs]
    stream = torch.cuda.current_stream().cuda_stream
    K.newton_schulz_native(xs, [o for o, _ in bufs], [w for _, w in bufs], COEFFS, 5, 1e-8, status, stream)
    for x, (out, _) in zip(xs, bufs):
        exact = K.newton_schulz(x.double(), COEFFS)
        e32 = float((K.newton_schulz(x, COEFFS).double() - exact).norm() / exact.norm())
        err = float((out.double() - exact).norm() / exact.norm())
        assert err < max(4 * e32, 1e-5), (tuple(x.shape), err, e32)
    assert int(status.item()) == 0


def test_newton_schulz_with_unbounded_coefficients_leaves_the_fp16_planes():
    from pylo_b200.optim import _common as K

    assert K.newton_schulz_bounded(COEFFS, 5) and not K.newton_schulz_bounded((9.0, -2.0, 1.0), 5)
    x = torch.randn(128, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    coeffs = (4.0, -3.0, 1.0)
    assert not K.newton_schulz_bounded(coeffs, 2)
    exact = K.newton_schulz(x.double(), coeffs, 2)
    cubic = K.newton_schulz(x.double(), (1.5, -0.5, 0.0), 3)   # no quintic term: one product less per round
    assert float((K.newton_schulz_tc(x, (1.5, -0.5, 0.0), 3).double() - cubic).norm() / cubic.norm()) < 1e-5
    assert float((K.newton_schulz_tc(x, coeffs, 2).double() - exact).norm() / exact.norm()) < 1e-5


@pytest.mark.parametrize("T", [1, 8, 9])
def test_velo_gates_at_group_edges(T):
    """One tensor, exactly one group of eight, one more than a group; 512 hidden units (weight rows in registers)."""
    from oracle import pylo_oracle as O
    from pylo_b200 import models, optim

    shapes = [(12 + i, 8) for i in range(T)]
    torch.manual_seed(0)
    rnn, mlp = models.VeLORNN(), models.VeLOMLP()
    with torch.no_grad():
        for name, p in mlp.named_parameters():
            if name.endswith("_") or "_." in name:
                p.mul_(0.05)
    ora = O.VeLOOracle(O.rnn_weights_from_module(rnn), O.bank_from_module(mlp), shapes, lr=1.0, num_steps=100)
    case = dict(shapes=shapes, init_seed=61, init_scale=0.1, grad_seed=62, grad_scale=0.3)
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    ref = [v.clone() for v in cases.init_values(case)]
    opt = optim.VeLO_CUDA(params, lr=1.0, num_steps=100, rnn=rnn, mlp=mlp)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        # a loss on the device, then a host number
        opt.step(torch.tensor(cases.velo_loss(t), device="cuda") if t == 1 else cases.velo_loss(t))
        ora.step(ref, grads, cases.velo_loss(t))
    e = float((opt.lstm_hidden_state[0].cpu() - ora.lstm_hidden_state[0]).abs().max())
    assert e < 1e-5, e
    res = CU.compare({2: [p.detach().cpu() for p in params]}, {2: ref}, cases.init_values(case))
    assert res[2][0] < 1e-5, res


def test_steps_that_changed_hands():
    """Step counters that differ between tensors, that are replaced, and gradients that move or are not contiguous."""
    shapes = [(40, 24), (24, 40), (24,)]
    runs = []
    for variant in (0, 1):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(dict(shapes=shapes, init_seed=71))]
        opt = _make("adafaclo", params)
        for t in (1, 2, 3, 4):
            grads = [g.cuda() for g in cases.grads_at(dict(grad_seed=72, grad_scale=0.3, shapes=shapes), t)]
            for k, (p, g) in enumerate(zip(params, grads)):
                if t == 2 and k == 1:
                    p.grad = None                      # this tensor falls a step behind
                elif variant and p.dim() == 2:
                    p.grad = g.t().contiguous().t()    # the same values with other strides
                else:
                    p.grad = g
            if t == 4 and variant:
                for p in params:                       # the same count in another tensor, as a loaded checkpoint has it
                    opt.state[p]["step"] = opt.state[p]["step"].clone()
            opt.step()
        assert [float(opt.state[p]["step"]) for p in params] == [4.0, 3.0, 4.0]
        runs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("cls", ["celo2", "elo_celo2"])
def test_adamw_tensors_of_any_length(cls):
    """Whole pieces of four, tails, and a length that keeps the three shared momenta unaligned."""
    from oracle import pylo_oracle as O

    shapes = [(4096,), (5,), (1027,), (1,), (2050,)]
    case = dict(shapes=shapes, init_seed=81, init_scale=0.1, grad_seed=82, grad_scale=0.3)
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    ref = [v.clone() for v in cases.init_values(case)]
    opt = _make(cls, params)
    kw = dict(weight_decay=0.1, clip_grad=True) if cls == "celo2" else dict(weight_decay=0.1, clip_grad=True, adam_lr_mult=20.0)
    ora = O.CELO2Oracle(_nets(cls).flat_weights(), lr=1e-2, shared_adam=(cls == "elo_celo2"), **kw)
    for t in (1, 2, 3):
        grads = cases.grads_at(case, t)
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        ora.step(ref, grads)
    res = CU.compare({3: [p.detach().cpu() for p in params]}, {3: ref}, cases.init_values(case))
    assert res[3][0] < 1e-5 and res[3][1] < 2e-5, res


@pytest.mark.parametrize("family", ["adafaclo", "elo", "celo2", "elo_celo2", "velo"])
def test_gradients_of_another_type_are_converted(family):
    """bf16 gradients of fp32 parameters (``grad_dtype``), through every path of a step (the norm, the sweeps, AdamW), give
    what the same values in fp32 give: also where a bf16 gradient comes to lie at an address that held an fp32 one."""
    shapes = [(40, 24), (24,), (300, 260), (1027,)]
    runs = []
    for half in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(dict(shapes=shapes, init_seed=91, init_scale=0.1))]
        pool = [torch.zeros(p.shape, device="cuda") for p in params]
        opt = _make(family, params)
        for t in (1, 2, 3):
            for k, (p, g) in enumerate(zip(params, cases.grads_at(dict(grad_seed=92, grad_scale=0.3, shapes=shapes), t))):
                g = g.cuda().to(torch.bfloat16)
                if half and t > 1 and k != 0:
                    p.grad_dtype = torch.bfloat16
                    p.grad = pool[k].view(-1).view(torch.bfloat16)[:p.numel()].view(p.shape).copy_(g)
                else:
                    p.grad = pool[k].copy_(g)
            _step(opt, family, t)
            for p in params:
                p.grad = None
        runs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("family", ["adafaclo", "elo", "celo2", "elo_celo2", "velo"])
def test_a_scheduled_tensor_learning_rate_is_followed(family):
    """A tensor learning rate that a scheduler changes in place gives what the same float learning rates give."""
    shapes = [(40, 24), (24,)]
    runs = []
    for tensor_lr in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(dict(shapes=shapes, init_seed=95, init_scale=0.1))]
        opt = _make(family, params)
        if tensor_lr:
            for group in opt.param_groups:
                group["lr"] = torch.tensor(0.5)
        for t in (1, 2, 3):
            for p, g in zip(params, cases.grads_at(dict(grad_seed=96, grad_scale=0.3, shapes=shapes), t)):
                p.grad = g.cuda()
            for group in opt.param_groups:
                if tensor_lr:
                    group["lr"].fill_(0.5 ** t)
                else:
                    group["lr"] = 0.5 ** t
            _step(opt, family, t)
        runs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


def _plans(opt):
    if getattr(opt, "_plan", None):
        return [opt._plan[1]["plan"]]
    return [v[1]["lo"] if isinstance(v[1], dict) else v[1] for v in opt._plans.values()]


@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"mlp_precision": "fp32"}), ("elo", {}), ("celo2", {}),
                                          ("elo_celo2", {}), ("velo", {})])
def test_a_reported_wait_keeps_the_parameters(family, extra):
    """The status word is set from the host (no wait runs out here): every kernel that writes parameters, on matrices of both
    kinds, must leave them, VeLO's LSTM must keep its state, and check_status() and the next step must say so."""
    shapes = [(40, 24), (33, 7)]
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(dict(shapes=shapes, init_seed=97, init_scale=0.1))]
    opt = _make(family, params, **extra)
    for p, g in zip(params, cases.grads_at(dict(grad_seed=98, grad_scale=0.3, shapes=shapes), 1)):
        p.grad = g.cuda()
    _step(opt, family, 1)
    opt.check_status()
    plan, = _plans(opt)
    plan.status[0] = 4 if "celo2" in family else 8
    with pytest.raises(pylo_lib.PyloLibError):
        opt.check_status()

    def kept():
        lstm = [*opt.lstm_hidden_state, *opt.loss_buffer.values()] if family == "velo" else []
        return [t.detach().clone() for t in params + lstm]

    before = kept()
    _step(opt, family, 2)      # its launches find the word set and pass it on to the host
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(before, kept()))
    with pytest.raises(pylo_lib.PyloLibError):
        _step(opt, family, 3)
    opt.clear_status()
    _step(opt, family, 4)
    opt.check_status()
    assert not any(torch.equal(a, p) for a, p in zip(before, params)), "a cleared optimizer goes on"


@pytest.mark.parametrize("family", ["adafaclo", "elo", "celo2", "elo_celo2", "velo"])
def test_a_refused_step_has_advanced_nothing(family):
    """A reported timeout of the second param group: the first group, the step counters, the gradients and the state stay."""
    shapes = [(40, 24), (33, 20)]
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(dict(shapes=shapes, init_seed=97, init_scale=0.1))]
    opt = _make(family, [{"params": [p]} for p in params])
    if family == "adafaclo":
        for group in opt.param_groups:
            group["max_grad_norm"] = 1e-3   # scales the gradients in place
    grads = [g.cuda() for g in cases.grads_at(dict(grad_seed=98, grad_scale=0.3, shapes=shapes), 1)]
    for p, g in zip(params, grads):
        p.grad = g
    _step(opt, family, 1)
    torch.cuda.synchronize()
    for g in grads:
        g.mul_(1e6)

    def everything():
        out = [t.clone() for t in grads] + [p.detach().clone() for p in params]
        for p in params:
            out += [v.clone() if torch.is_tensor(v) else torch.tensor(float(v)) for v in opt.state[p].values()]
        return out + [torch.tensor(float(g.get("step", 0))) for g in opt.param_groups]

    before = everything()
    _plans(opt)[-1]._status_view[0] = 8
    with pytest.raises(pylo_lib.PyloLibError):
        _step(opt, family, 2)
    torch.cuda.synchronize()
    after = everything()
    assert len(before) == len(after) and all(torch.equal(a, b) for a, b in zip(before, after))


@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"mlp_precision": "fp32"}), ("celo2", {"orthogonalize": False}),
                                          ("velo", {})])
@pytest.mark.parametrize("shapes", [[(40, 24), (33, 7)], [(2048, 1024), (33, 7)]], ids=["small", "many_tiles"])
def test_timed_phases_are_the_step_that_users_get(family, extra, shapes):
    """Timed phase by phase, a step launches what it launches otherwise (counted, and by its result bit for bit)."""
    case = dict(shapes=shapes, init_seed=97, init_scale=0.1, grad_seed=98, grad_scale=0.3)
    runs = []
    for timed in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **extra)
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            _step(opt, family, t)
            plan, = _plans(opt)
            if t == 1:
                plan.enable_profile(timed)
                plan.launch_count = 0
        torch.cuda.synchronize()
        runs.append(([p.detach().clone() for p in params], plan.launch_count))
    assert all(torch.equal(a, b) for a, b in zip(runs[0][0], runs[1][0])) and runs[0][1] == runs[1][1]
    times = plan.phase_times()
    assert ("finalize_moments" in times) == (not plan.sum_tiles) and plan.apply_kernel in times
    assert all(len(v) == 1 and v[0] > 0 for v in times.values())


def test_a_launch_without_factored_matrices_is_not_reported_as_the_main_kernel():
    """The benchmark sets the main kernel's mean time against its bytes: a bias' own launch is not one of them."""
    params = [torch.nn.Parameter(torch.randn(33, device="cuda"))]
    opt = _make("adafaclo", params)
    params[0].grad = torch.ones(33, device="cuda")
    opt.step()
    plan, = _plans(opt)
    plan.enable_profile()
    opt.step()
    torch.cuda.synchronize()
    assert plan.apply_kernel not in plan.phase_times() and "k_apply_adafac_tc<true>" in plan.phase_times()


@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("celo2", {"orthogonalize": False})])
@pytest.mark.parametrize("rows", [8 * 192, 8 * 192 + 8])
def test_tile_sums_on_both_sides_of_the_launch(family, extra, rows):
    """The most tiles that phase P adds up itself, and one more: the step with the other way of adding them."""
    case = dict(shapes=[(rows, 128)], init_seed=97, init_scale=0.1, grad_seed=98, grad_scale=0.3)
    runs = []
    for flip in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **extra)
        for t in (1, 2, 3):
            params[0].grad = cases.grads_at(case, t)[0].cuda()
            _step(opt, family, t)
            plan, = _plans(opt)
            if t == 1:
                assert plan.sum_tiles == (rows == 8 * 192) and plan.n_tiles == rows // 8
                if flip:
                    plan.step_plan.sum_tiles = int(not plan.sum_tiles)
        runs.append(params[0].detach().clone())
    # the partials are added up in fp64 on both ways and rounded once: they differ by the last bit of a sum at most, which
    # moves a normalised feature by 2^-24 of itself and the network's output, and so the step, by a few times that
    move = float((runs[0] - cases.init_values(case)[0].cuda()).abs().max())
    assert float((runs[0] - runs[1]).abs().max()) <= 1e-5 * move + 2 ** -23 * float(runs[0].abs().max())


# matrices and vectors of a small model: rows fewer than CTAs, one CTA's share full, odd sizes (no piece of 16 bytes), one row, one
# column, a single element; 1, 2, 8 and 16 CTAs a tensor
SMALL = [[(128, 784), (128,), (10, 128), (10,)], [(1, 4744), (3, 4), (1, 1)], [(5000, 1), (7, 1001), (1001, 7), (4099,)], [(512, 256)],
         [(64, 64)] * 40 + [(13,)] * 30, [(9, 20), (33, 7)] * 30]


@pytest.mark.parametrize("shapes", SMALL, ids=[str(s[0]) + "x" + str(len(s)) for s in SMALL])
@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("adafaclo", {"initial_momentum_decays": (0.2, 0.9, 0.99)}), ("elo", {}),
                                          ("celo2", {"orthogonalize": False}), ("velo", {})])
def test_small_models_front_in_one_launch(family, extra, shapes, monkeypatch):
    """Sums, factors and state of a small model by clusters, against the three launches that other models take."""
    from pylo_b200 import plan as pylo_plan

    case = dict(shapes=shapes, init_seed=51, init_scale=0.1, grad_seed=52, grad_scale=0.3)
    runs = []
    for ctas in (pylo_plan.SMALL_CTAS, 0):
        monkeypatch.setattr(pylo_plan, "SMALL_CTAS", ctas)
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **extra)
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            _step(opt, family, t)
        plan, = _plans(opt)
        assert bool(plan.small) == bool(ctas)
        runs.append(([p.detach().clone() for p in params], [opt.state[p] for p in params]))
    for (a, b, init) in zip(runs[0][0], runs[1][0], cases.init_values(case)):
        # sums of positive terms in another order: relative differences of a few 2^-24 (a thousand terms, in trees), which move
        # a factor by half of that and the network's output by a few times as much
        move = float((b - init.cuda()).abs().max())
        assert float((a - b).abs().max()) <= 2e-5 * move + 2 ** -23 * float(b.abs().max())
    for sa, sb in zip(runs[0][1], runs[1][1]):
        for key, x in sa.items():
            if torch.is_tensor(x) and x.is_floating_point() and x.numel():
                assert torch.allclose(x, sb[key], rtol=4e-6, atol=1e-12), key


@pytest.mark.parametrize("shapes,launches", [([(40, 24), (24,)], 1), ([(65, 77), (7,), (1,)], 1), ([(1001, 1028), (65, 77), (16385,), (3, 3, 5, 5)], 2),
                                             ([(3000, 2048), (2048,)], 1), ([(64, 64)], 1), ([(13,), (4099,)], 1)],
                         ids=["aligned", "ragged", "both", "many items", "matrices only", "vectors only"])
def test_velo_units_of_both_sweeps_in_one_launch(shapes, launches):
    """VeLO's packed items and the other units' tiles by one launch, against a launch for each: the same numbers."""
    from pylo_b200 import _lib as L

    case = dict(shapes=shapes, init_seed=53, init_scale=0.1, grad_seed=54, grad_scale=0.3)
    runs = []
    for apart in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make("velo", params)
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            if t == 2:
                plan, = _plans(opt)
                assert sum(n for ph, _, n in plan._phases() if ph & (L.STEP_APPLY | L.STEP_APPLY_REST)) == launches
                if apart:   # neither phase alone has both kinds
                    whole = plan._phases

                    def phases():
                        kept = [ph for ph in whole() if not ph[0] & (L.STEP_APPLY | L.STEP_APPLY_REST)]
                        return kept + [(L.STEP_APPLY, "items", 1), (L.STEP_APPLY_REST, "tiles", 1)]
                    plan._phases = phases
                    plan.enable_profile()
            _step(opt, "velo", t)
        torch.cuda.synchronize()
        runs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    assert all(float((a - v.cuda()).abs().max()) > 0 for a, v in zip(runs[0], cases.init_values(case)) if v.numel() > 1)


@pytest.mark.parametrize("shapes", [[(40, 24), (33, 28)], [(300, 1028), (7, 4)]], ids=["small", "blocks"])
@pytest.mark.parametrize("family,extra", [("celo2", {"orthogonalize": False}), ("adafaclo", {})])
def test_network_as_an_argument_is_the_folded_one(family, extra, shapes):
    """CELO2's packed sweep with the network as constants (features normalised) and with every unit's folded one (weights
    normalised): a product is rounded once more or less, 2^-24 of each of 30 terms.  AdafacLO's output layer as constants: the
    same numbers."""
    case = dict(shapes=shapes, init_seed=51, init_scale=0.1, grad_seed=52, grad_scale=0.3)
    runs = []
    for arg in (True, False):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make(family, params, **extra)
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            if not arg and t == 2:
                opt._prm.w_host = None
            opt.step()
        runs.append([p.detach().clone() for p in params])
    for a, b, init in zip(runs[0], runs[1], cases.init_values(case)):
        if family == "adafaclo":
            assert torch.equal(a, b)
        assert float((a - b).abs().max()) <= 1e-5 * float((b - init.cuda()).abs().max()) + 2 ** -23 * float(b.abs().max())


# rows that are not aligned: from the first width that goes with the others (64 columns) on, one and several blocks of 1024 columns,
# strips of 8 and 32 rows with remainders, a tile's last columns missing; narrower ones and aligned ones beside them
UNALIGNED = [(65, 65), (9, 1025), (33, 2051), (600, 67), (70, 63), (1, 101), (40, 24), (13,)]


@pytest.mark.parametrize("family,extra", [("adafaclo", {}), ("celo2", {"orthogonalize": False}), ("velo", {})])
def test_unaligned_rows_go_the_way_of_the_aligned_ones(family, extra, monkeypatch):
    """Sums and apply sweep of unaligned matrices against the oracle (small models' single launch off), and their work lists."""
    from pylo_b200 import plan as pylo_plan

    monkeypatch.setattr(pylo_plan, "SMALL_CTAS", 0)
    case = dict(shapes=UNALIGNED, init_seed=51, init_scale=0.1, grad_seed=52, grad_scale=0.3)
    params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
    init = [v.clone() for v in cases.init_values(case)]
    ref = [v.clone() for v in init]
    opt, ora = _make(family, params, **extra), _oracle(family, _nets(family), UNALIGNED)
    for t in (1, 2):
        grads = cases.grads_at(case, t)
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        _step(opt, family, t)
        ora.step(ref, grads, cases.velo_loss(t)) if family == "velo" else ora.step(ref, grads)
    res = CU.compare({2: [p.detach().cpu() for p in params]}, {2: ref}, init)
    assert res[2][0] < 1e-5 and res[2][1] < 2e-5, res
    plan, = _plans(opt)
    taken = {int(t) for t in plan.atiles.host["tensor"][:plan.n_ragged]}
    assert taken == {0, 1, 2, 3, 5} and len({int(u) for u in plan.rtiles.host["tensor"]}) == (0 if family == "adafaclo" else 5)


def test_squares_of_the_raw_steps_from_the_apply_sweep():
    """CELO2 without orthogonalisation: the apply sweep's sums of squares against the launch that reads the steps again, tiles and
    rows with remainders, several items a matrix; and a group that changes its mind between steps."""
    shapes = [(40, 24), (300, 1028), (1031, 68), (5, 4)]
    case = dict(shapes=shapes, init_seed=51, init_scale=0.1, grad_seed=52, grad_scale=0.3)
    runs = []
    for own in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make("celo2", params, orthogonalize=False)
        for t in (1, 2, 3, 4):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            opt.param_groups[0]["orthogonalize"] = t == 3
            opt.step()
            plan = opt._plans[0][1]
            if t == 1:
                assert plan["squares"] is not None
                if own:
                    it = plan["post"].items
                    it["part"][:], it["n_tiles"][:] = plan["squares"][3:5]
                    plan["squares"] = plan["post_key"] = None
        runs.append([p.detach().clone() for p in params])
    for a, b, init in zip(runs[0], runs[1], cases.init_values(case)):
        # the same terms in another order: each sum to a few 2^-24 of itself, half of that in its root
        assert float((a - b).abs().max()) <= 1e-5 * float((b - init.cuda()).abs().max()) + 2 ** -23 * float(b.abs().max())


def test_orthogonalised_groups_build_no_tables_of_squares():
    """They are made at the first step without orthogonalisation, with the results of the launch that reads the steps again."""
    case = dict(shapes=[(40, 24), (300, 1028), (5, 4)], init_seed=53, init_scale=0.1, grad_seed=54, grad_scale=0.3)
    runs = []
    for own in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = _make("celo2", params, orthogonalize=True)
        for t in (1, 2, 3, 4):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            opt.param_groups[0]["orthogonalize"] = t % 2 == 1
            opt.step()
            plan = opt._plans[0][1]
            if t == 1:
                assert plan.get("squares") is None
                if own:
                    plan["squares"] = None
        assert own or plan["squares"] is not None
        runs.append([p.detach().clone() for p in params])
    for a, b, init in zip(runs[0], runs[1], cases.init_values(case)):
        # the same terms in another order: each sum to a few 2^-24 of itself, half of that in its root
        assert float((a - b).abs().max()) <= 1e-5 * float((b - init.cuda()).abs().max()) + 2 ** -23 * float(b.abs().max())


@pytest.mark.parametrize("family", ["adafaclo", "elo", "celo2", "elo_celo2"])
def test_new_weights_of_the_network_reach_all_launches(family):
    """Weights written into the flat tensor between steps act as those of an optimizer that is made with them: parts of the network
    reach the kernels through descriptors, others as arguments of a launch."""
    from pylo_b200 import optim

    cls = {"adafaclo": optim.AdafacLO_CUDA, "elo": optim.ELO_CUDA, "celo2": optim.CELO2_CUDA, "elo_celo2": optim.ELO_CELO2_CUDA}[family]
    case = dict(shapes=[(40, 24), (300, 1028), (33, 35), (24,)], init_seed=55, init_scale=0.1, grad_seed=56, grad_scale=0.3)
    new = _nets(family)
    with torch.no_grad():
        for w in new.parameters():
            w.mul_(1.5)
    runs = []
    for late in (False, True):
        params = [torch.nn.Parameter(v.cuda()) for v in cases.init_values(case)]
        opt = cls(params, lr=1e-2, network=_nets(family))
        for t in (1, 2):
            for p, g in zip(params, cases.grads_at(case, t)):
                p.grad = g.cuda()
            if t == 2:
                made = cls(params, lr=1e-2, network=copy.deepcopy(new))
                if late:
                    opt._w_flat.copy_(made._w_flat)
                else:
                    made.load_state_dict(opt.state_dict())
                    opt = made
            opt.step()
        runs.append([p.detach().clone() for p in params])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    with pytest.raises(AttributeError):   # plans point to the old one
        opt._w_flat = made._w_flat
