"""The tensor-core network sweep of AdafacLO / ELO against fp64, for gradients and networks that stretch the range of its operands.

A step's movement is compared with the network evaluated in fp64 on the state that the step leaves.  With operands of 22 significant
bits and fp32 sums a dot product is within 2^-21.7 (3e-7) of the sum of its terms' magnitudes; two hidden layers, the heads and the
features' own roundings stay below 2^-20 of the magnitudes carried through the network, to which the rounding of the parameter is added.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

TIME_SCALES = [1.0, 3.0, 10.0, 30.0, 100.0, 300.0, 1000.0, 3000.0, 10000.0, 30000.0, 100000.0]
LR = 1e6   # the movement is then far larger than the parameter and its rounding


def _gradient(kind, shape, gen):
    g = torch.randn(*shape, device="cuda", generator=gen) * 1e-3
    if kind == "outliers":
        g[torch.rand(shape, device="cuda", generator=gen) < 0.01] *= 100
    elif kind == "one entry":     # its feature is sqrt(n) times the root mean square
        g.zero_()
        g.view(-1)[g.numel() // 3] = 1.0
    elif kind == "rows":
        g *= torch.exp(3 * torch.randn((shape[0],) + (1,) * (len(shape) - 1), device="cuda", generator=gen))
    elif kind == "tiny":
        g *= 1e-6
    return g


def _features(p, g, st, fd, axis):
    safe = lambda x: torch.rsqrt(x.clamp(min=1e-9))
    m, v = st["exp_avg"].double(), st["exp_avg_sq"].double().reshape(p.shape)
    r, c = st["exp_avg_sq_r"].double(), st["exp_avg_sq_c"].double()
    rs = torch.rsqrt(v + 1e-6)
    k = safe(r + 1e-9) if fd is None else safe(r / (r.mean(axis, keepdim=True) + 1e-9)) * safe(c)
    k, r, c = k.expand(m.shape), r.expand(m.shape), c.expand(m.shape)
    f = [g.double(), p.double(), *m, v, *(m * rs), rs, *(k * g.double()), *r, *c, *torch.rsqrt(r + 1e-8), *torch.rsqrt(c + 1e-8), *(k * m)]
    f = torch.stack([x.reshape(-1) for x in f])
    return f * torch.rsqrt(f.pow(2).mean(1, keepdim=True) + 1e-5)


def _step(shape, kind, scale, steps=2):
    from pylo_b200 import models, optim

    gen = torch.Generator(device="cuda").manual_seed(7)
    torch.manual_seed(3)
    net = models.MetaMLP(39, 32, 1)
    with torch.no_grad():
        for q in net.parameters():
            q.mul_(scale)
    p = torch.nn.Parameter(torch.randn(*shape, device="cuda", generator=gen) * 0.02)
    opt = optim.AdafacLO_CUDA([p], lr=1.0, network=net)
    for t in range(steps):
        opt.param_groups[0]["lr"] = LR if t == steps - 1 else 1.0
        p.grad = _gradient(kind, shape, gen)
        if kind == "not a number" and t == steps - 1:
            p.grad.view(-1)[5] = float("nan")
        before = p.detach().clone()
        opt.step()
    opt.check_status()
    W = [q.detach().double().cuda() for q in net.parameters()]
    time = torch.tanh((steps - 1) / torch.tensor(TIME_SCALES, device="cuda", dtype=torch.float64) - 1)
    return opt, p, before, W, W[1] + W[0][:, 28:] @ time


@pytest.mark.parametrize("scale", [1.0, 4.0, 0.01])   # larger ones overflow the heads' exponential
@pytest.mark.parametrize("kind", ["plain", "outliers", "one entry", "rows", "tiny"])
@pytest.mark.parametrize("shape", [(64, 128), (130, 1023), (1024, 2048), (70, 36, 3, 3), (129,)])
def test_movement_against_fp64(shape, kind, scale):
    opt, p, before, W, b1 = _step(shape, kind, scale)
    _, fd, axis = opt._factoring(tuple(shape))
    f = _features(before, p.grad, opt.state[p], fd, axis)
    h = torch.relu(W[0][:, :28] @ f + b1[:, None])
    h = torch.relu(W[2] @ h + W[3][:, None])
    o = W[4] @ h + W[5][:, None]
    size = W[0][:, :28].abs() @ f.abs() + b1.abs()[:, None]
    size = W[4].abs() @ (W[2].abs() @ size + W[3].abs()[:, None]) + W[5].abs()[:, None]
    grow = LR * float(opt.step_mult) * torch.exp(o[1] * float(opt.exp_mult))
    want = before.double().reshape(-1) - o[0] * grow
    error = (p.detach().double().reshape(-1) - want).abs()
    bound = 2.0 ** -20 * grow * (size[0] + o[0].abs() * float(opt.exp_mult) * size[1]) + 2.0 ** -23 * want.abs()
    assert bool((error <= bound).all()), float((error / bound).max())


@pytest.mark.parametrize("shape", [(64, 128), (33, 37)])
def test_a_gradient_that_is_not_a_number_counts_as_no_activation(shape):
    """It makes the tensor's normalisers, and with them every first-layer sum, not a number: relu, as fmaxf, gives zero then."""
    opt, p, before, W, _ = _step(shape, "not a number", 1.0)
    o = W[4] @ torch.relu(W[3]) + W[5]
    want = before.double() - LR * float(opt.step_mult) * o[0] * torch.exp(o[1] * float(opt.exp_mult))
    assert torch.allclose(p.detach().double(), want, rtol=1e-5, atol=0)


@pytest.mark.parametrize("family", ["adafaclo", "elo"])
@pytest.mark.parametrize("shapes", [[(5, 3)], [(128, 96), (128,), (10, 128), (10,)], [(33, 37), (40,)] * 3 + [(300, 64)],
                                    [(24, 16), (24,)] * 12, [(3, 5)] * 150])
def test_networks_made_by_the_front_launch(family, shapes, monkeypatch):
    """One launch less than with a preparation of its own, and the same step: the sums over a tensor's tiles are added up in fp64."""
    from pylo_b200 import plan
    from test_gpu_properties import _make

    outs = []
    for joined in (True, False):
        if not joined:
            monkeypatch.setattr(plan, "small_networks", lambda n, cluster: False)
        gen = torch.Generator(device="cuda").manual_seed(11)
        params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=gen) * 0.1) for s in shapes]
        opt = _make(family, params)
        for _ in range(3):
            for p in params:
                p.grad = torch.randn(*p.shape, device="cuda", generator=gen) * 0.3
            opt.step()
        opt.check_status()
        plans = [pl for _, pl in opt._plans.values()]
        assert all(pl.small for pl in plans)
        want = plan.small_networks(len(shapes), plans[0].small[0])
        assert all(bool(pl.step_plan.small_networks) == want for pl in plans)
        outs.append([p.detach().clone() for p in params])
    for a, b in zip(*outs):
        assert torch.allclose(a, b, rtol=1e-6, atol=1e-8)
