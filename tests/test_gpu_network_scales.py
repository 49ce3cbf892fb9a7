"""The tensor-core network sweep of AdafacLO / ELO against fp64, for networks whose hidden units have scales of their own and for tensors
of many elements.

Multiplying a hidden unit's weights and bias by s and its column in the next layer by 1 / s leaves the function as it is, and the sum of
its terms' magnitudes: the bound is that of evenly scaled networks, whatever s is and however many elements a tensor has.  It is the one
of test_gpu_tensor_core_planes.py (2^-20 of the magnitudes carried through the network, and the rounding of the parameter), with a floor
under a feature's magnitude: the planes hold a feature to 2^-25 of a unit 2^-q of its root mean square, 2^q sqrt(n) <= 2^15, q <= 6."""

import math

import pytest
import torch

from test_gpu_tensor_core_planes import LR, TIME_SCALES, _features, _gradient

pytestmark = pytest.mark.gpu


def _rescale(net, units, kind):
    """The same function with the first ``units`` hidden units of a layer scaled by ``kind``'s factors."""
    w1, b1, w2, b2, w3, _ = net.parameters()
    which, factor = kind
    s = torch.full((units,), factor)
    with torch.no_grad():
        if which == "first layer":
            w1[:units] *= s[:, None]
            b1[:units] *= s
            w2[:, :units] /= s
        elif which == "second layer":
            w2[:units] *= s[:, None]
            b2[:units] *= s
            w3[:, :units] /= s


def _run(shape, grad, kind, units):
    from pylo_b200 import models, optim

    gen = torch.Generator(device="cuda").manual_seed(7)
    torch.manual_seed(3)
    net = models.MetaMLP(39, 32, 1)
    if kind:
        _rescale(net, units, kind)
    p = torch.nn.Parameter(torch.randn(*shape, device="cuda", generator=gen) * 0.02)
    opt = optim.AdafacLO_CUDA([p], lr=1.0, network=net)
    for t in range(2):
        opt.param_groups[0]["lr"] = LR if t else 1.0
        p.grad = _gradient(grad, shape, gen)
        before = p.detach().clone()
        opt.step()
    opt.check_status()
    return opt, p, before, [q.detach().double().cuda() for q in net.parameters()]


def _check(opt, p, before, W):
    time = torch.tanh(1 / torch.tensor(TIME_SCALES, device="cuda", dtype=torch.float64) - 1)
    b1 = W[1] + W[0][:, 28:] @ time
    _, fd, axis = opt._factoring(tuple(p.shape))
    n = p.numel()
    st = opt.state[p]
    rows = max(1, min(p.shape[0], (1 << 20) // (n // p.shape[0])))   # fp64 features of about a million elements, at both ends
    grad = p.grad
    full = _root_mean_squares(before, grad, st, fd, axis)
    worst = 0.0
    for x0 in sorted({0, p.shape[0] - rows}):
        f = _raw(before, grad, st, fd, axis, x0, x0 + rows) * full[:, None]
        h = torch.relu(W[0][:, :28] @ f + b1[:, None])
        h = torch.relu(W[2] @ h + W[3][:, None])
        o = W[4] @ h + W[5][:, None]
        q = min(6, 14 - math.floor(math.log2(1.001 * math.sqrt(n))))
        size = W[0][:, :28].abs() @ (f.abs() + 2.0 ** (20 - 25 - q)) + b1.abs()[:, None]
        size = W[4].abs() @ (W[2].abs() @ size + W[3].abs()[:, None]) + W[5].abs()[:, None]
        grow = LR * float(opt.step_mult) * torch.exp(o[1] * float(opt.exp_mult))
        was = before[x0:x0 + rows].double().reshape(-1)
        want = was - o[0] * grow
        error = (p.detach()[x0:x0 + rows].double().reshape(-1) - want).abs()
        bound = 2.0 ** -20 * grow * (size[0] + o[0].abs() * float(opt.exp_mult) * size[1]) + 2.0 ** -23 * want.abs()
        worst = max(worst, float((error / bound).max()))
    assert worst <= 1.0, worst


def _raw(p, g, st, fd, axis, x0, x1):
    """The 28 features of rows x0 to x1, not normalised, in fp64."""
    safe = lambda x: torch.rsqrt(x.clamp(min=1e-9))
    part = lambda t, k=0: t.narrow(k, x0, x1 - x0) if t.shape[k] > 1 else t
    m = part(st["exp_avg"], 1).double()
    v = part(st["exp_avg_sq"].reshape(p.shape)).double()
    r, c = part(st["exp_avg_sq_r"], 1).double(), part(st["exp_avg_sq_c"], 1).double()
    mean = st["exp_avg_sq_r"].double().mean(axis, keepdim=True)
    mean = part(mean, 1)
    rs = torch.rsqrt(v + 1e-6)
    k = safe(r / (mean + 1e-9)) * safe(c)
    k, r, c = k.expand(m.shape), r.expand(m.shape), c.expand(m.shape)
    gd = part(g).double()
    f = [gd, part(p).double(), *m, v, *(m * rs), rs, *(k * gd), *r, *c, *torch.rsqrt(r + 1e-8), *torch.rsqrt(c + 1e-8), *(k * m)]
    return torch.stack([x.reshape(-1) for x in f])


def _root_mean_squares(p, g, st, fd, axis):
    """Reciprocals of them over the whole tensor, by pieces of rows."""
    total, step = 0.0, max(1, (1 << 22) // (p.numel() // p.shape[0]))
    for x0 in range(0, p.shape[0], step):
        total = total + _raw(p, g, st, fd, axis, x0, min(p.shape[0], x0 + step)).pow(2).sum(1)
    return torch.rsqrt(total / p.numel() + 1e-5)


def test_the_pieces_are_the_features():
    opt, p, before, _ = _run((70, 128), "plain", None, 0)
    _, fd, axis = opt._factoring(tuple(p.shape))
    want = _features(before, p.grad, opt.state[p], fd, axis)
    args = (before, p.grad, opt.state[p], fd, axis)
    assert torch.allclose(_raw(*args, 0, 70) * _root_mean_squares(*args)[:, None], want, rtol=1e-12, atol=0)


@pytest.mark.parametrize("kind", [("first layer", 1e-3), ("first layer", 1e-4), ("first layer", 1e4), ("second layer", 1e-3), ("second layer", 1e3)])
@pytest.mark.parametrize("units", [16, 1])
@pytest.mark.parametrize("shape", [(64, 128), (130, 1023), (4096, 4096)])
def test_units_with_scales_of_their_own(shape, units, kind):
    _check(*_run(shape, "plain", kind, units))


@pytest.mark.parametrize("grad", ["plain", "outliers", "one entry"])
@pytest.mark.parametrize("kind", [None, ("first layer", 1e-4)])
@pytest.mark.parametrize("shape", [(4096, 14336), (32000, 4096)])
def test_large_tensors(shape, kind, grad):
    _check(*_run(shape, grad, kind, 16))


@pytest.mark.parametrize("shape", [(64, 128), (37, 53), (1024, 1024), (64, 48, 3, 3)])
def test_small_values_are_rounded_not_cut(shape):
    """A network that hands one feature through, and a gradient whose entries but one lie below fp16's normal range after scaling: what
    the two planes hold is within half of fp16's smallest step, whichever way."""
    from pylo_b200 import models, optim

    gen = torch.Generator(device="cuda").manual_seed(9)
    net = models.MetaMLP(39, 32, 1)
    with torch.no_grad():
        for w in net.parameters():
            w.zero_()
        w1, _, w2, _, w3, _ = net.parameters()
        w1[0, 0] = w2[0, 0] = w3[0, 0] = 1.0
    p = torch.nn.Parameter(torch.zeros(*shape, device="cuda"))
    n = p.numel()
    q = min(6, 14 - math.floor(math.log2(1.001 * math.sqrt(n))))
    rms = 10.0
    g = torch.rand(shape, device="cuda", generator=gen) * (rms * 2.0 ** (-14 - q))
    g.view(-1)[n // 3] = rms * math.sqrt(n)
    p.grad = g
    opt = optim.AdafacLO_CUDA([p], lr=LR, network=net)
    opt.step()
    opt.check_status()
    scale = 1.0 / math.sqrt(float(g.double().pow(2).mean()) + 1e-5)
    got = -p.detach().double() / (LR * float(opt.step_mult))
    error = (got - g.double() * scale).view(-1)
    error[n // 3] = 0.0
    half = 2.0 ** (-25 - q)
    assert float(error.abs().max()) <= 1.01 * half, float(error.abs().max()) / half
    assert abs(float(error.mean())) <= 0.1 * half
