"""A rank's share of a model, stepped alone on one GPU, against the step of a process that has all of it: bit for bit.

The ranks take turns here, without a process group: ownership and the notes on the parameters are those of a sharded run, the
exchange of parameters is left out.  tests/test_gpu_multi.py runs the whole on two GPUs."""

import types

import pytest
import torch

import cases
from test_gpu_multi import SHAPES

pytestmark = pytest.mark.gpu

# the two-GPU tests' model (one rank of which owns (300, 260) alone); one that takes the launch of small models; a middling one, whose
# shares would have smaller tiles; one whose state sweep goes through the ring, which a share would not
MODELS = {"general": SHAPES + [(72, 48), (300, 260)], "small": [(128, 784), (128,), (128, 128), (128,), (10, 128), (10,)],
          "middling": [(1000, 1300), (1300,), (700, 1001), (64, 5, 3, 3), (2048, 1024), (300, 4100)],
          "large": [(4096, 4096)] * 4 + [(4096,), (1024, 4096), (8, 3, 5)]}


def _params(shapes):
    gen = torch.Generator(device="cuda").manual_seed(5)
    return [torch.nn.Parameter(torch.randn(s, device="cuda", generator=gen) * 0.05) for s in shapes]


def _build(family, params):
    from pylo_b200 import models, optim

    torch.manual_seed(0)
    if family == "adafaclo":
        return optim.AdafacLO_CUDA, dict(lr=1e-2, network=models.MetaMLP(39, 32, 1))
    if family == "elo":
        return optim.ELO_CUDA, dict(lr=1e-2, weight_decay=0.1, network=models.MetaMLP(39, 32, 1), mlp_precision="fp32")
    return optim.VeLO_CUDA, dict(lr=10.0, num_steps=100, rnn=models.VeLORNN(lstm_hidden_size=32), mlp=models.VeLOMLP())


def _step(opt, family, params, which, t):
    for i in which:
        gen = torch.Generator(device="cuda").manual_seed(100 * t + i)
        params[i].grad = torch.randn(params[i].shape, device="cuda", generator=gen) * 0.2
    opt.step(torch.tensor(cases.velo_loss(t))) if family == "velo" else opt.step()


def _results(opt, family, params, which, T):
    out = {i: [params[i].detach().clone()] if family != "velo" else [] for i in which}   # VeLO's wait for all ranks' LSTM inputs
    for i in which:
        st = opt.state[params[i]]
        out[i] += [x.clone() for x in st.values() if torch.is_tensor(x) and x.is_cuda]
        if family == "velo":
            out[i].append(opt._plan[1]["buf"]["x_in"][T - 1 - i].clone())   # rows are flipped
    return out


@pytest.mark.parametrize("model", sorted(MODELS))
@pytest.mark.parametrize("family", ["adafaclo", "elo", "velo"])
def test_a_share_steps_as_the_whole_does(family, model, monkeypatch):
    from pylo_b200 import zero

    shapes = MODELS[model]
    steps = 1 if family == "velo" else 2
    params = _params(shapes)
    cls, kw = _build(family, params)
    opt = cls(params, **kw)
    for t in range(1, steps + 1):
        _step(opt, family, params, range(len(shapes)), t)
    whole = _results(opt, family, params, range(len(shapes)), len(shapes))
    del opt, params
    for rank in range(2):
        monkeypatch.setattr(zero, "dist", types.SimpleNamespace(is_initialized=lambda: True, get_world_size=lambda pg: 2, get_rank=lambda pg, r=rank: r))
        params = _params(shapes)
        shard = zero.ShardedStep(params)
        cls, kw = _build(family, params)
        opt = zero.sharded_optimizer(cls, shard, **kw)
        for t in range(1, steps + 1):
            _step(opt, family, params, shard.owned, t)
        mine = _results(opt, family, params, shard.owned, len(shapes))
        assert shard.owned
        for i in shard.owned:
            for a, b in zip(mine[i], whole[i]):
                assert torch.equal(a, b), (rank, i, shapes[i])
        del opt, params, shard
