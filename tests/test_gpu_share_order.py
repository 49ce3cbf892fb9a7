"""A rank's share of a model of many tensors steps as the whole model does, bit for bit, in every launch whose shape follows from the
number of tensors: the factor phase's CTAs, and the networks beside the front launch of a small model."""

import types

import pytest
import torch

from test_gpu_shares import _build, _params, _results, _step

pytestmark = pytest.mark.gpu

# of 26 and 24 tensors with factors a share of two ranks has at most 18; 19 strips of rows, column vectors of either width, means of
# every kind; "small": the whole has more tensors than a further cluster makes networks for, a share has not
MANY = {"matrices": [(600, 260), (260,), (600, 1100)] * 8 + [(520, 264)] * 10,
        "convolutions": [(96, 128, 3, 3), (96,), (600, 36, 3), (40, 70, 2, 2), (40,)] * 8,
        "small": [(24, 16), (24,), (33, 37), (40,)] * 6}


@pytest.mark.parametrize("world", [2, 4])
@pytest.mark.parametrize("model", sorted(MANY))
@pytest.mark.parametrize("family", ["adafaclo", "elo", "velo"])
def test_a_share_of_many_tensors_steps_as_the_whole_does(family, model, world, monkeypatch):
    from pylo_b200 import zero

    shapes = MANY[model]
    steps = 1 if family == "velo" else 2
    params = _params(shapes)
    cls, kw = _build(family, params)
    opt = cls(params, **kw)
    for t in range(1, steps + 1):
        _step(opt, family, params, range(len(shapes)), t)
    whole = _results(opt, family, params, range(len(shapes)), len(shapes))
    del opt, params
    for rank in range(world):
        monkeypatch.setattr(zero, "dist", types.SimpleNamespace(is_initialized=lambda: True, get_world_size=lambda pg: world, get_rank=lambda pg, r=rank: r))
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


@pytest.mark.parametrize("shapes", [[(128, 784), (128,), (128, 128), (128,), (10, 128), (10,)], [(33, 37), (40,)] * 3 + [(300, 64)], [(2000, 37)]])
def test_networks_beside_the_front_launch_change_no_bit(shapes, monkeypatch):
    """The sweep and the preparation add a tensor's partials up in the same order."""
    from pylo_b200 import plan
    from test_gpu_properties import _make

    outs = []
    for joined in (True, False):
        monkeypatch.setattr(plan, "small_networks", lambda n, cluster: joined)
        gen = torch.Generator(device="cuda").manual_seed(11)
        params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=gen) * 0.1) for s in shapes]
        opt = _make("adafaclo", params)
        for _ in range(3):
            for p in params:
                p.grad = torch.randn(*p.shape, device="cuda", generator=gen) * torch.exp(7 * torch.randn(*p.shape, device="cuda", generator=gen))
            opt.step()
        opt.check_status()
        (_, pl), = opt._plans.values()
        assert bool(pl.step_plan.small_networks) == joined
        outs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*outs))
