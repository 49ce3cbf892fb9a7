"""Launches that small models share: the same steps as with launches of their own, and where the line between the two lies."""

import numpy as np
import pytest
import torch

from pylo_b200 import _lib as L
from pylo_b200 import plan


def test_state_tiles_end_in_whole_turns():
    assert plan.state_tile([118282]) == 1024                                   # one turn of single passes
    for sizes in ([4104100], [2359296, 1179648] + [589824] * 2, [11334246], [10715136]):
        e = plan.state_tile(sizes)
        tiles = sum(-(-n // e) for n in sizes)
        turns = -(-tiles // (2 * L.SM_COUNT))
        assert e % 1024 == 0 and 1024 <= e <= L.TILE_ELEMS
        assert e == plan.tile_elems(sum(sizes), 1024, 4 * L.SM_COUNT) or (turns != 2 and tiles > 0.8 * turns * 2 * L.SM_COUNT)
    assert plan.state_tile([86443776]) == plan.state_tile([2**29]) == L.TILE_ELEMS
    assert plan.state_tile([]) >= 1024 and plan.state_tile([1]) == 1024


def test_a_further_cluster_only_where_it_costs_no_turn():
    assert plan.small_networks(6, 16) and plan.small_networks(7, 16) and not plan.small_networks(8, 16)
    assert plan.small_networks(15, 8) and not plan.small_networks(16, 8)
    assert plan.small_networks(1, 1) and plan.small_networks(2, 1) and not plan.small_networks(3, 1) and not plan.small_networks(101, 2)


def _velo(shapes, steps=3):
    from pylo_b200 import models, optim

    torch.manual_seed(5)
    gen = torch.Generator(device="cuda").manual_seed(9)
    params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=gen) * 0.1) for s in shapes]
    mlp = models.VeLOMLP()
    with torch.no_grad():
        for name, w in mlp.named_parameters():
            if "weights_" in name:
                w.mul_(0.05)
    return params, optim.VeLO_CUDA(params, lr=1e-1, num_steps=100, rnn=models.VeLORNN(), mlp=mlp), gen


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(5, 3)], [(128, 96), (128,), (10, 128), (10,)], [(24, 16), (24,)] * 8, [(24, 16), (24,)] * 8 + [(7,)]])
def test_velo_inputs_in_one_launch(shapes, monkeypatch):
    """Sums, inputs and first layer have the order of the separate launches: the steps are the same to the last bit."""
    outs = []
    for most in (L.VELO_INPUTS_MOST, 0):
        monkeypatch.setattr(L, "VELO_INPUTS_MOST", most)
        params, opt, gen = _velo(shapes)
        for t in range(4):
            for p in params:
                p.grad = torch.randn(*p.shape, device="cuda", generator=gen) * 0.01
            opt.step(torch.tensor(2.5 - 0.1 * t, device="cuda"))
        assert opt._plan[1]["rnn"].mixed == int(len(shapes) <= most)
        outs.append([p.detach().clone() for p in params] + list(opt.lstm_hidden_state) + [opt.loss_buffer[k].clone() for k in ("means", "running_min", "iteration")])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["celo2", "elo_celo2"])
@pytest.mark.parametrize("orthogonalize", [True, False])
def test_the_tail_takes_adamw_along(family, orthogonalize, monkeypatch):
    from pylo_b200 import models, optim

    cls = optim.CELO2_CUDA if family == "celo2" else optim.ELO_CELO2_CUDA
    shapes = [(128, 96), (128,), (33, 37), (5001,), (10, 128), (1,)]
    outs = []
    for most in (L.TAIL_ONE_LAUNCH, 0):
        monkeypatch.setattr(L, "TAIL_ONE_LAUNCH", most)
        torch.manual_seed(5)
        gen = torch.Generator(device="cuda").manual_seed(9)
        params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=gen) * 0.1) for s in shapes]
        opt = cls(params, lr=1e-2, weight_decay=0.1, clip_grad=True, orthogonalize=orthogonalize, network=models.CELO2MLP())
        for _ in range(3):
            for p in params:
                p.grad = torch.randn(*p.shape, device="cuda", generator=gen) * 0.3
            opt.step()
        outs.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*outs))
