"""Tiles of the state sweep: how many turns of the CTAs that run at once, for models of units that go different ways."""

import numpy as np
import pytest

from pylo_b200 import _lib as L
from pylo_b200 import plan
from pylo_b200.optim.AdafacLO_cuda import AdafacLO_CUDA


def _order(shapes, family=L.FAM_VELO):
    d = np.zeros(len(shapes), dtype=L.DESC_DTYPE)
    for x, s in zip(d, shapes):
        _, fdims, axis = AdafacLO_CUDA._factoring(s)
        plan.fill_geometry(x, s, fdims, axis)
    return plan.sum_order(family, d, d["n"].tolist(), d["mode"], False)


def _turns(sizes, e):
    return -(-sum(-(-n // e) for n in sizes) // (2 * L.SM_COUNT))


def _vit(width, layers):
    block = [(width,), (width, 3 * width), (3 * width,), (width, width), (width,), (width,), (width, 4 * width), (4 * width,), (4 * width, width), (width,)]
    return [(width, 3, 16, 16), (width,), (197, width)] + block * layers


@pytest.mark.parametrize("width,layers", [(192, 6), (192, 8), (320, 2), (384, 2)])
def test_a_patch_embedding_is_not_one_turn(width, layers):
    """Its tiles take longer and come last: one turn of long tiles was 7 to 15 % slower per step than three."""
    shapes = _vit(width, layers)
    order = _order(shapes)
    assert order.small is None and _turns([int(np.prod(s)) for s in shapes], order.elems) >= 3


def test_two_turns_where_all_units_go_the_same_way():
    shapes = [(384, 1152), (1152,), (384, 384), (384,), (384, 1536), (1536,), (1536, 384), (384,)] * 3
    sizes = [int(np.prod(s)) for s in shapes]
    assert _turns(sizes, _order(shapes).elems) == 2
    assert _turns(sizes + [64 * 147], _order(shapes + [(64, 3, 7, 7)]).elems) != 2


def test_tiles_of_many_small_units_are_counted_by_what_is_in_them():
    """A matrix per unit, as CELO2 takes convolutions: their tiles are no longer for a larger limit, and smaller ones do not pay."""
    patches, rest = [256] * 1152, [384 * 1152, 384 * 384, 384 * 1536, 1536 * 384] * 5
    e = plan.state_tile(patches + rest)
    assert e >= plan.tile_elems(sum(patches + rest), 1024, 4 * L.SM_COUNT)
    assert plan.state_tile([9] * 4096) >= 1024
    assert plan.state_tile([2**33, 3]) == L.TILE_ELEMS
