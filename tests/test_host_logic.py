"""Host-side logic that needs no GPU: factored-dims rules, geometry, tiling, ownership, flat layout."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import pylo_oracle as O
from pylo_b200 import _lib as L
from pylo_b200 import plan, workloads, zero
from pylo_b200.optim import _common as K

SHAPES = [(64, 32), (32, 64), (48, 48), (7, 5, 3), (12, 3, 4, 4), (4, 4, 9, 9), (768, 3, 16, 16), (5,), ()]


@pytest.mark.parametrize("shape", SHAPES)
def test_factored_dims_rules_agree_with_the_oracle(shape):
    assert K.factored_dims_sorted(shape) == O.factored_dims_sorted(shape)
    assert K.factored_dims_argsort(shape) == O.factored_dims_argsort(shape)
    assert K.factored_dims_velo(shape) == O.factored_dims_velo(shape)


def test_velo_tie_rule():
    assert K.factored_dims_velo((1024, 1024)) == (1, 0)       # equal sizes swap (velo_cuda.py:121-131)
    assert K.factored_dims_velo((8, 8, 3, 3)) == (0, 1)       # except 4-D with axes (0, 1)
    assert K.factored_dims_sorted((4096, 4096)) == (0, 1)


@pytest.mark.parametrize("shape", [s for s in SHAPES if len(s) >= 2])
def test_geometry_indexes_like_broadcasting(shape):
    """a / b vector indices from the 5-D view equal what broadcasting a keep-dim vector would read."""
    fd = K.factored_dims_argsort(shape)
    dc, dr = fd
    Ov, X, M, Y, I, r_is_a = plan.geometry(shape, fd)
    n = int(np.prod(shape))
    idx = np.arange(n)
    i = idx % I; t = idx // I; y = t % Y; t //= Y; m = t % M; t //= M; x = t % X; o = t // X
    a = ((o * X + x) * M + m) * I + i
    b = ((o * M + m) * Y + y) * I + i
    r_shape, c_shape = list(shape), list(shape)
    r_shape[dr], c_shape[dc] = 1, 1
    rvec = np.arange(int(np.prod(r_shape))).reshape(r_shape)
    cvec = np.arange(int(np.prod(c_shape))).reshape(c_shape)
    r_b = np.broadcast_to(rvec, shape).reshape(-1)
    c_b = np.broadcast_to(cvec, shape).reshape(-1)
    assert np.array_equal(r_b, a if r_is_a else b)
    assert np.array_equal(c_b, b if r_is_a else a)


def test_tiles_cover_every_element_once():
    sizes = [1, L.TILE_ELEMS, L.TILE_ELEMS + 1, 5 * L.TILE_ELEMS - 3]
    tiles, ranges = plan.make_tiles(sizes)
    for i, n in enumerate(sizes):
        t0, k = ranges[i]
        mine = tiles[t0:t0 + k]
        assert (mine["tensor"] == i).all()
        assert mine["start"][0] == 0 and (np.diff(mine["start"]) == L.TILE_ELEMS).all()
        assert mine["start"][-1] < n <= mine["start"][-1] + L.TILE_ELEMS


@pytest.mark.parametrize("world", [1, 2, 4, 8])
def test_partition_is_deterministic_balanced_and_total(world):
    shapes = workloads.llama3_8b()
    owner = zero.partition(shapes, world)
    assert owner == zero.partition(shapes, world)
    loads = [sum(workloads.numel(s) for s, o in zip(shapes, owner) if o == r) for r in range(world)]
    assert sum(loads) == workloads.total_params(shapes)
    assert max(loads) / (sum(loads) / world) < 1.01
    offsets, shard = zero.flat_layout(shapes, owner, world)
    spans = sorted((off, off + workloads.numel(s)) for off, s in zip(offsets, shapes))
    assert all(a1 <= b0 for (_, a1), (b0, _) in zip(spans, spans[1:])), "tensors overlap in the flat buffer"
    assert all(off % zero.ALIGN == 0 for off in offsets)
    assert all(o * shard <= off < (o + 1) * shard for off, o in zip(offsets, owner))


@pytest.mark.parametrize("world", [1, 2, 4, 8])
@pytest.mark.parametrize("wl", ["llama3_8b", "gpt2_medium"])
def test_block_layout_keeps_gather_ranges_contiguous_and_tight(world, wl):
    shapes = workloads.WORKLOADS[wl]()
    blocks = 4
    owner, block, offsets, subs = zero.partition_blocks(shapes, world, blocks)
    total = workloads.total_params(shapes)
    spans = sorted((off, off + workloads.numel(s)) for off, s in zip(offsets, shapes))
    assert all(a1 <= b0 for (_, a1), (b0, _) in zip(spans, spans[1:])), "tensors overlap"
    base = [sum(subs[:b]) * world for b in range(blocks)]
    for off, s, o, b in zip(offsets, shapes, owner, block):
        lo = base[b] + o * subs[b]
        assert lo <= off and off + workloads.numel(s) <= lo + subs[b], "tensor outside its (block, rank) cell"
    if wl == "llama3_8b":
        assert sum(subs) * world < 1.01 * total  # indivisible 525 M-element tensors must not inflate the buffer


def test_workload_sizes():
    assert workloads.total_params(workloads.mlp_784()) == 118282
    assert workloads.total_params(workloads.celo2_4096()) == 4096 * 4096 + 4096
    assert abs(workloads.total_params(workloads.llama3_8b()) - 8.03e9) < 1e7
    assert abs(workloads.total_params(workloads.gpt2_medium()) - 354.8e6) < 1e6
    assert abs(workloads.total_params(workloads.vit_b16()) - 86.6e6) < 1e6


def test_cuda_classes_refuse_to_run_without_a_gpu():
    if torch.cuda.is_available():
        pytest.skip("GPU present")
    from pylo_b200 import models, optim

    p = [torch.nn.Parameter(torch.zeros(4, 4))]
    with pytest.raises(RuntimeError):
        optim.CELO2_CUDA(p, network=models.CELO2MLP())
    with pytest.raises(RuntimeError):
        optim.AdafacLO_CUDA(p, network=models.MetaMLP(39, 32, 1))


@pytest.mark.parametrize("tc", [False, True])
@pytest.mark.parametrize("family", [L.FAM_ADAFAC, L.FAM_CELO2])
@pytest.mark.parametrize("X,Y", [(4096, 4096), (14336, 4096), (4096, 14336), (128256, 4096), (40, 4100), (129, 300), (64, 128)])
def test_apply_items_cover_a_tensor_exactly_once(family, X, Y, tc):
    """Work items of the tiled apply sweeps: whole rows x column blocks, every element in exactly one item."""
    if tc and family != L.FAM_ADAFAC:
        pytest.skip("tensor-core kernels exist for the AdafacLO family only")
    rt, width, tag = (plan.tensor_core_rows([(X, Y)]), 128, 0) if tc else plan.apply_tile_shape(family, X, Y)
    n_r, n_c = (X + rt - 1) // rt, (Y + width - 1) // width
    assert (n_r - 1) * rt < X <= n_r * rt and (n_c - 1) * width < Y <= n_c * width
    if tc:
        # the busiest worker's items, each its rows and a row and a half of set-up: no other height makes it shorter
        share = lambda r: -(-(-(-X // r) * n_c) // L.TC_WORKERS) * (r + 1.5)
        assert rt in (1, 2, 4, 8, 16, 32, 64) and share(rt) == min(share(r) for r in (1, 2, 4, 8, 16, 32, 64))
    elif family == L.FAM_ADAFAC:
        assert width in (32, 64, 128, 256) and tag & 0xffff == width and rt == 32 * (tag >> 16)
    else:
        assert width == 4 * tag and rt == 16 * (256 // tag)


@pytest.mark.parametrize("family,tc", [(L.FAM_ADAFAC, True), (L.FAM_ADAFAC, False), (L.FAM_CELO2, False), (L.FAM_VELO, False)])
@pytest.mark.parametrize("fast,slow", [
    ([(1, 64, 128)], []),
    ([], [127, 129, 1]),
    ([(3, 129, 300), (2, 40, 4100)], [5, 4096, 70001]),
    ([(0, 1025, 4096), (1, 1, 4), (2, 33, 260)], [1]),
])
def test_apply_work_lists_cover_all_units_exactly_once(family, tc, fast, slow):
    """The whole list as the kernels decode it (tags, rows per thread, runs of 128 elements)."""
    slow = [(10 + k, n) for k, n in enumerate(slow)]
    seen = {u: np.zeros((X, Y), dtype=np.int32) for u, X, Y in fast}
    runs = {u: np.zeros(n, dtype=np.int32) for u, n in slow if tc}   # the CUDA-core sweeps leave these to another kernel
    n_gen = 0
    for k, it in enumerate(plan.apply_items(family, tc, fast, slow)):
        u, tag = int(it["tensor"]), int(it["pad_"])
        if tc and tag >= L.TC_GEN_ITEM:
            assert k == n_gen and it["cb"] == 0, "items on units that are not FAST2D come first"
            n_gen += 1
            step = 128 * (tag & 0xffff)
            runs[u][it["strip"] * step:(it["strip"] + 1) * step] += 1
            assert it["strip"] * step < len(runs[u])
            continue
        if tc:
            rt, w = tag, 128
        elif family == L.FAM_ADAFAC:
            rt, w = 32 * (tag >> 16), tag & 0xffff
        else:
            rt, w = (tag >> 16) * (256 // (tag & 0xffff)), 4 * (tag & 0xffff)
        r, c = int(it["strip"]) * rt, int(it["cb"]) * w
        assert rt > 0 and r < seen[u].shape[0] and c < seen[u].shape[1]
        seen[u][r:r + rt, c:c + w] += 1
    assert all((x == 1).all() for x in list(seen.values()) + list(runs.values()))


@pytest.mark.parametrize("layers,height", [(1, None), (2, None), (48, 8)])
def test_slow_units_of_a_large_model_have_a_height_of_their_own(layers, height):
    """From PYLO_TC_ONE_LAUNCH items on FAST2D units on, the others have a launch that ends with its longest item."""
    fast, slow = [(1 + k, 768, 3072) for k in range(layers)], [(0, 768 * 768), (99, 130)]
    items = plan.apply_items(L.FAM_ADAFAC, True, fast, slow)
    gen = items["pad_"] >= L.TC_GEN_ITEM
    of_slow, of_fast = set((items["pad_"][gen] & 0xffff).tolist()), set(items["pad_"][~gen].tolist())
    assert len(of_slow) == len(of_fast) == 1
    assert ((~gen).sum() >= L.TC_ONE_LAUNCH) == (height is not None)
    assert of_slow == ({height} if height else of_fast)
    assert gen.sum() == sum(-(-n // (128 * min(of_slow))) for _, n in slow)


def test_packed_rows_give_every_sm_its_tiles():
    """Rows per thread of the packed sweep: the most that still leave sixteen tiles per SM (four below 32 rows)."""
    for X, Y in ((4096, 4096), (1024, 1024), (300, 260), (16, 8), (50257, 768)):
        rt, w, _ = plan.apply_tile_shape(L.FAM_VELO, X, Y)
        items = lambda k: -(-X // (rt * k // 16)) * -(-Y // w)
        enough = lambda k: items(k) >= (16 if k > 16 else 4) * L.SM_COUNT
        k = plan.packed_rows([(X, Y, rt, w)])
        assert k in (2, 4, 8, 16, 32, 64) and (k == 2 or enough(k)) and not any(enough(q) for q in (4, 8, 16, 32, 64) if q > k)


def test_mulo_groups_follow_the_infinite_width_shapes():
    """MuLO_cuda.py:32-60: matrix-like parameters are grouped by width multiplier with lr / width_mult, the others
    keep lr; checked on stand-ins for mup's ``infshape`` (the grouping needs nothing else of mup)."""
    from pylo_b200.optim.MuLO_cuda import mulo_param_groups

    class Inf:
        def __init__(self, n, w):
            self.n, self.w = n, w

        def ninf(self):
            return self.n

        def width_mult(self):
            return self.w

    def param(shape, n, w):
        p = torch.nn.Parameter(torch.zeros(shape))
        p.infshape = Inf(n, w)
        return p

    a, b, c, d = param((8, 8), 2, 4.0), param((8, 4), 2, 2.0), param((8,), 1, 1.0), param((4, 8), 2, 4.0)
    groups = mulo_param_groups([a, b, c, d], lr=0.5, weight_decay=0.1)
    by_lr = {g["lr"]: g["params"] for g in groups}
    assert set(by_lr) == {0.125, 0.25, 0.5}
    assert by_lr[0.125] == [a, d] and by_lr[0.25] == [b] and by_lr[0.5] == [c]
    assert all(g["weight_decay"] == 0.1 for g in groups)
    two = mulo_param_groups([{"params": [a], "lr": 1.0}, {"params": [c]}], lr=0.5)
    assert [g["lr"] for g in two if g["params"]] == [0.25, 0.5]
    with pytest.raises(AssertionError):
        mulo_param_groups([torch.nn.Parameter(torch.zeros(2, 2))])
    with pytest.raises(NotImplementedError):
        mulo_param_groups([param((2, 2, 2), 3, 1.0)])


def test_a_rank_without_tensors_still_gets_a_param_group():
    """The sharded drivers hang collectives on the optimizer's per-group hook; a rank that owns nothing must keep
    (empty) groups so that the hook still runs there."""
    from pylo_b200.zero import split_in_groups

    assert split_in_groups([], 4) == [{"params": []}]
    ps = [torch.zeros(4), torch.zeros(8), torch.zeros(4)]
    groups = split_in_groups(ps, 2)
    assert [len(g["params"]) for g in groups] == [2, 1]


def test_gradients_of_another_type_are_not_taken_by_their_address():
    """An fp32 parameter may have a bf16 gradient (``grad_dtype``); its address alone would be read as fp32, beyond its end."""
    full, half = torch.arange(8.0), torch.arange(8.0).to(torch.bfloat16)
    assert plan.grad_pointers([full, full]) == [full.data_ptr()] * 2
    assert plan.grad_pointers([full, half]) is None
    assert plan.grad_pointers([full.view(2, 4).t()]) is None
    # the same address with another type in it: not what it was
    assert plan.grad_pointers([full[:4].view(torch.int32)]) is None
    assert plan.fp32_gradient(full) is full
    got = plan.fp32_gradient(half)
    assert got.dtype == torch.float32 and torch.equal(got, full)
    strided = plan.fp32_gradient(full.view(2, 4).t())
    assert strided.is_contiguous() and torch.equal(strided, full.view(2, 4).t())


def test_a_tensor_learning_rate_that_a_scheduler_changes_in_place_is_seen():
    """torch's schedulers ``fill_`` a tensor learning rate: what a step keeps for comparison must be its value."""
    from pylo_b200.optim._common import group_floats

    p = torch.nn.Parameter(torch.zeros(3))
    opt = torch.optim.SGD([p], lr=torch.tensor(0.5), weight_decay=0.1)
    sched = torch.optim.lr_scheduler.ExponentialLR(opt, gamma=0.5)
    group = opt.param_groups[0]
    lr = group["lr"]
    kept = group_floats(group, "lr", "weight_decay")
    p.grad = torch.zeros(3)
    opt.step()
    sched.step()
    assert group["lr"] is lr, "the scheduler changes the tensor in place"
    assert kept == (0.5, 0.1) and group_floats(group, "lr", "weight_decay") == (0.25, 0.1)


@pytest.mark.parametrize("name", ["AdafacLO_CUDA", "ELO_CUDA", "CELO2_CUDA", "ELO_CELO2_CUDA", "VeLO_CUDA"])
def test_every_class_that_reports_a_timeout_can_be_cleared(name):
    from pylo_b200 import optim

    cls = getattr(optim, name)
    assert callable(cls.check_status) and callable(cls.clear_status)


def test_no_source_file_names_a_path_of_one_machine():
    """Where the reference checkout lies comes from an argument or PYLO_REFERENCE."""
    import os
    import re

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    paths = [os.path.join(root, name) for name in os.listdir(root)]
    for top in ("include", "oracle", "perf", "pylo_b200", "tests"):
        paths += [os.path.join(folder, name) for folder, _, files in os.walk(os.path.join(root, top)) for name in files]
    for path in paths:
        if path.endswith((".py", ".cu", ".cuh", ".h")):
            assert not re.search(r"/(root|home)/\w", open(path).read()), path


def test_small_models_are_dealt_to_clusters_that_hold_them():
    """Every share fits, all clusters run at once (or, with the fewest CTAs that hold the tensors, in two turns)."""
    cases = [([(128, 784), (128, 128), (10, 128)], [128, 128, 10]), ([(64, 64)] * 40, [13] * 30), ([(512, 256)], []), ([], [5]),
             ([(1, 4747)], []), ([(1, 4748)], []), ([(1, 8193)], []), ([(513, 256)], []), ([(4096, 4096)], []), ([(64, 64)] * 296, []), ([(64, 64)] * 297, [])]
    for mats, vectors in cases:
        got, T = plan.small_front(mats, vectors), len(mats) + len(vectors)
        up = lambda n: -(-n // 4) * 4
        fits = lambda cl: (all(-(-X // cl) * Y <= L.SMALL_SLICE for X, Y in mats) and all(-(-n // cl) <= L.SMALL_SLICE for n in vectors)
                           and 6 * up(max([-(-X // cl) * Y for X, Y in mats], default=0)) + 4 * up(max([-(-X // cl) for X, _ in mats], default=0))
                           + 5 * up(max([Y for _, Y in mats], default=0)) <= L.SMALL_FLOATS)
        if got is None:
            assert not any(fits(cl) and T * cl <= 2 * plan.SMALL_CTAS for cl in (1, 2, 4, 8, 16))
            continue
        cl, share, rows, cols = got
        assert cl in (1, 2, 4, 8, 16) and fits(cl)
        assert T * cl <= plan.SMALL_CTAS or not any(fits(c) for c in (1, 2, 4, 8) if c < cl)
    assert plan.small_front([(128, 784)], [10])[0] == 16 and plan.small_front([(64, 64)] * 40, [13] * 30)[0] == 2

    for sizes, k in (([1], 16), ([100352, 10, 7], 16), ([8192], 1)):
        tiles, ranges = plan.equal_tiles(sizes, k)
        for i, (n, (t0, m)) in enumerate(zip(sizes, ranges)):
            mine = tiles[t0:t0 + m]
            assert m == k and (mine["tensor"] == i).all() and (mine["elems"] % 4 == 0).all()
            assert int(np.clip(n - mine["start"], 0, mine["elems"]).sum()) == n


def test_a_rank_s_plan_takes_the_order_of_sums_of_the_whole_model():
    """What ShardedStep notes on the parameters, when the plan takes it, and that the order then does not depend on the share."""
    from pylo_b200.optim.AdafacLO_cuda import AdafacLO_CUDA

    shapes = ((96, 64), (64,), (8, 6, 5), (300, 260))
    params = [torch.nn.Parameter(torch.zeros(s)) for s in shapes]
    assert plan.model_shapes(params) is None
    zero._note_model(params)
    assert plan.model_shapes(params) == shapes and plan.model_shapes(params[2:]) == shapes
    assert plan.model_shapes(params[:1] + [torch.nn.Parameter(torch.zeros(7))]) is None      # a tensor without the note
    foreign = torch.nn.Parameter(torch.zeros(500, 500))
    foreign._pylo_model_shapes = shapes
    assert plan.model_shapes([foreign]) is None and plan.model_shapes([params[3], params[3]]) is None   # not of this model
    assert plan.model_shapes([]) is None

    def order(which):
        d = np.zeros(len(which), dtype=L.DESC_DTYPE)
        for row, s in zip(d, which):
            _, fd, axis = AdafacLO_CUDA._factoring(s)
            plan.fill_geometry(row, s, fd, axis)
        return plan.sum_order(L.FAM_ADAFAC, d, d["n"].tolist(), d["mode"], False)

    # the share alone would take the launch of small models, which the whole one does not: why the note is needed
    assert order(shapes[3:]).small and not order(shapes).small


# (stacks of one call, launches, which of them have a workspace): a chain is two launches and three a round
NS_ROUTES = [([(1, 512, 512), (1, 128, 512), (1, 1792, 512)], 17, (1, 1, 1)),
             ([(1, 512, 784), (1, 512, 512), (1, 100, 512)], 17, (1, 1, 1)),
             ([(12, 768, 768), (1, 50, 768), (4, 768, 3072), (1, 10, 128)], 18, (1, 1, 1, 0)),
             ([(1, 256, 256), (63, 128, 128)], 17, (1, 1)),
             ([(1, 256, 256), (40, 128, 128), (24, 128, 512)], 18, (1, 0, 0)),   # too many to ride: clusters, then the chain
             ([(1, 256, 256), (64, 128, 128), (1, 10, 128)], 18, (1, 0, 0)),     # which take a small matrix along
             ([(1, 128, 784), (1, 128, 128), (1, 10, 128)], 1, (0, 0, 0)),
             ([(1, 65, 64)], 1, (0,)), ([(2, 10, 128)], 1, (0,)), ([(1, 129, 129)], 17, (1,))]


@pytest.mark.parametrize("stacks,launches,spaces", NS_ROUTES, ids=[str(s[:2]) for s, _, _ in NS_ROUTES])
def test_small_matrices_ride_in_the_newton_schulz_launches_of_larger_ones(stacks, launches, spaces):
    """Up to 63 matrices that would fit a cluster add no launch to a call that has larger ones; without a workspace they do."""
    descs = K._ns_descs([torch.empty(s, device="meta") for s in stacks], 5)
    need = (ctypes.c_int64 * len(stacks))()
    assert L.lib.pylo_b200_newton_schulz_workspaces(descs, len(stacks), need) == 0
    assert tuple(int(b > 0) for b in need) == spaces
    for d, b in zip(descs, need):
        if b:
            d.work, d.work_bytes = 1 << 20, b
    assert L.lib.pylo_b200_newton_schulz_launches(descs, len(stacks)) == launches
    for d in descs:   # what a caller has that asks for every stack by itself
        d.work_bytes = L.lib.pylo_b200_newton_schulz_workspace(d.rows, d.cols, d.batch, d.iters)
        d.work = (1 << 20) if d.work_bytes else None
    small = any(b and not d.work_bytes for b, d in zip(need, descs))
    assert L.lib.pylo_b200_newton_schulz_launches(descs, len(stacks)) == launches + (small and not (10, 128) in [s[1:] for s in stacks])
    descs[0].rows = 0
    assert L.lib.pylo_b200_newton_schulz_workspaces(descs, len(stacks), need) == -1
