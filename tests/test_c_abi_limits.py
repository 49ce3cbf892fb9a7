"""Calls of the C ABI that the sweeps' own assumptions do not cover are refused, or answered in full."""

import ctypes as C

import numpy as np
import pytest
import torch

from pylo_b200 import _lib as L


def test_scales_from_the_partials_need_the_variant_that_makes_them():
    """no_tables = 4 without generic would run on whatever the scales hold: refused on the host, before anything is launched."""
    prm, some = L.StepParams(), C.c_void_p(256)
    prm.family, prm.no_tables = L.FAM_ADAFAC, 4
    assert L.lib.pylo_b200_apply_adafac_tc(some, some, 1, 0, C.byref(prm), None, None, None) == -1
    assert L.lib.pylo_b200_apply_adafac_tc(some, some, 0, 1, C.byref(prm), None, None, None) == 0


def _tensors(n_tiles, device):
    gen = torch.Generator(device=device).manual_seed(3)
    part = torch.rand(len(n_tiles), max(n_tiles), L.STAT_STRIDE, device=device, generator=gen)
    closed, sums = torch.zeros(len(n_tiles), L.STAT_STRIDE, device=device), torch.zeros(len(n_tiles), L.SUMS_STRIDE, device=device)
    d = np.zeros(len(n_tiles), dtype=L.DESC_DTYPE)
    for i, k in enumerate(n_tiles):
        d["n"][i], d["n_tiles"][i] = 1000 * k, k
        d["tile_part"][i], d["closed"][i], d["sums"][i] = part[i].data_ptr(), closed[i].data_ptr(), sums[i].data_ptr()
    table = torch.from_numpy(d.view(np.uint8).copy()).to(device)
    return table, (part, closed, sums)


@pytest.mark.gpu
@pytest.mark.parametrize("n_tiles", [[1, 16], [17, 3, 20], [15, 40, 1, 33]])
def test_velo_inputs_add_up_all_tiles(n_tiles):
    dev, T, H = torch.device("cuda"), len(n_tiles), 128
    table, keep = _tensors(n_tiles, dev)
    gen = torch.Generator(device=dev).manual_seed(4)
    rank = torch.rand(T, 5, device=dev, generator=gen)
    w = {k: torch.randn(*s, device=dev, generator=gen) for k, s in dict(mix2_w=(H, 30), mix2_b=(H,), fmix_w=(H, 30), fmix_b=(H,)).items()}
    x_in, xmix = torch.zeros(T, 30, device=dev), torch.zeros(T, H, device=dev)
    r = L.VeloRnn(T=T, H=H, B=256, x_in=x_in.data_ptr(), xmix=xmix.data_ptr(), **{k: v.data_ptr() for k, v in w.items()})
    buf = dict(means=torch.rand(10, device=dev), iteration=torch.ones(1, dtype=torch.int32, device=dev), running_min=torch.rand(10, device=dev),
               decays=torch.full((10,), 0.9, device=dev))
    loss = L.VeloLoss(value=1.5, **{k: v.data_ptr() for k, v in buf.items()})
    stream = torch.cuda.current_stream().cuda_stream
    L.check(L.lib.pylo_b200_velo_inputs(table.data_ptr(), None, rank.data_ptr(), 0.25, C.byref(loss), C.byref(r), stream), "velo_inputs")
    got = x_in.clone()
    L.check(L.lib.pylo_b200_velo_tensor_features(table.data_ptr(), T, None, T, rank.data_ptr(), 0.25, C.byref(loss), x_in.data_ptr(), stream), "features")
    assert torch.allclose(got, x_in, rtol=1e-6, atol=1e-7)
    del keep
