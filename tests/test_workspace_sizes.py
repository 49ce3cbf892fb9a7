"""Workspace sizes follow from what a family's kernels read."""

import pytest
import torch

from pylo_b200 import _lib as L
from pylo_b200 import models, optim


def test_the_folded_network_is_as_long_as_the_family_needs():
    """Units of CELO2 can be matrices of 3 x 3: only the AdafacLO family has the tensor cores' operands behind its network."""
    floats = {f: L.workspace_layout(f, L.MODE_VEC1D, 9).wfold for f in (L.FAM_ADAFAC, L.FAM_CELO2, L.FAM_VELO)}
    assert floats[L.FAM_ADAFAC] == L.WFOLD_STRIDE
    for family, hidden in ((L.FAM_CELO2, 8), (L.FAM_VELO, 4)):
        network = 30 * hidden + hidden + hidden * hidden + hidden + 2 * hidden + 2   # the two outputs that are used
        assert network + 30 <= floats[family] < 2 * network + 64


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["3xtf32", "fp32"])
def test_tables_only_where_a_sweep_reads_them(precision):
    p = torch.nn.Parameter(torch.zeros(600, 260, device="cuda"))
    p.grad = torch.ones_like(p)
    opt = optim.AdafacLO_CUDA([p], network=models.MetaMLP(39, 32, 1), mlp_precision=precision)
    opt.step()
    (_, plan), = opt._plans.values()
    tables = [bool(plan.tdesc.host[f][0]) for f in ("h_a", "h_b")]
    assert tables == [precision == "fp32"] * 2
