"""Workspace sizes follow from what a family's kernels read."""

from pylo_b200 import _lib as L


def test_the_folded_network_is_as_long_as_the_family_needs():
    """Units of CELO2 can be matrices of 3 x 3: only the AdafacLO family has the tensor cores' operands behind its network."""
    floats = {f: L.workspace_layout(f, L.MODE_VEC1D, 9).wfold for f in (L.FAM_ADAFAC, L.FAM_CELO2, L.FAM_VELO)}
    assert floats[L.FAM_ADAFAC] == L.WFOLD_STRIDE
    for family, hidden in ((L.FAM_CELO2, 8), (L.FAM_VELO, 4)):
        network = 30 * hidden + hidden + hidden * hidden + hidden + 2 * hidden + 2   # the two outputs that are used
        assert network + 30 <= floats[family] < 2 * network + 64
