"""Calls of the C ABI that the sweeps' own assumptions do not cover are refused, or answered in full."""

import ctypes as C

from pylo_b200 import _lib as L


def test_scales_from_the_partials_need_the_variant_that_makes_them():
    """no_tables = 4 without generic would run on whatever the scales hold: refused on the host, before anything is launched."""
    prm, some = L.StepParams(), C.c_void_p(256)
    prm.family, prm.no_tables = L.FAM_ADAFAC, 4
    assert L.lib.pylo_b200_apply_adafac_tc(some, some, 1, 0, C.byref(prm), None, None, None) == -1
    assert L.lib.pylo_b200_apply_adafac_tc(some, some, 0, 1, C.byref(prm), None, None, None) == 0
