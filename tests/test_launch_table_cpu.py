"""The SOR variant that the library picks by launch size, where a limit lies at a
number of teams that the device holds."""
import ctypes as C
import os

import pytest

from gpg import lib as gpglib


@pytest.mark.parametrize("npatch,variant", [(1, 14), (75, 14), (148, 14), (256, 14), (296, 14), (297, 10), (4096, 10)])
def test_fp64_ghost4(npatch, variant):
    # one staged patch per team, two teams per SM of 148
    if not os.path.exists(gpglib.LIB_PATH):
        pytest.skip("library not built")
    v = C.c_int()
    gpglib.check(gpglib.library().gpg_sor_variant_for_launch(8, 4, npatch, C.byref(v)))
    assert v.value == variant
