"""The choice among the ring kernel's launch variants, with scripted times: the
fastest is found whichever single launch something else disturbs."""
import ctypes as C

import numpy as np
import pytest

from abhsf_b200 import capi


def _pick(s, ms, disturbed):
    layout, bulk = C.c_int32(-1), C.c_int32(-1)
    n = capi.lib.abhsf_test_pick_variant(s, (C.c_float * 8)(*ms), disturbed, C.byref(layout), C.byref(bulk))
    return n, 2 * layout.value + bulk.value


@pytest.mark.parametrize("s", [32, 64])
def test_a_disturbed_launch_costs_no_variant_its_place(s):
    kinds = 6 if s == 32 else 8
    for seed in range(20):
        ms = np.random.default_rng(seed).uniform(0.1, 0.14, 8)
        best = int(np.argmin(ms[:kinds]))
        launches, got = _pick(s, ms, -1)
        assert got == best and launches == 2 * kinds + 9
        for d in range(launches):
            assert _pick(s, ms, d) == (launches, best)
