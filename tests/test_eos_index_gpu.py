"""The tabulated EOS's table index from the single-precision logarithm equals the
one from the double-precision logarithm, on and next to the steps' edges, for
coarse and fine steps and for energies and densities far from one."""
import ctypes as C

import pytest

from boxzyhydro_b200 import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("low,step,steps", [(-9.0, 0.5, 9), (-24.0, 0.05, 600),
                                            (-0.96, 0.052, 40), (11.0, 0.002, 1000)])
def test_index_at_the_edges(low, step, steps):
    bad, ex = C.c_ulonglong(), C.c_double()
    rc = _lib.lib().bx_check_log_steps(20_000_000, 7, low, step, steps, C.byref(bad),
                                       C.byref(ex))
    assert rc == 0
    assert bad.value == 0, f"{bad.value} mismatches, e.g. x = {ex.value!r}"
