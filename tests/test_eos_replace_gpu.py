"""A second set of EOS tables on a handle that has run chunks of steps with the first:
the graphs bx_run caches hold the tables' addresses and extents by value, so they go
with the tables.  Against the oracle given the same tables; tolerance: none."""
import dataclasses

import pytest

from tests.helpers import compare, make_pair, small_random_box, synthetic_eos_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,second", [((40, 9), (25, 8)), ((25, 8), (40, 9))])
def test_tables_replaced_between_runs(first, second):
    """70 steps (one on the per-phase kernels, two whole chunks, five steps), tables
    of other extents and values, 70 steps more from the same input planes."""
    st = small_random_box(nx=20, ny=18, nz=14, walls=(0,) * 6, seed=41)
    st.params = dataclasses.replace(st.params, h2stat=1)
    o, g = make_pair(st)
    for k, dims in enumerate((first, second)):
        tab = synthetic_eos_table(*dims, seed=k)
        o.set_eos_table(tab)
        g.set_eos_table(tab)
        assert o.run(nsteps=70) == 70 and g.run(nsteps=70) == 70
        assert g.status()[1] == 1, "expected the fused stage kernels"
        co, cg = o.clock(), g.clock()
        for key in ("time", "dt", "dtold", "step"):
            assert co[key] == cg[key], f"tables {k}: clock {key} {co[key]!r} vs {cg[key]!r}"
        compare(o, g, f"after the run with tables {k}")
    o.close()
    g.close()
