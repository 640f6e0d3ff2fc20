"""flux(avg) on arrays whose outer ghost layer holds no numbers, against the oracle.

A ghost cell's slopes are zero whatever lies beyond it (flux.f90:53-57), so the outer
of the two ghost layers enters no interior cell's fluxes: NaN, infinities and the
largest finite values there must leave the result as it is.  Tolerance: none."""
import numpy as np
import pytest

from boxzyhydro_b200 import grid as G
from tests.helpers import compare, make_pair, small_random_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("junk", [np.nan, np.inf, -np.inf, 1.7e308])
@pytest.mark.parametrize("nx,ny,nz,dx", [(39, 21, 13, 1.0 / 16), (14, 12, 10, 0.07),
                                         (37, 13, 2, 1.0 / 16), (9, 21, 1, 0.07)])
@pytest.mark.parametrize("avg", [0, 1])
def test_flux_does_not_read_the_outer_layer(nx, ny, nz, dx, junk, avg):
    st = small_random_box(nx=nx, ny=ny, nz=nz, dx=dx, seed=nx + nz)
    outer = G.boundary_flags(nx, ny, nz) == 1
    c, u, p = st.cons.copy(), st.u.copy(), st.p.copy()
    c[outer, 4] = u[outer] = p[outer] = junk
    st.cons, st.u, st.p = c, u, p
    o, g = make_pair(st)
    o.save_cons_old()
    g.save_cons_old()
    o.set_clock(dt=0.002)
    g.set_dt(0.002)
    o.flux(avg)
    g.flux(avg)
    assert np.isfinite(g.download()[0]).all()
    compare(o, g, f"flux({avg}), outer ghosts {junk}", u_and_p=False)
    o.close()
    g.close()
