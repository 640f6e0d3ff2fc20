"""The tiled stage kernels (and the per-phase flux on them) at the edges of their
tiles, against the oracle.

Interior sizes of one cell, one short of, at and one beyond a tile's columns (32 x 8;
32 x 6 with flux_ang) and of a z chunk, with and without walls and with a cell
size that is and is not a power of two: cons, u, p and the clock after every step.
Tolerance: none (every operation rounds as the oracle's does)."""
import dataclasses

import numpy as np
import pytest

from boxzyhydro_b200.hydro import ghost_plan
from tests.helpers import make_pair, small_random_box, step_both

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 2), (2, 8, 3), (31, 9, 2), (33, 7, 5), (32, 8, 2), (65, 17, 3), (64, 1, 2),
         (3, 41, 9), (75, 61, 47)]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("walls,dx", [((0,) * 6, 1.0 / 16), ((0, 1, 1, 0, 0, 1), 0.07)])
def test_tile_edges_3d(n, walls, dx):
    st = small_random_box(nx=n[0] + 4, ny=n[1] + 4, nz=n[2] + 4, walls=walls, dx=dx,
                          seed=sum(n))
    o, g = make_pair(st)
    step_both(o, g, 4)
    # one-cell axes with a mirror wall lie off the stage kernels' ghost rule
    assert g.status()[1] == ghost_plan(st.params)["fused_ok"]
    o.close()
    g.close()


@pytest.mark.parametrize("n", [(1, 1, 1), (33, 9, 2), (32, 8, 1), (5, 200, 1)])
def test_tile_edges_2d(n):
    st = small_random_box(nx=n[0] + 4, ny=n[1] + 4, nz=n[2], walls=(1,) * 6, dx=0.02, seed=3)
    o, g = make_pair(st)
    step_both(o, g, 4)
    # one-cell axes with a mirror wall lie off the stage kernels' ghost rule
    assert g.status()[1] == ghost_plan(st.params)["fused_ok"]
    o.close()
    g.close()


@pytest.mark.parametrize("n", [(2, 6, 3), (32, 7, 2), (34, 13, 4)])
def test_tile_edges_with_flux_ang(n):
    st = small_random_box(nx=n[0] + 4, ny=n[1] + 4, nz=n[2] + 4, seed=5)
    st.params = dataclasses.replace(st.params, fluxangmom=True, yoffset=3.0)
    o, g = make_pair(st)
    step_both(o, g, 4)
    assert g.status()[1] == 1 and np.isfinite(g.download()[0]).all()
    o.close()
    g.close()


@pytest.mark.parametrize("n", [(1, 1, 2), (33, 9, 3), (32, 8, 2), (65, 7, 9), (33, 9, 2), (5, 17, 1)])
@pytest.mark.parametrize("walls,dx", [((1,) * 6, 1.0 / 16), ((0, 1, 1, 0, 0, 1), 0.07)])
def test_tile_edges_per_phase(n, walls, dx):
    """The per-phase path's flux on the same tiles, on the reference's arrays."""
    nz = n[2] + 4 if n[2] > 1 else 1
    st = small_random_box(nx=n[0] + 4, ny=n[1] + 4, nz=nz, walls=walls, dx=dx, seed=2 + sum(n))
    o, g = make_pair(st, phase_only=True)
    step_both(o, g, 3)
    assert g.status()[1] == 0
    o.close()
    g.close()


@pytest.mark.parametrize("phase_only", [False, True])
@pytest.mark.parametrize("n", [(8, 1, 1), (32, 32, 32), (75, 61, 47)])
def test_dependent_launches(n, phase_only):
    """Launches that start before the one ahead of them is through (a run's, and single
    steps') against launches with events between them, and the oracle."""
    nz = n[2] + 4 if n[2] > 1 else 1
    st = small_random_box(nx=n[0] + 4, ny=n[1] + 4, nz=nz, seed=7)
    o, g = make_pair(st, phase_only=phase_only)
    step_both(o, g, 12)
    other = make_pair(st, phase_only=phase_only)
    timed = other[1]
    for k in range(12):
        timed.profile(k % 2 == 0)
        timed.step()
    run = make_pair(st, phase_only=phase_only)
    run[1].run(nsteps=12)
    want = g.download()[0]
    assert np.array_equal(want, timed.download()[0]) and np.array_equal(want, run[1].download()[0])
    for x in (o, g, *other, *run):
        x.close()
