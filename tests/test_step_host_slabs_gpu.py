"""bx_step_host with more than two slabs of its pipeline where the smaller grids of
test_step_host_gpu.py have one or two (a slab holds 2^17 cells or 8 planes): ragged
grids with walls and pageable memory, dirty ghosts, a 2-D grid of two slabs.
Against the three calls and the oracle, bit for bit, with the slab count."""
import pytest

from boxzyhydro_b200.hydro import ghost_plan

from .helpers import small_random_box
from .test_step_host_gpu import run_pair

pytestmark = pytest.mark.gpu


def slabs(g, st):
    """The slab count of g's pipeline, from the timeline of one more call."""
    g.step_host_profile(True)
    g.step_host(st.cons.copy())
    n = g.step_host_timeline().shape[0]
    g.step_host_profile(False)
    return n


# count 0: walls that meet in a corner whose ghosts lag a sweep (no fused path, so no
# slabs: the call runs the three)
@pytest.mark.parametrize("dims,walls,count", [((37, 21, 53), (0, 1, 1, 0, 0, 1), 7),
                                              ((37, 21, 44), (1, 0, 0, 1, 1, 0), 0),
                                              ((14, 70, 31), (0,) * 6, 4)])
@pytest.mark.parametrize("pinned,in_place", [(False, False), (True, True)])
def test_ragged_grids(dims, walls, count, pinned, in_place):
    st = small_random_box(nx=dims[0], ny=dims[1], nz=dims[2], walls=walls, seed=21, dx=0.07)
    ga, gb = run_pair(st, 4, pinned=pinned, in_place=in_place)
    assert ga.status()[1] == ghost_plan(st.params)["fused_ok"] == (count > 0)
    if count:
        assert slabs(ga, st) == count
    ga.close()
    gb.close()


def test_dirty_ghosts():
    st = small_random_box(nx=20, ny=18, nz=36, walls=(0,) * 6, seed=23)
    st.cons[0, 4] *= 1.5  # a corner ghost
    ga, gb = run_pair(st, 3, pinned=True, in_place=True)
    assert ga.status() == gb.status()
    assert slabs(ga, st) == 4
    ga.close()
    gb.close()


def test_two_dimensional_grid_of_two_slabs():
    st = small_random_box(nx=515, ny=261, nz=4, walls=(0, 1, 1, 0, 0, 0), seed=22)
    ga, gb = run_pair(st, 3, pinned=True, in_place=False)
    assert ga.status()[1] == 1
    assert slabs(ga, st) == 2
    ga.close()
    gb.close()


@pytest.mark.parametrize("dims,count", [((132, 132, 20), 6), ((204, 100, 24), 7),
                                        ((204, 204, 9), 3)])
def test_flat_grids_have_thin_slabs(dims, count):
    """Few planes: thinner slabs than 8 planes or 2^17 cells, whose pipeline would be
    two or three slabs long."""
    st = small_random_box(nx=dims[0], ny=dims[1], nz=dims[2], walls=(0, 1, 1, 0, 0, 0), seed=24)
    ga, gb = run_pair(st, 2, pinned=True, in_place=True)
    assert ga.status()[1] == 1
    assert slabs(ga, st) == count
    ga.close()
    gb.close()
