"""With bx_profile on, every launch of a step is an ordinary one, on the fused stages and on
the per-phase kernels: no kernel starts before the one ahead of it in the stream is
through (test_dependent_launches compares such steps with dependent launches)."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from boxzyhydro_b200.hydro import Hydro
from tests.helpers import small_random_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phase_only,launches", [(False, 4), (True, 22)])
def test_profiled_steps_run_one_kernel_at_a_time(phase_only, launches):
    torch.zeros(1, device="cuda")
    st = small_random_box(nx=52, ny=52, nz=52, seed=7)
    g = Hydro(st.params, phase_only=phase_only)
    g.upload(st.cons, st.u, st.p)
    for _ in range(2):
        g.step()
    assert g.status()[1] == (0 if phase_only else 1)
    g.profile(True)
    g.step()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as pr:
        for _ in range(2):
            g.step()
    g.close()
    k = sorted((e.time_range.start, e.time_range.end, e.name) for e in pr.events()
               if e.device_type == torch.autograd.DeviceType.CUDA and "bx::" in e.name)
    if not k:
        pytest.skip("the profiler records no kernels here")
    assert len(k) == 2 * launches
    early = [(a[2], b[2]) for a, b in zip(k, k[1:]) if b[0] < a[1]]
    assert not early, early
