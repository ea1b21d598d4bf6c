"""Host steps copy the particles out beside the last step's solve when there
is more than a megabyte of them: positions, velocities and the whole state
equal those of plain steps, for fluids and batches, with one and several steps
a call, repeated calls, and either output missing."""
import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from aquarius_b200.scenes import batch_configs
from scenes import ball_drop

pytestmark = pytest.mark.gpu

FIELDS = ["position", "velocity_p", "new_velocity", "pressure", "cell_start"]


@pytest.mark.parametrize("size", [(12, 12, 12), (40, 36, 42)])  # below and above a megabyte
@pytest.mark.parametrize("solver", [dict(pressure_iterations=30), dict(
    solve_mode=_abi.SOLVE_RESIDUAL, rel_residual=1e-3, max_iterations=80, check_interval=20)])
def test_fluid_host_steps_equal_steps(size, solver):
    cfg = ball_drop(size, pool=0.5, **solver)
    with aq.Fluid(cfg) as a, aq.Fluid(cfg) as b:
        n = a.particleCount
        assert (24 * n >= 1 << 20) == (size[0] > 12)
        pos, vel = np.empty((3, n), np.float32), np.empty((3, n), np.float32)
        for steps, p, v in ((1, pos, vel), (3, pos, None), (2, None, vel), (1, pos, vel)):
            a.step_host(steps, None, None, p, v)
            b.step(steps)
            want = b.download_state(FIELDS)
            if p is not None:
                np.testing.assert_array_equal(p, want["position"])
            if v is not None:
                np.testing.assert_array_equal(v, want["velocity_p"])
        got = a.download_state(FIELDS)
        for k in FIELDS:
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
        # in and out through the same buffers
        a.step_host(1, pos, vel, pos, vel)
        b.step(1)
        np.testing.assert_array_equal(pos, b.download_state(["position"])["position"])


@pytest.mark.parametrize("sizes", [(8, 12), (32,)])
def test_batch_host_steps_equal_steps(sizes):
    cfgs = batch_configs(4, seed=2, sizes=sizes, check_interval=20, max_iterations=80, rel_residual=1e-3)
    with aq.Batch(cfgs) as a, aq.Batch(cfgs) as b:
        n = sum(a.particle_counts)
        assert (24 * n >= 1 << 20) == (sizes == (32,))
        pos, vel = np.empty((3, n), np.float32), np.empty((3, n), np.float32)
        for steps in (1, 2):
            a.step_host(steps, None, None, pos, vel)
            b.step(steps)
        at = 0
        for s in range(4):
            want, got = b.download_scene(s, FIELDS), a.download_scene(s, FIELDS)
            for k in FIELDS:
                np.testing.assert_array_equal(got[k], want[k], err_msg=k)
            m = a.particle_counts[s]
            np.testing.assert_array_equal(pos[:, at:at + m], want["position"])
            np.testing.assert_array_equal(vel[:, at:at + m], want["velocity_p"])
            at += m


def test_launch_counts_after_host_steps_alone():
    cfg = ball_drop((40, 36, 42), pool=0.5, pressure_iterations=30)
    with aq.Fluid(cfg) as a, aq.Fluid(cfg) as b:
        pos = np.empty((3, a.particleCount), np.float32)
        a.step_host(1, None, None, pos, None)
        b.step(1)
        assert a.launch_counts() == b.launch_counts() != (0, 0)
        assert a.launches_per_step() == b.launches_per_step()
