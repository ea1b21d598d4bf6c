"""Fluids that outgrow the cluster they are solved in: particles strewn over the
whole grid touch more units of 2 x 1 x 4 cells than the cluster's shared memory
holds.  The state stays that of the sweeps over the whole machine, bit for bit,
in graphs (whole and split for host steps) and outside of them, and a step takes
no longer than with those sweeps; a scene of a batch, which is solved in a wider
cluster or by the row sweeps then, stays the scene alone."""
import time

import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from scenes import ball_drop

pytestmark = pytest.mark.gpu

FIELDS = ["position", "velocity_p", "new_velocity", "pressure", "particle_count_cell"]
MODES = {
    "fixed": dict(pressure_iterations=37),
    "residual": dict(solve_mode=_abi.SOLVE_RESIDUAL, pressure_init=_abi.PRESSURE_ZERO, rel_residual=1e-3,
                     max_iterations=120, check_interval=20),
}


def _strewn(n, size, seed):
    rng = np.random.default_rng(seed)
    ext = np.array(size, np.float32)[:, None] * np.float32(10.0 / size[1])
    return ((0.02 + 0.96 * rng.random((3, n))) * ext).astype(np.float32)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("size,wide", [((96, 64, 96), (1, 3, 1)), ((90, 61, 75), (2, 16, 16))])
def test_strewn_fluid_is_solved_by_the_machine_wide_sweeps(size, wide, mode):
    def fluid(plan):
        f = aq.Fluid(ball_drop(size, pool=0.2, dt=0.001, **MODES[mode]))
        if plan is None:
            assert f.jacobi_plan() == (1, 5, 16)
        else:
            f.set_jacobi_plan(*plan)
        return f

    def timed(f):
        f.step(2)
        f.synchronize()
        best = np.inf
        for _ in range(3):
            t = time.perf_counter()
            f.step(4)
            f.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    pos = None
    out, stats, secs = [], [], []
    for plan, graph in ((wide, True), (None, True), (None, False)):
        with fluid(plan) as f:
            n = f.particleCount
            pos = _strewn(n, size, 5) if pos is None else pos
            vel = np.zeros((3, n), np.float32)
            f.set_graph_mode(graph)
            f.step(1)  # the pool: held by the cluster
            f.step_host(1, pos, vel, np.empty_like(pos), vel)
            f.step(2)
            out.append(f.download_state(FIELDS))
            stats.append(f.solve_stats())
            if graph:
                secs.append(timed(f))
    cells = (out[0]["particle_count_cell"].reshape(size) > 0).astype(int)
    units = (np.add.reduceat(np.add.reduceat(cells, range(0, size[0], 2), 0), range(0, size[2], 4), 2) > 0).sum()
    assert units > 16 * 2048
    for got, s in zip(out[1:], stats[1:]):
        for k in FIELDS:
            np.testing.assert_array_equal(got[k], out[0][k], err_msg=k)
        assert s == stats[0]
    # one conditional node a step apart
    assert secs[1] <= 1.5 * secs[0]


def test_stages_solve_a_pool_in_the_cluster():
    """Outside of a step's graph too: the pressure stage of a fluid that its
    cluster holds takes less than the tiled sweeps' (some 0.2 of it)."""
    def stage(plan):
        with aq.Fluid(ball_drop((90, 61, 75), pool=0.2, dt=0.001, pressure_iterations=200)) as f:
            if plan is not None:
                f.set_jacobi_plan(*plan)
            f.step(2)
            return min(f.profile_step()["pressure"] for _ in range(5))
    assert stage(None) < 0.7 * stage((2, 16, 16))


@pytest.mark.parametrize("mode", MODES)
def test_strewn_scenes_of_a_batch_stay_the_scenes_alone(mode):
    sizes = [(16, 16, 16), (32, 32, 32), (96, 64, 96), (24, 32, 48)]  # 32^3: a wider cluster; 96 x 64 x 96: row sweeps
    cfgs = [ball_drop(s, pool=0.2, dt=0.001, **MODES[mode]) for s in sizes]
    with aq.Batch(cfgs) as b:
        counts = list(b.particle_counts)
        pos = np.concatenate([_strewn(n, s, i) for i, (n, s) in enumerate(zip(counts, sizes))], 1)
        vel = np.zeros_like(pos)
        b.step(1)
        b.step_host(1, pos, vel, np.empty_like(pos), vel)
        b.step(2)
        at = 0
        for i, c in enumerate(cfgs):
            with aq.Fluid(c) as f:
                p = np.ascontiguousarray(pos[:, at:at + counts[i]])
                v = np.zeros_like(p)
                f.step(1)
                f.step_host(1, p, v, np.empty_like(p), v)
                f.step(2)
                want, got = f.download_state(FIELDS), b.download_scene(i, FIELDS)
                for k in FIELDS:
                    np.testing.assert_array_equal(got[k], want[k], err_msg=f"scene {i} {k}")
                sa, sb = b.solve_stats(i), f.solve_stats()
                for k in ("iterations", "rel_residual", "fluid_cells", "blocks", "total_sweeps", "total_blocks"):
                    assert sa[k] == sb[k], (i, k)
            at += counts[i]
