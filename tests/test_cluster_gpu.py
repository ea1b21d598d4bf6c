"""The cluster solve (plan rows 5) computes the other plans' iterates: the
whole state after steps is equal bit for bit, in fixed and residual modes, at
the shapes where its units (2 x 1 x 4 cells) meet the walls, its shares meet
other CTAs, and a thread owns one to four units, and with more fluid units
than its shared memory holds."""
import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from scenes import ball_drop

pytestmark = pytest.mark.gpu

# size, pool depth, cluster widths
CASES = [
    ((16, 16, 16), 0.3, (1, 2, 16)),    # one CTA; shares thinner than a plane
    ((17, 13, 21), 0.5, (1, 16)),       # odd sx: half a unit beyond the wall; sz % 4 == 1
    ((9, 8, 14), 0.6, (1, 4)),          # sz % 4 == 2
    ((5, 4, 7), 0.9, (1, 16)),          # sz % 4 == 3; CTAs without a unit
    ((4, 4, 4), 0.9, (1, 8)),           # the smallest grid
    ((50, 50, 50), 0.2, (8, 16)),       # one and two units a thread
    ((64, 24, 64), 0.9, (8, 16)),       # three and two units a thread, full rows
    ((48, 40, 64), 0.9, (16, 4)),       # two units a thread; four CTAs: through global memory
    ((32, 32, 32), 0.8, (1, 2)),        # through global memory; four units a thread
    ((30, 33, 26), 0.9, (1,)),          # through global memory, ragged
]
MODES = {
    "fixed": dict(pressure_iterations=37),
    "residual": dict(solve_mode=_abi.SOLVE_RESIDUAL, pressure_init=_abi.PRESSURE_ZERO, rel_residual=1e-3,
                     max_iterations=120, check_interval=20),
}


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("size,pool,widths", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_cluster_solve_equals_one_sweep_per_launch(size, pool, widths, mode):
    def fluid(plan):
        f = aq.Fluid(ball_drop(size, pool=pool, center=(0.5, 0.7, 0.5), radius=0.15, **MODES[mode]))
        f.set_jacobi_plan(*plan)
        f.step(3)
        return f
    with fluid((1, 0, 1) if size[2] % 4 == 0 else (2, 16, 16)) as f:
        want, stats = f.download_state(), f.solve_stats()
    for w in widths:
        with fluid((1, 5, w)) as f:
            got, s = f.download_state(), f.solve_stats()
        for k in want:
            if k != "physical_time":
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k}, {w} CTAs")
        assert s["iterations"] == stats["iterations"] and s["fluid_cells"] == stats["fluid_cells"]
        # the same FP64 terms in another order: under 1e5 of them, each sum within n * 2^-53
        assert abs(s["rel_residual"] - stats["rel_residual"]) <= 1e5 * 2.0 ** -53 * stats["rel_residual"]


def test_cluster_solve_without_fluid():
    with aq.Fluid(_abi.make_config((16, 12, 10), [], **MODES["residual"])) as f:
        assert f.jacobi_plan()[1] == 5
        f.step(2)
        s = f.solve_stats()
        assert s["converged"] and s["iterations"] == 20 and s["rel_residual"] == 0.0


def test_cluster_solve_writes_zeros_as_the_sweeps_do():
    """Cells without fluid beside fluid ones hold +0 after a solve, whatever the
    sign of the sums around them: bit patterns, not values, are compared."""
    def pressure(plan):
        with aq.Fluid(ball_drop((24, 20, 28), pool=0.4, pressure_iterations=30)) as f:
            f.set_jacobi_plan(*plan)
            f.step(4)
            return f.download_state(["pressure"])["pressure"]
    want = pressure((1, 3, 1))
    assert (want < 0).any()
    np.testing.assert_array_equal(pressure((1, 5, 16)).view(np.uint32), want.view(np.uint32))
