"""Multiphase runs: the per-phase concentration mass (sum of the particles'
volume fractions, FP64) against the CPU oracle's, and the single-phase case
(the particle count).  The change of this sum over a run is the
concentration-mass conservation error of multiphase diffusion."""
import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from oracle_binding import Oracle
from scenes import SCENES, ball_drop, rel_l2

pytestmark = pytest.mark.gpu


def test_phase_mass_matches_oracle_fractions():
    cfg = SCENES["multi_16"]()
    f, o = aq.Fluid(cfg), Oracle(cfg)
    for _ in range(3):
        f.step(1)
        o.step(1)
        m = np.array(f.phase_mass())
        fr = o.get_state(["fractions"])["fractions"].reshape(4, -1).astype(np.float64)
        np.testing.assert_allclose(m, fr.sum(axis=1), rtol=1e-5, atol=1e-3)
    assert abs(sum(m) - f.particleCount) <= 1e-3 * f.particleCount  # fractions are normalised
    f.close()


def test_single_phase_mass_is_the_particle_count():
    cfg = SCENES["cfg1_16"]()
    with aq.Fluid(cfg) as f:
        f.step(2)
        m = f.phase_mass()
        assert m[cfg.volumes[0].phase] == f.particleCount and sum(m) == f.particleCount


@pytest.mark.parametrize("size", [(16, 16, 16), (21, 19, 37), (40, 9, 65)])
@pytest.mark.parametrize("tiny", [0.25, 1e-20, 1e-33])
def test_diffusion_sweeps_match_oracle(size, tiny):
    """Ragged tiles, and a second phase of ordinary fractions, of fractions
    small enough to check the range of the shared-divisor division and of ones
    below it (the IEEE division).  A sweep rounds at most 10 times in a chain,
    so 21 sweeps differ by at most 210 half-ulps (1.3e-5) however the
    multiplications and additions are contracted."""
    cfg = ball_drop(size, pool=0.4, phase_ball=1, diffusion_coeff=0.01, diffusion_iterations=21)
    with aq.Fluid(cfg) as f:
        f.step(1)
        st = f.download_state()
        rng = np.random.default_rng(5)
        fr = np.zeros_like(st["fractions"]).reshape(4, -1)
        fr[1] = tiny * rng.uniform(0.0, 1.0, fr.shape[1]) * (rng.uniform(size=fr.shape[1]) < 0.5)
        fr[0] = 1.0 - fr[1]
        st = dict(st, fractions=fr.reshape(st["fractions"].shape).astype(np.float32))
        o = Oracle(cfg)
        got = want = None
        f.upload_state(st)
        o.set_state(st)
        for stage in (_abi.STAGE_P2G, _abi.STAGE_DIFFUSE):
            f.run_stage(stage)
            o.stage(stage)
        got = f.download_state(["new_volume_fractions"])["new_volume_fractions"].reshape(4, -1)
        want = o.get_state(["new_volume_fractions"])["new_volume_fractions"].reshape(4, -1)
        o.close()
    for k in range(2):
        assert np.any(want[k] > 0)
        assert rel_l2(got[k], want[k]) <= 1.3e-5, k
    assert not np.any(got[2:]) and not np.any(want[2:])
