"""The shared-memory staged particle-to-grid kernel (the default) against the
one-thread-per-node L1 gather: the same terms summed in the same
(dx, dy, dz, j) order (transferToCellAccumPhase, Fluid/Fluid_3D_FLIP.cu:8-70),
so every P2G output must be bit for bit the same, including cells holding
more particles than the staged slots (the rest are read from global memory),
multiphase fractions and the transfer without forces at init; and the stage
still matches the CPU oracle."""
import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from oracle_binding import Oracle
from scenes import SCENES, ball_drop, rel_l2

pytestmark = pytest.mark.gpu

P2G_FIELDS = ["content", "velocity", "new_velocity", "density", "volume_fractions", "new_volume_fractions"]


def _variant(v):
    assert aq.load_library().aq_p2g_set_variant(v) == 0


def _p2g(cfg, state):
    with aq.Fluid(cfg) as f:
        f.upload_state(state)
        f.run_stage(_abi.STAGE_P2G)
        return f.download_state(P2G_FIELDS)


def _state(cfg, steps):
    with aq.Fluid(cfg) as f:
        f.step(steps)
        f.synchronize()
        return f.download_state()


@pytest.mark.parametrize("scene,steps", [("cfg2_32", 3), ("aniso", 2), ("multi_16", 2), ("cfg1_24", 0)])
def test_staged_p2g_equals_l1_gather(scene, steps):
    cfg = SCENES[scene]()
    st = _state(cfg, steps)
    try:
        _variant(0)
        a = _p2g(cfg, st)
        _variant(1)
        b = _p2g(cfg, st)
    finally:
        _variant(1)
    for k in P2G_FIELDS:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


def test_staged_p2g_overflowing_cells_and_init_transfer():
    """Crowd 40 particles into one cell and 13 into another (more than the
    staged slots), then compare the kernels; the fluid's init runs the
    transfer without forces with the staged kernel."""
    cfg = SCENES["cfg2_32"]()
    st = _state(cfg, 1)
    pos = st["position"].copy()
    h = cfg.domain_size / cfg.size_y
    n = pos.shape[1]
    rng = np.random.default_rng(3)
    for first, count, cell in ((0, 40, (10, 3, 12)), (100, 13, (20, 4, 7))):
        for k in range(3):
            pos[k, first:first + count] = (cell[k] + rng.uniform(0.05, 0.95, count)) * h
    st = dict(st, position=pos)
    with aq.Fluid(cfg) as f:  # re-sort so the crowded cells' particles are contiguous
        f.upload_state(st)
        f.run_stage(_abi.STAGE_SORT)
        sorted_state = f.download_state()
    try:
        _variant(0)
        a = _p2g(cfg, sorted_state)
        for v in (2, 3, 1):
            _variant(v)
            b = _p2g(cfg, sorted_state)
            for k in P2G_FIELDS:
                np.testing.assert_array_equal(b[k], a[k], err_msg=f"{v} {k}")
    finally:
        _variant(1)
    counts = np.bincount(sorted_state["particle_hash"], minlength=cfg.size_x * cfg.size_y * cfg.size_z)
    assert counts.max() >= 40 and (counts > 12).sum() >= 2
    # against the oracle too
    o = Oracle(cfg)
    o.set_state(sorted_state)
    o.stage(_abi.STAGE_P2G)
    want = o.get_state(P2G_FIELDS)
    for k in ("velocity", "new_velocity", "density"):
        assert rel_l2(b[k], want[k]) <= 1e-5, k
    np.testing.assert_array_equal(b["content"], want["content"])
    o.close()
    assert n > 200


@pytest.mark.parametrize("size,multi", [((48, 64, 70), False), ((67, 83, 65), False), ((67, 83, 65), True),
                                        ((33, 130, 129), False), ((81, 95, 97), True)])
def test_staged_p2g_chunks_of_planes(size, multi):
    """Grids large enough for 2, 3, 4 and 5 x planes to a CTA, with ragged last
    chunks, rows and columns."""
    cfg = ball_drop(size, pool=0.25, center=(0.5, 0.7, 0.5), radius=0.12, dt=0.005, phase_ball=1 if multi else 0,
                    pressure_iterations=20)
    st = _state(cfg, 1)
    try:
        _variant(0)
        a = _p2g(cfg, st)
        _variant(1)
        b = _p2g(cfg, st)
    finally:
        _variant(1)
    for k in P2G_FIELDS:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


@pytest.mark.parametrize("multi", [False, True])
@pytest.mark.parametrize("size", [(37, 29, 30), (38, 29, 30), (40, 40, 40)])
def test_staged_p2g_at_the_line_of_the_small_grids(size, multi):
    """148 CTAs of 8 rows, which take the small grids' kernel, four more, which
    march in chunks of one plane, and crowded cells in both."""
    cfg = ball_drop(size, pool=0.3, center=(0.5, 0.7, 0.5), radius=0.15, dt=0.005, phase_ball=1 if multi else 0,
                    pressure_iterations=20)
    st = _state(cfg, 1)
    pos = st["position"].copy()
    h = cfg.domain_size / cfg.size_y
    rng = np.random.default_rng(1)
    for first, count, cell in ((0, 40, (10, 3, 12)), (100, 13, (size[0] - 1, 0, size[2] - 1))):
        for k in range(3):
            pos[k, first:first + count] = (cell[k] + rng.uniform(0.05, 0.95, count)) * h
    with aq.Fluid(cfg) as f:
        f.upload_state(dict(st, position=pos))
        f.run_stage(_abi.STAGE_SORT)
        st = f.download_state()
    try:
        _variant(0)
        a = _p2g(cfg, st)
        for v in (2, 3, 1):
            _variant(v)
            b = _p2g(cfg, st)
            for k in P2G_FIELDS:
                np.testing.assert_array_equal(b[k], a[k], err_msg=f"{v} {k}")
    finally:
        _variant(1)
