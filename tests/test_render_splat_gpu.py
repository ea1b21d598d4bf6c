"""The phase thickness by counting (fractions all 0 or 1) against the oracle's
sums in submission order: bit for bit, for points in cell order and shuffled
(a CTA's box too large for shared memory), one and several phases, sprites of
one pixel to most of the window, numbers of points around a CTA's share, and
with a fraction that is neither 0 nor 1, which takes the ordered lists."""
import numpy as np
import pytest

import aquarius_b200 as aq
from aquarius_b200 import _abi
from oracle_binding import RenderOracle
from test_render_gpu import _draw

pytestmark = pytest.mark.gpu


def _points(n, seed, phases, shuffled):
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*(np.arange(side),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    p = np.zeros((n, 7), np.float32)
    p[:, :3] = (grid + rng.random((n, 3))) * (10.0 / side)
    f = np.eye(4, dtype=np.float32)[rng.integers(0, phases, n)] if phases else np.zeros((n, 4), np.float32)
    if phases > 1:
        f[::7] = 1.0  # several at once, and none
        f[::11] = 0.0
    p[:, 3:] = f
    return np.ascontiguousarray(p[rng.permutation(n)] if shuffled else p)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,phases,shuffled,radius,window", [
    (1, 1, False, 0.2, (64, 32)),
    (511, 1, False, 0.2, (333, 197)),
    (512, 4, False, 0.1, (128, 64)),
    (513, 2, True, 0.4, (200, 100)),
    (20000, 1, False, 0.05, (640, 320)),
    (20000, 4, True, 0.1, (1728, 864)),
    (700, 2, False, 20.0, (160, 120)),   # sprites over most of the window
    (3000, 0, False, 0.1, (160, 120)),   # no fraction at all
])
def test_counted_thickness_equals_the_ordered_sums(n, phases, shuffled, radius, window, mixed):
    pts = _points(n, n, phases, shuffled)
    if mixed:
        pts[n // 2, 3:] = (0.25, 0.75, 0.0, 0.0)
    dc = aq.draw_command_default(*window, 10.0, 32)
    dc.render_mode = _abi.RENDER_MULTIPHASE_MESH
    dc.point_radius = radius
    r = aq.Renderer(0)
    img, got = _draw(r, dc, pts, None)
    want_img, want = RenderOracle().frame(dc, pts, None)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(img, want_img)
    assert phases == 0 or n < 100 or got.any()
    # the same renderer again, the other way round
    pts2 = _points(n, n + 1, max(phases, 1), shuffled)
    if not mixed:
        pts2[0, 3] = 0.5
    _, got2 = _draw(r, dc, pts2, None)
    _, want2 = RenderOracle().frame(dc, pts2, None)
    np.testing.assert_array_equal(got2, want2)
    r.close()


def test_frames_of_mixed_phases_start_with_the_lists():
    """A renderer whose last frame met mixed phases does not count first: that
    frame launches less than the first of its kind, and one whose phases are
    apart again shows the same texture on either path."""
    apart, mixed = _points(5000, 1, 4, False), _points(5000, 1, 4, False)
    mixed[7, 3:] = (0.25, 0.75, 0.0, 0.0)
    dc = aq.draw_command_default(320, 160, 10.0, 32)
    dc.render_mode = _abi.RENDER_MULTIPHASE_MESH
    r = aq.Renderer(0)
    launches, got = [], []
    for pts in (apart, mixed, mixed, apart, apart):
        got.append(_draw(r, dc, pts, None)[1])
        launches.append(r.launches())
    r.close()
    for k, pts in ((0, apart), (1, mixed)):
        np.testing.assert_array_equal(got[k], RenderOracle().frame(dc, pts, None)[1])
    for k, same in ((2, 1), (3, 0), (4, 0)):
        np.testing.assert_array_equal(got[k], got[same])
    assert launches[2] < launches[1] and launches[3] == launches[2] and launches[4] == launches[0]


@pytest.mark.parametrize("n", [300, 20000])
def test_large_sprites_take_the_lists(n):
    """Counting visits every pixel of a sprite, the lists every 8 x 8 tile: from
    some 20 pixels a side on the lists are faster.  The same texture."""
    pts = _points(n, n, 2, False)
    dc = aq.draw_command_default(640, 320, 10.0, 32)
    dc.render_mode = _abi.RENDER_MULTIPHASE_MESH
    launches = []
    r = aq.Renderer(0)
    for radius in (0.1, 3.0):  # 2 and 64 pixels a side
        dc.point_radius = radius
        _, got = _draw(r, dc, pts, None)
        launches.append(r.launches())
        np.testing.assert_array_equal(got, RenderOracle().frame(dc, pts, None)[1])
    r.close()
    assert launches[0] < launches[1]


def test_too_many_sprite_tile_pairs_are_refused():
    """2^24 sprites of over 128 tiles each, close to the camera: more pairs than
    a frame takes, also where the thickness is counted."""
    import torch
    dc = aq.draw_command_default(1728, 864, 10.0, 128)
    dc.render_mode = _abi.RENDER_MULTIPHASE_MESH
    dc.point_radius = 0.2  # 11.6 pixels a side at the container's centre, 18 away; 119 at 1.75
    cam = np.array(list(dc.camera_position))
    at = cam + (5.0 - cam) / np.linalg.norm(5.0 - cam) * 1.75
    pts = torch.zeros(1 << 24, 7, device="cuda")
    pts[:, :3] = torch.tensor(at, dtype=torch.float32)
    pts[:, 3] = 1.0
    torch.cuda.synchronize()
    r = aq.Renderer(0)
    with pytest.raises(aq.AquariusError, match="primitive-tile pairs"):
        r.draw(dc, pts.data_ptr(), pts.shape[0], 0, 0)
    few = pts[:100000].contiguous()
    torch.cuda.synchronize()
    r.draw(dc, few.data_ptr(), few.shape[0], 0, 0)
    r.synchronize()
    assert r.phase_thickness().max() == 100000.0
    r.close()
