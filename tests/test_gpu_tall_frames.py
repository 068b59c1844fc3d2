"""Frames of more rows than a grid of eight-row tiles counts in one launch."""
import numpy as np
import oracle_lib
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("H", [524280, 524281, 600003])
def test_tall_frame_matches_oracle(fs3d, orc, layout, H):
    g = np.random.default_rng(2).choice(np.array([0, 1, 2, 3, 9], np.uint8), (20, 24, 17), p=[0.8, 0.05, 0.08, 0.05, 0.02])
    cam = fs3d.camera_world_view(17, 20, 24, 3, H)
    cam.aspect = 1.5  # (the rows' own: a view of the whole world)
    with fs3d.World(g, 1, 0, layout) as w:
        img = w.render(cam, 3, H)
    exp = orc.render_dda(g, oracle_lib.camera_from(cam), 3, H)
    assert img[..., :3].any()
    assert float(np.abs(img - exp).max()) <= 1e-5
