"""A colour that is not finite reaches the pixels that blend its Gaussian, and no
other: not the block's pixels that skip it, nor those that had ended before it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
import parity  # noqa: E402
from test_gpu_parity import _orc  # noqa: E402
from word2world_b200 import camera, scenes  # noqa: E402


def _check(arrays, cam, queue):
    orc = _orc(arrays, cam)
    with gh.tuned(blend_queue=queue):
        f = gh.forward(arrays, cam)
    shape = f["n_contrib"].shape
    keep = np.asarray(orc["blend_margin"]).reshape(shape) >= 1e-5
    for k in ("color", "depth_img", "alpha"):
        a, b = f[k][:, keep], np.asarray(orc[k]).reshape(f[k].shape)[:, keep]
        fine = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), fine), (k, int((np.isfinite(a) != fine).sum()))
        assert parity.err_stats(a[fine], b[fine])["n_bad"] == 0, k
    return f, orc


@pytest.mark.parametrize("queue", [0, 1])
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("P", [60, 400, 3000])
def test_pixels_that_skip_it(P, value, queue):
    arrays = scenes.make_scene(P, seed=5, layout="ball", log_scale=(-4.0, -2.5)).activate()
    cam = camera.orbit_camera(15.0, 5.0, 2.5, 72, 44)
    seen = _orc(arrays, cam)
    order = np.argsort(-np.where(seen["visible"], seen["radii"] * arrays[1][:, 0] - seen["depth"], -np.inf))
    arrays[4][order[:5], 0] = value
    _, orc = _check(arrays, cam, queue)
    assert not np.isfinite(orc["color"]).all()


# the entry's place in its group of 32, and in the next one
@pytest.mark.parametrize("queue", [0, 1])
@pytest.mark.parametrize("at", [5, 9, 31, 40])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_pixels_that_had_ended(at, value, queue):
    n = at + 1
    cam = camera.orbit_camera(0.0, 0.0, 2.5, 24, 12)
    means = np.zeros((n, 3), np.float32)
    means[:, 2] = np.linspace(0.1, -0.1, n)  # nearest first
    sh = np.ones((n, 16, 3), np.float32) * np.array([1.0] + [0.0] * 15, np.float32)[:, None]
    sh[at, 0] = value
    arrays = (means, np.full((n, 1), 0.999, np.float32), np.full((n, 3), 4.0, np.float32),
              np.tile(np.array([[1, 0, 0, 0]], np.float32), (n, 1)), sh)
    f, orc = _check(arrays, cam, queue)
    assert np.isfinite(orc["color"]).all() and np.isfinite(f["color"]).all()
