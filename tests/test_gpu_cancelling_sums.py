"""Gradients whose other sums cancel.  Faint Gaussians centred between two pixel
columns (rows) of one 8x4 block, under an upstream gradient of opposite signs on
the two sides: the block's sums for opacity, colour and the squared offsets are
exactly 0, and the mean's gradient is not; under one that changes sign from
quadrant to quadrant every sum but that of the offsets' product is 0."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
import oracle  # noqa: E402
import parity  # noqa: E402
from test_gpu_parity import _orc  # noqa: E402
from word2world_b200 import camera  # noqa: E402

W, H = 24, 12  # the centre (11.5, 5.5) is also the centre of the block at (8, 4)


def centred(n):
    """n equal Gaussians on the view axis: standard deviation sqrt(1/2) pixels, the nearest pixels within alpha 1/255."""
    cam = camera.orbit_camera(0.0, 0.0, 2.5, W, H)
    z = np.linspace(-0.1, 0.1, n) if n > 1 else np.zeros(1)
    means = np.zeros((n, 3), np.float32)
    means[:, 2] = z
    dist = 2.5 - z if n > 1 else np.full(1, 2.5)
    scales = np.repeat((np.sqrt(0.5) * dist / cam.focal_x)[:, None], 3, 1).astype(np.float32)
    rots = np.tile(np.array([[1, 0, 0, 0]], np.float32), (n, 1))
    sh = np.zeros((n, 16, 3), np.float32)
    sh[:, 0] = 1.0
    return (means, np.full((n, 1), 0.02, np.float32), scales, rots, sh), cam


# 1, 12 and 24 entries: four, two and one lanes to an entry
@pytest.mark.parametrize("n", [1, 12, 24])
@pytest.mark.parametrize("sides", ["columns", "rows", "quadrants"])
@pytest.mark.parametrize("mode", ["reference", "exact"])
def test_gradients_of_centred_gaussians(n, sides, mode):
    arrays, cam = centred(n)
    f, orc = gh.forward(arrays, cam), _orc(arrays, cam)
    assert np.all(f["means2D"] == np.array([11.5, 5.5], np.float32))
    x, y = np.sign(np.arange(W) - 11.5), np.sign(np.arange(H) - 5.5)
    up = {"columns": x + 0 * y[:, None], "rows": 0 * x + y[:, None], "quadrants": x * y[:, None]}[sides]
    up = np.repeat(up[None], 3, 0).astype(np.float32)
    mine = gh.backward(f, arrays, cam, up, grad_mode=0 if mode == "reference" else 1)
    want = oracle.backward(orc, up, mode=mode)
    # what the cancelling sums leave: a column of the mean's gradient, or the covariance's off-diagonal one
    kept = np.asarray(want["dL_dcov3D"])[:, 1] if sides == "quadrants" else \
        np.asarray(want["dL_dmeans2D"])[:, 0 if sides == "columns" else 1]
    assert np.all(np.abs(kept) > 0.1)
    for k in parity.GRAD_NAMES:
        c = parity.grad_check(mine[k], want[k])
        assert c["n_bad"] == 0, (k, c)
        if np.abs(want[k]).max() > 0.01:
            assert c["norm_rel"] <= 1e-4, (k, c)
