"""An infinite opacity: its alpha is 0.99 wherever the Gaussian is listed, also
where its value underflows to 0 (infinity times 0), in the exact backward as in
the forward; clamped there, it passes no gradient to its own geometry."""
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
from word2world_b200 import camera, scenes  # noqa: E402

W, H = 72, 44


# few, some and many entries to a block: four, two and one lanes to an entry
@pytest.mark.parametrize("P", [60, 400, 3000])
def test_exact_gradients_beside_an_infinite_opacity(P):
    arrays = scenes.make_scene(P, seed=6, layout="ball", log_scale=(-4.0, -2.5)).activate()
    cam = camera.orbit_camera(15.0, 5.0, 2.5, W, H)
    rng = np.random.default_rng(P)
    up = rng.normal(size=(3, H, W)).astype(np.float32)
    dep, al = rng.normal(size=(2, 1, H, W)).astype(np.float32)
    plain = oracle.backward(_orc(arrays, cam), up, mode="reference")
    i = int(np.argmax(np.abs(plain["dL_dcolors"]).sum(1)))  # one that counts, made small: 0 at most of its tile's pixels
    arrays[1][i], arrays[2][i] = np.inf, 0.01
    orc = _orc(arrays, cam)
    keep = np.asarray(orc["blend_margin"]).reshape(H, W) >= 1e-5
    up, dep, al = up * keep, dep * keep, al * keep
    want = oracle.backward(orc, up, dep, al, mode="exact")
    f = gh.forward(arrays, cam)
    assert np.array_equal(f["n_contrib"], np.asarray(orc["n_contrib"]).reshape(H, W))
    mine = gh.backward(f, arrays, cam, up, dep, al, grad_mode=1)
    assert np.abs(want["dL_dcolors"][i]).max() > 0.1
    for k in parity.GRAD_NAMES:
        assert np.isfinite(want[k]).all() and np.isfinite(mine[k]).all(), k
        c = parity.grad_check(mine[k], want[k])
        assert c["norm_rel"] <= 1e-4, (k, c)
