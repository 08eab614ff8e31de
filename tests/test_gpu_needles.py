"""Needles and other Gaussians whose determinant cancels to almost nothing, of
either sign: the per-tile blend's values are the IEEE division's, which the
queue-fed blend uses for them, bit for bit, and the oracle's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
import oracle  # noqa: E402
import parity  # noqa: E402
from test_gpu_parity import _check_forward, _orc  # noqa: E402
from word2world_b200 import camera, scenes  # noqa: E402


@pytest.mark.parametrize("P", [30, 4000])
@pytest.mark.parametrize("scale", [(3e-2, 1e-6, 1e-6), (8e-2, 1e-5, 1e-5), (2e-2, 2e-2, 1e-7), (6e-4, 4e-4, 1e-4)])
def test_needles(scale, P):
    arrays = [a.copy() for a in scenes.make_scene(P, seed=3, layout="ball", log_scale=(-5.0, -3.0)).activate()]
    arrays[2][:] = scale
    cam = camera.orbit_camera(20.0, 10.0, 2.5, 250, 210)
    f, orc = gh.forward(arrays, cam), _orc(arrays, cam)
    with gh.tuned(blend_queue=1):
        q = gh.forward(arrays, cam)
    for k in ("n_contrib", "color", "alpha", "depth_img", "T_final"):
        assert np.array_equal(f[k], q[k]), k
    _check_forward(f, orc)


@pytest.mark.parametrize("scale", [(3e-2, 1e-6, 1e-6), (8e-2, 1e-5, 1e-5)])
def test_needles_exact_gradients(scale):
    """The exact backward re-evaluates the forward's pairs: finite, and the same from either blend's state."""
    arrays = [a.copy() for a in scenes.make_scene(2000, seed=3, layout="ball", log_scale=(-5.0, -3.0)).activate()]
    arrays[2][:] = scale
    cam = camera.orbit_camera(20.0, 10.0, 2.5, 250, 210)
    up = np.random.default_rng(1).normal(size=(3, 210, 250)).astype(np.float32)
    f = gh.forward(arrays, cam)
    got = gh.backward(f, arrays, cam, up, grad_mode=1)
    keep = np.asarray(_orc(arrays, cam)["blend_margin"]).reshape(210, 250) >= 1e-5
    want = oracle.backward(_orc(arrays, cam), up * keep, mode="exact")
    mine = gh.backward(f, arrays, cam, up * keep, grad_mode=1)
    for k in ("dL_dcolors", "dL_dopacity", "dL_dsh"):  # the geometric ones divide by the cancelled determinant twice
        assert np.isfinite(got[k]).all()
        c = parity.grad_check(mine[k], want[k])
        assert c["norm_rel"] <= 1e-4, (k, c)
