"""Gaussians of radius 0 -- a covariance that is not a number, an opacity of
exactly 1/255 -- emit nothing, whatever the emission rectangle: the list is that
of the others."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from word2world_b200 import camera, scenes  # noqa: E402


@pytest.mark.parametrize("what", ["covariance", "opacity"])
@pytest.mark.parametrize("spill", [True, False])
@pytest.mark.parametrize("P", [40, 3000])
def test_list_of_the_others(P, spill, what):
    arrays = [a.copy() for a in scenes.make_scene(P, seed=5, layout="ball", log_scale=(-4.0, -2.5)).activate()]
    cam = camera.orbit_camera(15.0, 5.0, 2.5, 172, 144)
    gone = np.arange(P) % 5 == 2
    if what == "covariance":
        arrays[2][gone] = np.nan
    else:
        arrays[1][gone] = np.float32(1) / np.float32(255)  # times 255 it is 1, and its logarithm 0
    f = gh.forward(arrays, cam, compat_spill=spill)
    g = gh.forward([a[~gone] for a in arrays], cam, compat_spill=spill)
    assert np.all(f["radii"][gone] == 0)
    assert np.array_equal(f["point_list"], np.flatnonzero(~gone)[g["point_list"]].astype(np.uint32))
    for k in ("keys", "ranges", "n_contrib", "color", "alpha", "depth_img"):
        assert np.array_equal(f[k], g[k]), k
