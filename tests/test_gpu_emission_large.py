"""Key emission of Gaussians that cover more than 2^16 tiles (whose rows are
found by division) beside ones that cover fewer (by multiplication)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from test_gpu_depth_order import _expected  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402


# 257 x 257 tiles: the whole grid is above 2^16; one row of tiles; in index and (from 2M instances) in depth order
@pytest.mark.parametrize("P,W,H,scale,above", [
    (5, 4112, 4112, (1.0, 1.5), True),
    (45, 4112, 4099, (0.5, 1.5), True),
    (40, 4112, 9, (-4.0, 1.0), False),
    (33, 17, 4099, (-4.0, 1.0), False),
])
def test_emission_of_large_rectangles(P, W, H, scale, above):
    arrays = scenes.make_scene(P, seed=5, layout="ball", log_scale=scale).activate()
    cam = camera.orbit_camera(33.0, 5.0, 2.5, W, H)
    f = gh.forward(arrays, cam, degree=0, compat_spill=False)
    keys, ids = _expected(f, P, W, H)
    if above:
        assert np.bincount(ids).max() > 65536
    assert np.array_equal(f["keys"], keys)
    assert np.array_equal(f["point_list"], ids)
    _C.check_device_errors()
