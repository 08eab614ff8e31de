"""The sorted list of a large view, emitted in depth order and sorted by tile
only: its keys and ids are the stable sort, by the full key, of what the
geometry state says every Gaussian owns."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402


def _expected(fwd, P, W, H):
    """(keys, ids) from the state: Gaussian i owns the slots from its start, or the furthest earlier reach, up to its
    own reach; entry k of its rectangle lies row-major."""
    g = fwd["_tensors"]["geom"].cpu().numpy()
    field = lambda name, n: g[_C.geometry_offset(P, name):][:4 * n].view(np.uint32).astype(np.int64)
    start = field("offsets", P) - field("tiles_touched", P)
    rect, reach0 = field("rect", 2 * P).reshape(P, 2), field("prev_reach", P)
    x0, y0, x1, y1 = rect[:, 0] & 0xffff, rect[:, 0] >> 16, rect[:, 1] & 0xffff, rect[:, 1] >> 16
    w = np.maximum(x1 - x0, 0)
    first = np.maximum(start, reach0)
    count = np.maximum(np.minimum(start + w * np.maximum(y1 - y0, 0), fwd["num_rendered"]) - first, 0)
    ids = np.repeat(np.arange(P), count)
    k = np.arange(len(ids)) - np.repeat(np.cumsum(count) - count, count) + np.repeat(first - start, count)
    tile = (y0[ids] + k // w[ids]) * ((W + 15) // 16) + x0[ids] + k % w[ids]
    keys = (tile.astype(np.uint64) << np.uint64(32)) | field("depth", P)[ids].astype(np.uint64)
    order = np.argsort(keys, kind="stable")
    return keys[order], ids[order].astype(np.uint32)


# the instance threshold, one and two words of key, P a multiple of the scan's block and not, few large Gaussians
@pytest.mark.parametrize("P,W,H,scale,radius,spill", [
    (102400, 800, 800, (-5.0, -3.0), 2.5, True),
    (99991, 1001, 777, (-5.0, -3.0), 2.5, False),
    (60013, 1700, 1650, (-5.0, -3.0), 2.4, True),
    (3001, 1024, 1030, (-3.0, -1.5), 2.5, True),
])
@pytest.mark.parametrize("planned", [0, 1])
def test_depth_ordered_emission(P, W, H, scale, radius, spill, planned):
    arrays = scenes.make_scene(P, seed=21, layout="ball", log_scale=scale).activate()
    cam = camera.orbit_camera(33.0, 5.0, radius, W, H)
    with gh.tuned(planned_forward=planned):
        gh.forward(arrays, cam, degree=0, compat_spill=spill)  # a planned render needs one of its size before it
        f = gh.forward(arrays, cam, degree=0, compat_spill=spill)
    assert f["num_rendered"] >= 2_000_000  # the rule's threshold: this list was emitted in depth order
    keys, ids = _expected(f, P, W, H)
    assert np.array_equal(f["keys"], keys)
    assert np.array_equal(f["point_list"], ids)
    _C.check_device_errors()
