"""Values that are not finite stay where they belong: a pair that the blend
skipped takes nothing from its Gaussian's colour or its pixel's upstream
gradient."""
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


def _scene(P, seed=5):
    return (scenes.make_scene(P, seed=seed, layout="ball", log_scale=(-4.0, -2.5)).activate(),
            camera.orbit_camera(15.0, 5.0, 2.5, W, H))


def _agrees(mine, want):
    """No value that the oracle has finite is not, and the rows finite in both agree."""
    for k in parity.GRAD_NAMES:
        a, b = mine[k].reshape(len(mine[k]), -1), np.asarray(want[k]).reshape(len(mine[k]), -1)
        spread = ~np.isfinite(a) & np.isfinite(b)
        assert not spread.any(), (k, int(spread.any(1).sum()))
        rows = np.isfinite(a).all(1) & np.isfinite(b).all(1)
        assert rows.sum() >= 10, (k, int(rows.sum()))
        c = parity.grad_check(a[rows], b[rows])
        assert c["norm_rel"] <= 1e-4, (k, c)


def _case(P, where, value):
    """Arrays, camera and upstream gradients."""
    arrays, cam = _scene(P)
    rng = np.random.default_rng(P)
    up = rng.normal(size=(3, H, W)).astype(np.float32)
    dep, al = rng.normal(size=(2, 1, H, W)).astype(np.float32)
    orc = _orc(arrays, cam)
    plain = oracle.backward(orc, up, mode="reference")
    # pixels that no decision at a threshold separates from the oracle's
    keep = (np.asarray(orc["blend_margin"]).reshape(H, W) >= 1e-5) & (plain["backward_margin"] >= 1e-5)
    up, dep, al = up * keep, dep * keep, al * keep
    if where == "colour":  # the Gaussian that counts most
        arrays[4][int(np.argmax(np.abs(plain["dL_dcolors"]).sum(1))), 0] = value
    else:
        y, x = divmod(int(np.argmax(orc["alpha"])), W)
        up[1, y, x] = value
    return arrays, cam, (up, dep, al)


# few, some and many entries to a block: four, two and one lanes to an entry
@pytest.mark.parametrize("P", [60, 400, 3000])
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("where", ["colour", "upstream"])
@pytest.mark.parametrize("mode", ["reference", "exact"])
def test_skipped_pairs_stay_finite(P, value, where, mode):
    arrays, cam, up = _case(P, where, value)
    f = gh.forward(arrays, cam)
    # the oracle starts from the same alpha image (test_gpu_parity's _grads says why)
    orc = dict(_orc(arrays, cam), alpha=f["alpha"])
    with np.errstate(all="ignore"):
        want = oracle.backward(orc, *up, mode=mode, error_bounds=False)
    assert any(not np.isfinite(want[k]).all() for k in parity.GRAD_NAMES)
    _agrees(gh.backward(f, arrays, cam, *up, grad_mode=0 if mode == "reference" else 1), want)
