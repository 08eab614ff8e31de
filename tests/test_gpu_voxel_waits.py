"""The voxel field's scan and sort with a tile that does not publish: the call
reports the wait that ran out, reads and writes nothing out of range, and the
next one is right."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

from oracle import voxel as ovox  # noqa: E402
from test_gpu_voxel_routes import _close, _field, _gaussians  # noqa: E402
from test_gpu_waits import STAGE_SCAN, STAGE_SORT, hooked  # noqa: E402


# block slots: three tiles of 2048 pairs.  Counted: a scan of 12289 counts in four tiles, and its pairs' sort
@pytest.mark.parametrize("stage,tile,n,b,relax", [
    (STAGE_SORT, 0, 700, 5, 0.1), (STAGE_SORT, 1, 12289, 7, 3.0), (STAGE_SCAN, 0, 12289, 7, 3.0),
    (STAGE_SCAN, 2, 12289, 7, 3.0)])
def test_wait_runs_out_and_is_reported(stage, tile, n, b, relax):
    r = 12
    args = _gaussians(n, seed=n)
    with hooked(stage, tile):
        with pytest.raises(RuntimeError, match="timed out|timeout"):
            _field(*args, r, b, relax)
    _close(_field(*args, r, b, relax), ovox.voxel_field(*args, r, b, relax), n)
