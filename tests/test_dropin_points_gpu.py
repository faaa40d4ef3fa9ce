"""model_points either side of the component count at which its kernel goes
from five CTAs an SM to four (csrc/predict.cu, FEW_POINTS), and of a staged
chunk, against the FP64 oracle."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import _lib  # noqa: E402
from test_failure_gpu import DropinPoints, assert_f32_close  # noqa: E402


@pytest.mark.parametrize("nc", [1, 4, 5, 64, 65])
def test_model_points(oracle, nc):
    prob = DropinPoints(oracle, ntiles=25, nf=3, nc=nc, seed=nc)
    vis = torch.zeros((prob.nf, prob.nbl, 8), dtype=torch.float32, device="cuda")
    _lib.check_str(prob.call(vis), "model_points")
    torch.cuda.synchronize()
    assert_f32_close(vis.cpu().numpy(), prob.ref)
