"""The warm-start network's kernels at the edges of their tiles, batch splits
and vector loads, against the float64 oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import warmstart as ws  # noqa: E402
from oracle import mlp_ref  # noqa: E402


@pytest.mark.parametrize("hidden,layers", [(37, 3), (64, 1), (65, 9)])
@pytest.mark.parametrize("batch,offset", [(1, 0), (17, 1), (257, 0), (9000, 0)])
def test_forward_and_gradients(hidden, layers, batch, offset):
    rng = np.random.default_rng(batch)
    m = ws.WarmStartMLP(hidden=hidden, num_hidden=layers, seed=3)
    p = (m.get_params() + rng.normal(0, 0.05, m.num_params)).astype(np.float32)
    m.set_params(p)
    x = rng.normal(size=(batch, ws.IN_DIM)).astype(np.float32)
    t = rng.normal(size=(batch, ws.OUT_DIM)).astype(np.float32)
    # an input that starts `offset` floats into its allocation
    d_x = torch.from_numpy(np.concatenate([np.zeros(offset, np.float32), x.ravel()])).cuda()[offset:].view(batch, -1)
    loss, g = m.gradients(d_x, torch.from_numpy(t).cuda())
    ref_loss, ref_g = mlp_ref.gradients(p, m.dims, x, t, ws.CENTRE)
    # FP32 sums of at most 9000 terms, nine layers deep
    assert abs(loss - ref_loss) <= 1e-5 * ref_loss
    assert np.linalg.norm(g - ref_g) < 2e-4 * np.linalg.norm(ref_g)
    y = torch.empty((batch, ws.OUT_DIM), device="cuda")
    m.forward_device(d_x, y)
    yr, _ = mlp_ref.forward(p, m.dims, x, ws.CENTRE)
    np.testing.assert_allclose(y.cpu().numpy(), yr, rtol=1e-4, atol=1e-4)


def test_output_over_the_input():
    """The output may overlap the input: it is written once that has been read."""
    m = ws.WarmStartMLP(hidden=32, num_hidden=2, seed=1)
    m.set_params(m.get_params() + np.float32(0.01))
    x = torch.randn((300, ws.IN_DIM), device="cuda")
    y = torch.empty((300, ws.OUT_DIM), device="cuda")
    m.forward_device(x, y)
    m.forward_device(x, x)
    torch.testing.assert_close(x.flatten()[: y.numel()], y.flatten(), rtol=0, atol=0)
