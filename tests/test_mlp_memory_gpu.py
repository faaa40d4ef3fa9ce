"""Device memory of the warm-start network: prediction does not take the
gradient's parts, gradients grow them with the batch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import warmstart as ws  # noqa: E402
from oracle import mlp_ref  # noqa: E402


def test_forward_takes_activations_only():
    hidden, batch = 2048, 8192
    x = torch.randn((batch, ws.IN_DIM), device="cuda")
    y = torch.empty((batch, ws.OUT_DIM), device="cuda")
    m = ws.WarmStartMLP(hidden=hidden, num_hidden=3, seed=1)
    m.forward_device(x[:1], y[:1])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    m.forward_device(x, y)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    m.close()
    # activations and their gradients of three hidden layers, 0.4 GB; the
    # parts of 32 splits would be another 1.1 GB
    assert used < 2 * 3 * 4 * batch * hidden + (64 << 20), used


def test_gradients_after_forward_and_with_growing_batches():
    rng = np.random.default_rng(2)
    m = ws.WarmStartMLP(hidden=24, num_hidden=2, seed=3)
    p = m.get_params()
    for batch in (3000, 10, 300, 9000):
        x = rng.normal(size=(batch, ws.IN_DIM)).astype(np.float32)
        t = rng.normal(size=(batch, ws.OUT_DIM)).astype(np.float32)
        d_x = torch.from_numpy(x).cuda()
        if batch == 3000:
            m.forward_device(d_x, torch.empty((batch, ws.OUT_DIM), device="cuda"))
            continue
        loss, g = m.gradients(d_x, torch.from_numpy(t).cuda())
        ref_loss, ref_g = mlp_ref.gradients(p, m.dims, x, t, ws.CENTRE)
        # FP32 sums of at most 9000 terms
        assert abs(loss - ref_loss) <= 1e-5 * ref_loss
        assert np.linalg.norm(g - ref_g) < 2e-4 * np.linalg.norm(ref_g)
