"""model_points either side of the component count at which its kernel goes
from five CTAs an SM to four, with per-tile beams from three to two
(csrc/predict.cu, FEW_POINTS), and of a staged chunk, against the FP64 oracle and
the tensor-core predict."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import _lib  # noqa: E402
from test_failure_gpu import DropinPoints, assert_f32_close  # noqa: E402
from test_reference_gpu import dev, dropin_inputs  # noqa: E402


@pytest.mark.parametrize("nc", [1, 4, 5, 64, 65])
def test_model_points(oracle, nc):
    prob = DropinPoints(oracle, ntiles=25, nf=3, nc=nc, seed=nc)
    vis = torch.zeros((prob.nf, prob.nbl, 8), dtype=torch.float32, device="cuda")
    _lib.check_str(prob.call(vis), "model_points")
    torch.cuda.synchronize()
    assert_f32_close(vis.cpu().numpy(), prob.ref)


@pytest.mark.parametrize("per_group", [1, 2])
def test_per_tile_beams(oracle, per_group):
    comps, a, uvws, beam, (nf, nbl), obs = dropin_inputs(oracle, 30, 4, per_group, 0, 5, want_obs=True)
    ref = torch.zeros((nf, nbl, 8), dtype=torch.float64, device="cuda")
    _lib.check_str(_lib.lib().model_points_f64out(ctypes.byref(comps), ctypes.byref(a), uvws, beam, ref.data_ptr()), "")
    got = torch.zeros((nf, nbl, 8), dtype=torch.float32, device="cuda")
    xyz = dev(obs.tile_xyzs)
    _lib.check_str(_lib.lib().model_points_tc(ctypes.byref(comps), ctypes.byref(a), xyz.data_ptr(),
                                              float(obs.lsts[0]), _lib.RADec(*obs.phase_centre), beam,
                                              got.data_ptr()), "")
    # the tensor-core predict's bar
    assert (got - ref).norm() < 1e-6 * ref.norm()
