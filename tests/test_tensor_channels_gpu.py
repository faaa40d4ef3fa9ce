"""Per-tile beams in the tensor form with tens of thousands of channels, each
a beam frequency of its own: channels and beam frequencies together exceed the
65535 of a grid's y extent (csrc/tensor.cu, beam_bounds_kernel)."""

import numpy as np
import pytest

from mwa_hyperdrive_b200 import srclist, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200.model import SkyModeller  # noqa: E402


@pytest.mark.parametrize("channels", [32767, 32768, 40001])
def test_many_channels_and_beam_frequencies(channels):
    centre = (0.0, -0.47)
    sky = srclist.SkyModelArrays.from_components(synth.point_sky(3, centre, 10.0, 5))
    xyzs = synth.tiles_in_disk(3, 300.0, 7)
    freqs = 150e6 + 1e3 * np.arange(channels)
    gains = np.ones((3, 2, 16))
    gains[1, 0, 4] = gains[2, 1, 9] = 0.0
    out = {}
    for form in ("direct", "tensor"):
        m = SkyModeller(sky, xyzs, freqs, centre, synth.MWA_LAT_RAD, beam="per_tile", form=form, dipole_gains=gains,
                        beam_freq_res_hz=1e3)
        vis = torch.zeros((channels, 3, 8), dtype=torch.float64, device="cuda")
        m.model_timestep_with(0.02, vis, return_uvws=False)
        out[form] = vis
        torch.cuda.synchronize()
        m.close()
    # FP32 phasors and beams (6e-8 each) against FP64: a few parts in 1e7
    err = (out["tensor"] - out["direct"]).norm() / out["direct"].norm()
    assert err < 1e-6, err
