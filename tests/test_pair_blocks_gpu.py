"""The predicts factored by tile (csrc/pairs.cu) at the edges of their blocks:
16 x 16 pairs and strips of the last tiles on small grids, 32 x 32 with the last
group padded or in strips on large ones, either side of two components, against
the CPU oracle."""

import math

import numpy as np
import pytest

from mwa_hyperdrive_b200 import srclist as sl
from mwa_hyperdrive_b200 import synth
from test_pairs_gpu import LST, PC, components, dipole_gains, expected

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200.model import SkyModeller  # noqa: E402


def check(oracle, ntiles, nf, kind, n, form, beam, dtype, channels):
    """`channels` of an nf-channel predict into a buffer that holds ones."""
    obs = synth.Obs(synth.tiles_in_disk(ntiles, 750.0, ntiles), 167e6 + np.arange(nf) * 20e3, PC, np.array([LST]))
    sky = sl.SkyModelArrays.from_components(components(kind, n, 400 + n))
    kw = {"dipole_gains": dipole_gains(ntiles)} if beam == "per_tile" else {}
    m = SkyModeller(sky, obs.tile_xyzs, obs.freqs, PC, obs.latitude, form=form, beam=beam, **kw)
    vis = torch.ones((nf, obs.num_baselines, 8), dtype=dtype, device="cuda")
    m.model_timestep_with(LST, vis)
    m.close()
    got = vis[channels].cpu().numpy().astype(np.float64) - 1.0
    # (per-tile beams are evaluated at each channel's nearest multiple of 1.28
    # MHz, whichever channels there are)
    ref = expected(oracle, sky, synth.Obs(obs.tile_xyzs, obs.freqs[channels], PC, obs.lsts), beam)
    if form == "direct":
        # the FP64 form's bar
        assert np.max(np.abs(got - ref)) < 1e-10 * max(1.0, math.sqrt(np.mean(ref**2)))
    else:
        # the chosen form's bar
        assert np.linalg.norm(got - ref) < 1e-6 * max(np.linalg.norm(ref), math.sqrt(ref.size))


SMALL = [2, 3, 15, 16, 18, 24, 31, 32, 40, 47, 48, 49, 79, 81]


@pytest.mark.parametrize("form,beam,kind", [("direct", "none", "points"), ("direct", "per_tile", "points"),
                                            ("direct", "none", "gaussians"), ("direct", "per_tile", "shapelets"),
                                            ("tensor", "none", "gaussians"), ("tensor", "per_tile", "gaussians")])
@pytest.mark.parametrize("ntiles", SMALL)
def test_small_grids(oracle, ntiles, form, beam, kind):
    check(oracle, ntiles, 2, kind, 17, form, beam, torch.float64, [0, 1])


# on 148 SMs two groups of 32 need 124 to 395 channels by type, one group of 32
# up to 1184
@pytest.mark.parametrize("form,beam,kind", [("direct", "none", "points"), ("direct", "per_tile", "gaussians"),
                                            ("direct", "none", "gaussians"), ("tensor", "none", "gaussians"),
                                            ("tensor", "per_tile", "gaussians")])
@pytest.mark.parametrize("ntiles,nf", [(32, 1190), (33, 1190), (55, 400), (63, 400), (64, 124), (64, 198), (64, 400), (65, 400),
                                       (80, 400), (86, 400), (87, 400)])
def test_large_grids(oracle, ntiles, nf, form, beam, kind):
    dtype = torch.float32 if form == "tensor" and beam == "none" else torch.float64
    check(oracle, ntiles, nf, kind, 3, form, beam, dtype, [0, nf // 2, nf - 1])


@pytest.mark.parametrize("form,kind", [("direct", "points"), ("direct", "gaussians"), ("tensor", "gaussians")])
@pytest.mark.parametrize("n", [1, 2, 3])
def test_few_components(oracle, n, form, kind):
    check(oracle, 37, 3, kind, n, form, "analytic", torch.float64, [0, 1, 2])
