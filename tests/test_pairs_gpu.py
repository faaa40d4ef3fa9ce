"""The predicts factored by tile (csrc/pairs.cu) and the shapelet kernel of the
chosen form (csrc/predict.cu) at the edges of their 32 x 32 blocks of tile
pairs and of their staged chunks of components, against the CPU oracle."""

import math

import numpy as np
import pytest

from mwa_hyperdrive_b200 import srclist as sl
from mwa_hyperdrive_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200.model import SkyModeller  # noqa: E402

PC = (0.2, math.radians(-27.0))
LST = 0.25


def components(kind, n, seed):
    if kind == "points":
        return synth.point_sky(n, PC, 10.0, seed, curved_q_sigma=0.2)
    if kind == "gaussians":
        return synth.gaussians_and_shapelets(n, 0, PC, seed)
    return synth.gaussians_and_shapelets(0, n, PC, seed)


def predict(sky, obs, form, beam, dtype):
    kw = {}
    if beam == "per_tile":
        kw["dipole_gains"] = dipole_gains(obs.num_tiles)
    m = SkyModeller(sky, obs.tile_xyzs, obs.freqs, obs.phase_centre, obs.latitude, form=form, beam=beam, **kw)
    vis = torch.zeros((obs.freqs.size, obs.num_baselines, 8), dtype=dtype, device="cuda")
    m.model_timestep_with(LST, vis)
    m.close()
    return vis.cpu().numpy()


def dipole_gains(ntiles):
    g = np.ones((ntiles, 2, 16))
    for t in range(0, ntiles, 3):
        g[t, t % 2, (t // 3) % 4] = 0.0
    return g


def expected(oracle, sky, obs, beam):
    if beam == "per_tile":
        uniq, tmap, ufreqs, fmap = oracle.unique_tile_beams(dipole_gains(obs.num_tiles), obs.freqs)
        tables = [oracle.tile_beam_table(sky, ty, LST, obs.latitude, uniq, ufreqs)
                  if np.any(sky.comp_type == ty) else None for ty in range(3)]
        b = oracle.beam_struct(2, tables, tmap, fmap, ufreqs.size)
    else:
        b = oracle.beam_struct({"none": 0, "analytic": 1}[beam])
    return oracle.model_timestep(sky, obs.tile_xyzs, obs.freqs, PC, LST, obs.latitude, beam=b, out_f64=True)[0]


def observation(ntiles, seed):
    return synth.Obs(synth.tiles_in_disk(ntiles, 750.0, seed), 167e6 + np.arange(3) * 1.28e6, PC, np.array([LST]))


@pytest.mark.parametrize("beam", ["none", "analytic", "per_tile"])
@pytest.mark.parametrize("kind", ["points", "gaussians", "shapelets"])
@pytest.mark.parametrize("ntiles,n", [(2, 1), (16, 8), (17, 9), (33, 33), (64, 16), (65, 17)])
def test_fp64(oracle, kind, beam, ntiles, n):
    obs = observation(ntiles, ntiles)
    sky = sl.SkyModelArrays.from_components(components(kind, n, 100 + n))
    got = predict(sky, obs, "direct", beam, torch.float64)
    ref = expected(oracle, sky, obs, beam)
    rms = math.sqrt(np.mean(ref**2))
    assert np.max(np.abs(got - ref)) < 1e-10 * rms  # the FP64 form's bar


@pytest.mark.parametrize("kind", ["gaussians", "shapelets"])
@pytest.mark.parametrize("ntiles,n", [(2, 1), (17, 15), (33, 33), (64, 64), (65, 17)])
def test_chosen_form(oracle, kind, ntiles, n):
    obs = observation(ntiles, ntiles)
    sky = sl.SkyModelArrays.from_components(components(kind, n, 200 + n))
    for dtype in (torch.float64, torch.float32):
        got = predict(sky, obs, "tensor", "analytic", dtype)
        ref = expected(oracle, sky, obs, "analytic")
        # the chosen form's bar
        assert np.linalg.norm(got - ref) < 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("kind", ["points", "gaussians", "shapelets"])
@pytest.mark.parametrize("ntiles,n", [(2, 1), (16, 8), (17, 9), (33, 33), (65, 17), (130, 16)])
def test_chosen_form_per_tile(oracle, kind, ntiles, n):
    obs = observation(ntiles, ntiles)
    sky = sl.SkyModelArrays.from_components(components(kind, n, 300 + n))
    ref = expected(oracle, sky, obs, "per_tile")
    for dtype in (torch.float64, torch.float32):
        got = predict(sky, obs, "tensor", "per_tile", dtype)
        # the chosen form's bar
        assert np.linalg.norm(got - ref) < 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("nuniq", [28, 29])
def test_shapelets_per_tile_either_side_of_the_rule(nuniq):
    """More CTAs than an SM each: two share one up to 28 unique tiles."""
    ntiles, nf = 128, 48
    obs = synth.Obs(synth.tiles_in_disk(ntiles, 750.0, 4), 167e6 + np.arange(nf) * 40e3, PC, np.array([LST]))
    sky = sl.SkyModelArrays.from_components(components("shapelets", 9, 11))
    gains = np.random.default_rng(9).uniform(0.5, 1.0, (nuniq, 2, 16))[np.arange(ntiles) % nuniq]
    vis = {}
    for form in ("direct", "tensor"):
        m = SkyModeller(sky, obs.tile_xyzs, obs.freqs, PC, obs.latitude, form=form, beam="per_tile", dipole_gains=gains)
        vis[form] = torch.zeros((nf, obs.num_baselines, 8), dtype=torch.float64, device="cuda")
        m.model_timestep_with(LST, vis[form])
        m.close()
    assert torch.linalg.norm(vis["tensor"] - vis["direct"]) < 1e-6 * torch.linalg.norm(vis["direct"])


def test_points_per_tile_in_chunks_of_channels():
    """More components than a pass takes and a table that exceeds its cap, so
    that channels go through it in turn, against the FP64 form."""
    ntiles, nf = 80, 45
    obs = synth.Obs(synth.tiles_in_disk(ntiles, 750.0, 3), 167e6 + np.arange(nf) * 40e3, PC, np.array([LST]))
    sky = sl.SkyModelArrays.from_components(components("points", 8011, 7))
    gains = np.random.default_rng(8).uniform(0.5, 1.0, (ntiles, 2, 16))
    vis = {}
    for form in ("direct", "tensor"):
        m = SkyModeller(sky, obs.tile_xyzs, obs.freqs, PC, obs.latitude, form=form, beam="per_tile", dipole_gains=gains)
        vis[form] = torch.zeros((nf, obs.num_baselines, 8), dtype=torch.float64, device="cuda")
        m.model_timestep_with(LST, vis[form])
        m.close()
    assert torch.linalg.norm(vis["tensor"] - vis["direct"]) < 1e-6 * torch.linalg.norm(vis["direct"])


def test_chosen_form_shapelets_beyond_the_staged_window(oracle):
    """Sources of a degree on long baselines: positions far from the basis
    table's centre, and past its ends."""
    obs = synth.Obs(synth.tiles_in_disk(20, 3000.0, 5), 180e6 + np.arange(5) * 80e3, PC, np.array([LST]))
    rng = np.random.default_rng(6)
    comps = []
    for k, maj in enumerate(np.radians([0.02, 0.2, 1.0, 4.0])):
        co = [sl.ShapeletCoeff(int(rng.integers(0, 6)), int(rng.integers(0, 6)), float(rng.normal())) for _ in range(8)]
        comps.append(sl.SourceComponent(PC[0] + 0.01 * k, PC[1], sl.Shapelet(maj, 0.7 * maj, 0.3 * k, co),
                                        sl.PowerLaw(-0.7, sl.FluxDensity(150e6, 1.0 + k))))
    sky = sl.SkyModelArrays.from_components(comps)
    ref = expected(oracle, sky, obs, "none")
    got = predict(sky, obs, "tensor", "none", torch.float64)
    assert np.linalg.norm(got - ref) < 1e-6 * np.linalg.norm(ref)
    got = predict(sky, obs, "direct", "none", torch.float64)
    assert np.linalg.norm(got - ref) < 1e-10 * np.linalg.norm(ref)
