"""Calls that do with less device scratch: the plain calibration's streaming
kernel and its groups of chanblocks, and the tensor predict's table of per-tile
beams one channel at a time.  hdc_test_limit_scratch makes the scratch
unavailable."""

import contextlib
import ctypes

import numpy as np
import pytest

from mwa_hyperdrive_b200 import srclist, synth
from test_calibrate_gpu import identity
from test_reference_gpu import dev, dropin_inputs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import _lib  # noqa: E402
from mwa_hyperdrive_b200 import calibrate as cal  # noqa: E402
from mwa_hyperdrive_b200.model import SkyModeller  # noqa: E402


@contextlib.contextmanager
def limit(nbytes):
    _lib.lib().hdc_test_limit_scratch(nbytes)
    try:
        yield
    finally:
        _lib.lib().hdc_test_limit_scratch(0)


def cov_bytes(ntiles):
    """FP64 covariances of a chanblock: 48 numbers a pair of a 16 x 16 block."""
    n = (ntiles + 15) // 16
    return 8 * 48 * 256 * n * (n + 1) // 2


def problem(ntiles, nt, nch):
    """A chanblock starts from zero gains and is retried; one has no data."""
    rng = np.random.default_rng(ntiles + nch)
    model = synth.random_model(nt, nch, ntiles * (ntiles - 1) // 2, rng)
    data = synth.corrupt(model, synth.truth_gains(ntiles, nch, rng), rng, 20.0)
    start = identity(ntiles, nch)
    start[:, 2] = 0.0
    data[:, 4] = 0.0
    model[:, 4] = 0.0
    return data, model, start


def compare(got, res, want, ores):
    assert [(r.num_iterations, r.converged, r.num_failed) for r in res] == \
        [(r["num_iterations"], r["converged"], r["num_failed"]) for r in ores]
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    if ok.any():
        assert np.linalg.norm(got[ok] - want[ok]) / np.linalg.norm(want[ok]) < 1e-10


# 0 chanblocks a group: the data and model are streamed every iteration
@pytest.mark.parametrize("group", [0, 1, 2, 5])
@pytest.mark.parametrize("ntiles", [2, 7, 17, 49, 128, 256])
def test_plain_calibration(oracle, ntiles, group):
    nt, nch = 2, 6
    data, model, start = problem(ntiles, nt, nch)
    d, m = torch.from_numpy(data).cuda(), torch.from_numpy(model).cuda()
    dj = torch.from_numpy(start).cuda()
    with limit(max(1, group * cov_bytes(ntiles))):
        res = cal.calibrate_timeblock(d, m, dj, (0, nt), 20, 1e-8, 1e-4)
        many, mres = cal.calibrate_timeblocks(d, m, [(0, 1), (1, 2)], 20, 1e-8, 1e-4)
    compare(dj.cpu().numpy(), res, *oracle.calibrate_timeblock(data, model, start, 0, nt, 20, 1e-8, 1e-4, 0))
    for k in range(2):
        compare(many[k], mres[k], *oracle.calibrate_timeblock(data, model, identity(ntiles, nch), k, k + 1, 20, 1e-8,
                                                              1e-4, 0))


@pytest.mark.parametrize("group", [0, 2])
def test_listed_chanblocks(oracle, group):
    ntiles, nt, nch = 20, 2, 9
    data, model, start = problem(ntiles, nt, nch)
    d, m = torch.from_numpy(data).cuda(), torch.from_numpy(model).cuda()
    dj = torch.from_numpy(start).cuda()
    listed = (ctypes.c_int * 3)(7, 0, 3)
    res = (_lib.HdcCalResult * nch)()
    with limit(max(1, group * cov_bytes(ntiles))):
        assert _lib.lib().hdc_calibrate_chanblocks(d.data_ptr(), m.data_ptr(), nt, 0, nt, nch, data.shape[2],
                                                   dj.data_ptr(), 20, 1e-8, 1e-4, 0, listed, 3, res, 0, None) == 0
    got = dj.cpu().numpy()
    want, ores = oracle.calibrate_timeblock(data, model, start, 0, nt, 20, 1e-8, 1e-4, 0)
    for c in range(nch):
        if c in (7, 0, 3):
            assert (res[c].num_iterations, bool(res[c].converged)) == (ores[c]["num_iterations"], ores[c]["converged"])
            assert np.linalg.norm(got[:, c] - want[:, c]) / np.linalg.norm(want[:, c]) < 1e-10
        else:
            np.testing.assert_array_equal(got[:, c], start[:, c])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_tensor_predict_with_the_least_workspace(dtype):
    """The same table values a channel at a time: the same visibilities."""
    centre, nf, ntiles = (0.0, -0.47), 7, 45
    sky = srclist.SkyModelArrays.from_components(synth.point_sky(130, centre, 10.0, 3))
    xyzs = synth.tiles_in_disk(ntiles, 600.0, 2)
    gains = np.random.default_rng(1).uniform(0.4, 1.0, (ntiles, 2, 16))
    out = []
    for nbytes in (0, 1):
        with limit(nbytes):
            m = SkyModeller(sky, xyzs, 167e6 + 1e6 * np.arange(nf), centre, synth.MWA_LAT_RAD, beam="per_tile",
                            form="tensor", dipole_gains=gains)
            vis = torch.zeros((nf, ntiles * (ntiles - 1) // 2, 8), dtype=dtype, device="cuda")
            for lst in (0.0, 0.01):
                m.model_timestep_with(lst, vis, return_uvws=False)
            torch.cuda.synchronize()
            m.close()
        out.append(vis.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])


def test_dropin_tensor_points_with_the_least_workspace(oracle):
    comps, a, _, beam, (nf, nbl), obs = dropin_inputs(oracle, 40, 5, 9, 0, 8, ntile_beams=7, want_obs=True)
    xyz = dev(obs.tile_xyzs)
    out = []
    for nbytes in (0, 1):
        vis = torch.zeros((nf, nbl, 8), dtype=torch.float32, device="cuda")
        with limit(nbytes):
            _lib.check_str(_lib.lib().model_points_tc(ctypes.byref(comps), ctypes.byref(a), xyz.data_ptr(),
                                                      float(obs.lsts[0]), _lib.RADec(*obs.phase_centre), beam,
                                                      vis.data_ptr()), "model_points_tc")
        torch.cuda.synchronize()
        out.append(vis.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
