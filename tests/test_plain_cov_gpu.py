"""The plain calibration form on call-scoped covariances (csrc/calibrate.cu,
PlainCov): more chanblocks than one group of scratch holds, listed chanblocks
and retries give the collapsed FP64 form's solutions bit for bit."""

import ctypes

import numpy as np
import pytest

from mwa_hyperdrive_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import _lib  # noqa: E402
from mwa_hyperdrive_b200 import calibrate as cal  # noqa: E402


def problem(ntiles, nt, nch, seed=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    model = synth.polarised_model_device(nt, nch, ntiles * (ntiles - 1) // 2, gen)
    g = synth.truth_gains(ntiles, nch, np.random.default_rng(seed))
    data = synth.corrupt_device(model, g)
    data[:, 1] = torch.randn(data[:, 1].shape, device="cuda", generator=gen)  # a chanblock that fails
    return data, model


def identity(ntiles, nch):
    dj = torch.zeros((ntiles, nch, 8), dtype=torch.float64, device="cuda")
    dj[..., 0] = dj[..., 6] = 1.0
    return dj


# 256 tiles: 80 chanblocks a group; 200: 119; a group of one wave and a
# remainder; a single timestep and several
@pytest.mark.parametrize("ntiles,nt,nch", [(256, 1, 81), (200, 2, 121), (17, 3, 5), (2, 1, 3)])
def test_groups(ntiles, nt, nch):
    data, model = problem(ntiles, nt, nch)
    out = {}
    for form in ("plain", "collapsed"):
        dj = identity(ntiles, nch)
        res = cal.calibrate_timeblock(data, model, dj, (0, nt), 14, 1e-8, 1e-4, form=form)
        many, _ = cal.calibrate_timeblocks(data, model, [(0, nt), (nt - 1, nt)], 14, 1e-8, 1e-4, form=form)
        out[form] = (dj.cpu().numpy(), [(r.num_iterations, r.converged, r.num_failed) for r in res], many)
    np.testing.assert_array_equal(out["plain"][0], out["collapsed"][0])
    assert out["plain"][1] == out["collapsed"][1]
    np.testing.assert_array_equal(out["plain"][2], out["collapsed"][2])


def test_listed_chanblocks():
    ntiles, nt, nch = 20, 2, 9
    data, model = problem(ntiles, nt, nch)
    listed = (ctypes.c_int * 3)(7, 0, 4)
    got = {}
    for form in (0, 1):
        dj = identity(ntiles, nch)
        res = (_lib.HdcCalResult * nch)()
        rc = _lib.lib().hdc_calibrate_chanblocks(data.data_ptr(), model.data_ptr(), nt, 0, nt, nch, data.shape[2],
                                                 dj.data_ptr(), 20, 1e-8, 1e-4, 0, listed, 3, res, form, None)
        assert rc == 0
        got[form] = dj.cpu().numpy()
    np.testing.assert_array_equal(got[0], got[1])
    untouched = [c for c in range(nch) if c not in (7, 0, 4)]
    np.testing.assert_array_equal(got[0][:, untouched], identity(ntiles, nch).cpu().numpy()[:, untouched])
