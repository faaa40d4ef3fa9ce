"""FP64 covariance forms around the tile count where the iteration kernel goes
from one group of threads to two (csrc/calibrate.cu, ONE_GROUP_TILES), against
the CPU oracle, with a chanblock that is retried; the forms' usual bounds."""

import numpy as np
import pytest

from mwa_hyperdrive_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import calibrate as cal  # noqa: E402


@pytest.mark.parametrize("form", ["plain", "collapsed"])
@pytest.mark.parametrize("ntiles", [2, 6, 15, 16, 17, 32, 33, 47, 48, 49, 64, 65])
def test_against_the_oracle(oracle, ntiles, form):
    rng = np.random.default_rng(ntiles)
    nt, nch = 2, 5
    model = synth.random_model(nt, nch, ntiles * (ntiles - 1) // 2, rng)
    data = synth.corrupt(model, synth.truth_gains(ntiles, nch, rng), rng, 20.0)
    start = np.zeros((ntiles, nch, 8))
    start[..., 0] = start[..., 6] = 1.0
    start[:, 2] = 0.0
    dj = torch.from_numpy(start).cuda()
    res = cal.calibrate_timeblock(torch.from_numpy(data).cuda(), torch.from_numpy(model).cuda(), dj, (0, nt), 30, 1e-8,
                                  1e-4, form=form)
    got = dj.cpu().numpy()
    want, ores = oracle.calibrate_timeblock(data, model, start, 0, nt, 30, 1e-8, 1e-4, 0)
    assert [(r.num_iterations, r.converged, r.num_failed) for r in res] == \
        [(r["num_iterations"], r["converged"], r["num_failed"]) for r in ores]
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    if ok.any():
        assert np.linalg.norm(got[ok] - want[ok]) / np.linalg.norm(want[ok]) < 1e-9
