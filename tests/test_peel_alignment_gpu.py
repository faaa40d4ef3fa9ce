"""A residual whose address is a multiple of 4 bytes only (a view into a larger
buffer): the source-by-source loop takes it as any other, the batched form
refuses it."""

import math

import numpy as np
import pytest

from mwa_hyperdrive_b200 import peel
from mwa_hyperdrive_b200 import srclist as sl
from mwa_hyperdrive_b200 import synth
from mwa_hyperdrive_b200._lib import HdcError

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

PC = (0.1, math.radians(-27.0))


def run(offset, comps, batched=False):
    rng = np.random.default_rng(3)
    ntiles, nt, nf = 19, 2, 6
    shape = (nt, nf, ntiles * (ntiles - 1) // 2, 8)
    flat = torch.zeros(math.prod(shape) + 8, device="cuda")
    resid = flat[offset:offset + math.prod(shape)].view(shape)
    resid.copy_(torch.from_numpy(rng.normal(0.0, 0.3, shape).astype(np.float32)))
    weights = torch.from_numpy(rng.uniform(0.1, 8.0, shape[:3]).astype(np.float32)).cuda()
    lsts = 0.12 + np.arange(nt) * 6e-4
    pos = [(PC[0] + 0.02, PC[1] - 0.01), (PC[0] - 0.01, PC[1] + 0.02)]
    skies = [sl.SkyModelArrays.from_components(
        [sl.SourceComponent(*p, sl.Point(), sl.PowerLaw(-0.8, sl.FluxDensity(150e6, 4.0 / comps)))] * comps)
        for p in pos]
    got = peel.peel_timeblock(resid, weights, 170e6 + np.arange(nf) * 640e3, synth.tiles_in_disk(ntiles, 750.0, 1), lsts,
                              float(lsts.mean()), PC, skies, pos, [peel.IonoConsts()] * 2, 2, 4, 1.0, 3,
                              synth.MWA_LAT_RAD, batched=batched)
    assert not flat[:offset].any() and not flat[offset + math.prod(shape):].any()
    return [(c.alpha, c.beta, c.gain) for c in got], resid.cpu().numpy()


# one component a source: the point table; two: materialised models
@pytest.mark.parametrize("comps", [1, 2])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_source_by_source(offset, comps):
    want, want_r = run(0, comps)
    got, got_r = run(offset, comps)
    assert got == want
    np.testing.assert_array_equal(got_r, want_r)


@pytest.mark.parametrize("offset", [1, 2])
def test_batched_refuses(offset):
    with pytest.raises(HdcError, match="multiple of 16 bytes"):
        run(offset, 1, batched=True)
