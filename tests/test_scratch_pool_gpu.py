"""Device memory that the library keeps between calls: its pool holds on to no
more than 1 GiB of freed scratch (csrc/runtime.cu, POOL_KEEP)."""

import numpy as np
import pytest

from mwa_hyperdrive_b200 import srclist, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import peel  # noqa: E402

CENTRE = (0.0, -0.47)


def run_peel(sources, tiles, channels, timesteps):
    comps = synth.point_sky(sources, CENTRE, 10.0, 3)
    resid = torch.zeros((timesteps, channels, tiles * (tiles - 1) // 2, 8), device="cuda")
    weights = torch.ones(resid.shape[:3], device="cuda")
    lmsts = 1e-4 * np.arange(timesteps)
    return peel.peel_timeblock(resid, weights, 167e6 + 8e4 * np.arange(channels), synth.tiles_in_disk(tiles, 750.0, 1),
                               lmsts, float(lmsts.mean()), CENTRE,
                               [srclist.SkyModelArrays.from_components([c]) for c in comps],
                               [(c.ra, c.dec) for c in comps], [peel.IonoConsts() for _ in comps], 1, 2, 1.0, 16,
                               synth.MWA_LAT_RAD, batched=True)


def free_bytes():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_scratch_beyond_the_bound_is_given_back():
    run_peel(2, 8, 16, 1)
    before = free_bytes()
    # two tables of sources x timesteps x channels x tiles x 16 bytes: 1.2 GB,
    # and 0.5 GB of low-resolution traces
    run_peel(400, 128, 192, 4)
    kept = before - free_bytes()
    assert kept <= (1 << 30) + (32 << 20), kept


def test_a_peel_that_cannot_fit_is_refused_before_it_allocates():
    """40000 sources' phasor tables are 2 x 126 GB; their models 1 GB."""
    from mwa_hyperdrive_b200._lib import HdcError

    tiles, channels, timesteps, sources = 128, 384, 4, 40000
    assert torch.cuda.mem_get_info()[1] < 2 * 16 * sources * timesteps * channels * tiles
    before = free_bytes()
    with pytest.raises(HdcError, match=r"status 3.*device memory"):  # HDC_ERR_ALLOC
        run_peel(sources, tiles, channels, timesteps)
    assert before - free_bytes() <= 32 << 20
