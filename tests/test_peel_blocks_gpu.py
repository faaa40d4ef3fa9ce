"""The batched peel's sweeps at the edges of their 32 x 32 blocks of tile
pairs, groups of sources and staged samples: points kept as one Jones per
(timestep, channel) against the same sources materialised (two halves of each
flux at one position), and against a float64 restatement of one pass."""

import math

import numpy as np
import pytest

from mwa_hyperdrive_b200 import peel as P
from mwa_hyperdrive_b200 import srclist as sl
from mwa_hyperdrive_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

PC = (0.1, math.radians(-27.0))
VEL_C = 299792458.0


def uvws(xyzs, lst, ra, dec):
    h = lst - ra
    s, c, sd, cd = math.sin(h), math.cos(h), math.sin(dec), math.cos(dec)
    x, y, z = xyzs.T
    t = np.stack([s * x + c * y, -sd * c * x + sd * s * y + cd * z, cd * c * x - cd * s * y + sd * z], -1)
    i, j = np.triu_indices(len(xyzs), 1)
    return t[i] - t[j]


def one_pass(resid, weights, freqs, xyzs, lsts, avg_lst, sources, favg, loops):
    """The batched pass in float64: every source fitted against the same
    residual, from unit constants."""
    nt, nf, nbl = resid.shape[:3]
    r = resid[..., 0::2].astype(np.float64) + 1j * resid[..., 1::2]
    w = weights.astype(np.float64)
    lam, nlo = VEL_C / freqs, nf // favg
    lam_lo = (VEL_C / freqs.reshape(nlo, favg).mean(1))[:, None]
    wsum = w.reshape(nt, nlo, favg, nbl).sum((0, 2))
    out, change = [], np.zeros_like(r)
    for ra, dec, flux in sources:
        d, m = np.zeros((nlo, nbl), complex), np.zeros((nlo, nbl), complex)
        for t in range(nt):
            dw = uvws(xyzs, lsts[t], ra, dec)[:, 2] - uvws(xyzs, lsts[t], *PC)[:, 2]
            rot = np.exp(-2j * np.pi * dw / lam[:, None])
            src = 2.0 * flux[:, None] * np.ones(nbl)
            d += ((((r[t, ..., 0] + r[t, ..., 3]) * rot + src) * w[t]).reshape(nlo, favg, nbl)).sum(1)
            m += (src * w[t]).reshape(nlo, favg, nbl).sum(1)
        d, m = d / wsum, m / wsum
        u, v, _ = uvws(xyzs, avg_lst, ra, dec).T
        a, b, g = 0.0, 0.0, 1.0
        for _ in range(loops):
            mi = m * g * np.exp(-2j * np.pi * (u * a + v * b) * lam_lo)
            mr, mm = mi.real * (d.imag - mi.imag), mi.real**2
            auu, auv, avv = ((wsum * mm * q * lam_lo**2).sum() for q in (u * u, u * v, v * v))
            au, av = ((wsum * mr * q * -lam_lo).sum() for q in (u, v))
            den = 2.0 * np.pi * (auu * avv - auv * auv)
            a, b = a + (au * avv - av * auv) / den, b + (av * auu - au * auv) / den
            g *= (wsum * mi.real * d.real).sum() / (wsum * mm).sum()
        out.append((a, b, g))
        for t in range(nt):
            q = uvws(xyzs, lsts[t], ra, dec)
            rot = np.exp(-2j * np.pi * (q[:, 2] - uvws(xyzs, lsts[t], *PC)[:, 2]) / lam[:, None])
            io = g * np.exp(-2j * np.pi * (q[:, 0] * a + q[:, 1] * b) * lam[:, None])
            for k in (0, 3):
                change[t, ..., k] += flux[:, None] * (1.0 - io) * rot.conj()
    return np.array(out), r + change


# tiles at and past the edges of a block; 1, one group and a group and a rest
# of sources, more than a staged chunk; samples of whole and part stages
@pytest.mark.parametrize("ntiles,nsrc,nt,favg", [(12, 1, 1, 3), (32, 4, 2, 4), (33, 5, 3, 2), (65, 18, 1, 5)])
def test_pass(ntiles, nsrc, nt, favg):
    rng = np.random.default_rng(ntiles)
    xyzs = synth.tiles_in_disk(ntiles, 750.0, ntiles)
    freqs = 170e6 + np.arange(2 * favg) * 640e3
    lsts = 0.12 + np.arange(nt) * 6e-4
    nbl = ntiles * (ntiles - 1) // 2
    i_ref = rng.uniform(2.0, 6.0, nsrc)
    pos = [(PC[0] + math.radians(rng.uniform(-3, 3)), PC[1] + math.radians(rng.uniform(-3, 3))) for _ in range(nsrc)]
    sources = [(p[0], p[1], i_ref[k] * (freqs / 150e6) ** -0.8) for k, p in enumerate(pos)]
    resid = rng.normal(0.0, 0.3, (nt, freqs.size, nbl, 8)).astype(np.float32)
    weights = rng.uniform(0.1, 8.0, (nt, freqs.size, nbl)).astype(np.float32)
    want, want_r = one_pass(resid, weights, freqs, xyzs, lsts, float(lsts.mean()), sources, favg, 6)

    def comps(k, halves):
        fd = sl.FluxDensity(150e6, i_ref[k] / halves)
        return sl.SkyModelArrays.from_components(
            [sl.SourceComponent(*pos[k], sl.Point(), sl.PowerLaw(-0.8, fd)) for _ in range(halves)])

    for halves in (1, 2):  # the point table, the materialised models
        d = torch.from_numpy(resid.copy()).cuda()
        got = P.peel_timeblock(d, torch.from_numpy(weights).cuda(), freqs, xyzs, lsts, float(lsts.mean()), PC,
                               [comps(k, halves) for k in range(nsrc)], pos, [P.IonoConsts()] * nsrc, 1, 6, 1.0, favg,
                               synth.MWA_LAT_RAD, batched=True)
        g = np.array([[c.alpha, c.beta, c.gain] for c in got])
        # FP32 phasors and sums of terms of unit size (1e-6 of the largest
        # offset and of the flux allows some ten roundings)
        assert np.max(np.abs(g[:, :2] - want[:, :2])) < 1e-5 * np.max(np.abs(want[:, :2])) + 1e-11
        assert np.max(np.abs(g[:, 2] - want[:, 2])) < 1e-5
        r = d.cpu().numpy().astype(np.float64)
        r = r[..., 0::2] + 1j * r[..., 1::2]
        assert np.max(np.abs(r - want_r)) < 1e-6 * 6.0 * nsrc


@pytest.mark.parametrize("halves", [1, 2])
@pytest.mark.parametrize("ntiles,nsrc,nt,favg", [(12, 1, 1, 3), (33, 3, 2, 5)])
def test_source_by_source(ntiles, nsrc, nt, favg, halves):
    """The source-by-source loop (FP64 steps, the reference's roundings) on the
    point table and on materialised models: one source is one pass in float64;
    several agree with batched sub-batches of one."""
    rng = np.random.default_rng(ntiles)
    xyzs = synth.tiles_in_disk(ntiles, 750.0, ntiles)
    freqs = 170e6 + np.arange(2 * favg) * 640e3
    lsts = 0.12 + np.arange(nt) * 6e-4
    nbl = ntiles * (ntiles - 1) // 2
    i_ref = rng.uniform(2.0, 6.0, nsrc)
    pos = [(PC[0] + math.radians(rng.uniform(-3, 3)), PC[1] + math.radians(rng.uniform(-3, 3))) for _ in range(nsrc)]
    resid = rng.normal(0.0, 0.3, (nt, freqs.size, nbl, 8)).astype(np.float32)
    weights = rng.uniform(0.1, 8.0, (nt, freqs.size, nbl)).astype(np.float32)
    skies = [sl.SkyModelArrays.from_components(
        [sl.SourceComponent(*pos[k], sl.Point(), sl.PowerLaw(-0.8, sl.FluxDensity(150e6, i_ref[k] / halves)))
         for _ in range(halves)]) for k in range(nsrc)]
    out = {}
    for batched in (False, True):
        d = torch.from_numpy(resid.copy()).cuda()
        got = P.peel_timeblock(d, torch.from_numpy(weights).cuda(), freqs, xyzs, lsts, float(lsts.mean()), PC, skies,
                               pos, [P.IonoConsts()] * nsrc, 2, 6, 1.0, favg, synth.MWA_LAT_RAD, batched=batched,
                               batch_size=1)
        out[batched] = np.array([[c.alpha, c.beta, c.gain] for c in got]), d.cpu().numpy()
    a, b = out[False], out[True]
    assert np.max(np.abs(a[0][:, :2] - b[0][:, :2])) < 1e-5 * np.max(np.abs(a[0][:, :2])) + 1e-11
    assert np.max(np.abs(a[0][:, 2] - b[0][:, 2])) < 1e-5
    assert np.max(np.abs(a[1] - b[1])) < 2e-6 * 6.0 * nsrc
    if nsrc == 1:
        d = torch.from_numpy(resid.copy()).cuda()
        got = P.peel_timeblock(d, torch.from_numpy(weights).cuda(), freqs, xyzs, lsts, float(lsts.mean()), PC, skies,
                               pos, [P.IonoConsts()], 1, 6, 1.0, favg, synth.MWA_LAT_RAD)
        want, want_r = one_pass(resid, weights, freqs, xyzs, lsts, float(lsts.mean()),
                                [(*pos[0], i_ref[0] * (freqs / 150e6) ** -0.8)], favg, 6)
        assert abs(got[0].alpha - want[0, 0]) < 1e-6 * np.max(np.abs(want[0, :2]))
        assert abs(got[0].gain - want[0, 2]) < 1e-6
        r = d.cpu().numpy().astype(np.float64)
        r = r[..., 0::2] + 1j * r[..., 1::2]
        assert np.max(np.abs(r - want_r)) < 1e-6 * 6.0
