"""The work that programs have this framework do, as measurable cases.

Every case runs a public entry point of the package on seeded synthetic
observations with the shapes of the repository's benchmark configurations and
of the ranges around them.  ``listed()`` gives the named cases, ``draw()``
more of the same ranges, ``prepare()`` the inputs and handles a program keeps,
``run()`` one pass, ``work()`` the bytes and operations a pass cannot do
without and ``exact()`` the outputs in 64 bits from plain torch and numpy.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from mwa_hyperdrive_b200 import calibrate as cal
from mwa_hyperdrive_b200 import peel as peel_mod
from mwa_hyperdrive_b200 import srclist, synth
from mwa_hyperdrive_b200.fee import FeeBeam
from mwa_hyperdrive_b200.model import SkyModeller
from mwa_hyperdrive_b200.warmstart import CENTRE, IN_DIM, OUT_DIM, WarmStartMLP

VEL_C = 299792458.0
PHASE_CENTRE = (0.0, math.radians(-27.0))
LATITUDE = synth.MWA_LAT_RAD
TIMESTEP_RAD = 8.0 * synth.SIDEREAL_RATE
CHANNEL0_HZ, CHANNEL_HZ = 167.0e6, 80.0e3


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _predict(name, form, beam, tiles, channels, timesteps, points, gaussians, shapelets, out="float32", host=False,
             unique=0):
    return {"name": name, "kind": "predict", "form": form, "beam": beam, "tiles": tiles, "channels": channels,
            "timesteps": timesteps, "points": points, "gaussians": gaussians, "shapelets": shapelets, "out": out,
            "host": host, "unique": unique}


def listed():
    return [
        # one coarse channel of a small point-source sky in the default form,
        # FP64 visibilities (the parity configuration): latency counts
        _predict("points_f64", "direct", "none", 128, 32, 1, 200, 0, 0, out="float64"),
        # the default form of new_sky_modeller on a calibrator field of every
        # component type, all fine channels of an observation at 80 kHz
        _predict("mixed_direct", "direct", "analytic", 128, 384, 1, 1000, 120, 24),
        # the benchmark's mixed sky in the chosen (tensor) form
        _predict("mixed_tensor", "tensor", "analytic", 128, 384, 2, 4000, 500, 100),
        # the same trait call on host buffers (upload, predict, download), an
        # odd count of tiles as flagging leaves it
        _predict("mixed_host", "tensor", "analytic", 123, 192, 1, 2100, 260, 50, host=True),
        # per-tile FEE beams: dead dipoles make 17 tiles' beams differ
        _predict("mixed_fee", "tensor", "fee", 128, 192, 1, 2000, 250, 50, unique=17),
        # DI calibration of one observation on the collapsed FP32 covariances
        {"name": "dical_f32", "kind": "dical", "form": "collapsed_f32", "tiles": 128, "chanblocks": 384,
         "timesteps": 8, "timeblocks": 1, "max_iterations": 50, "snr": 10.0},
        # the default form, a few timeblocks of ragged sizes
        {"name": "dical_plain", "kind": "dical", "form": "plain", "tiles": 113, "chanblocks": 100,
         "timesteps": 10, "timeblocks": 2, "max_iterations": 50, "snr": 30.0},
        # raw visibilities averaged to chanblocks and weighted before DI
        # calibration: bound by memory
        {"name": "prep", "kind": "prep", "tiles": 128, "channels": 768, "timesteps": 4, "average": 2, "flagged": 12},
        # peeling, every source of a pass fitted together
        {"name": "peel_batched", "kind": "peel", "batched": True, "batch": 0, "beam": "analytic", "tiles": 128,
         "channels": 384, "timesteps": 8, "average": 16, "sources": 30, "passes": 2, "loops": 10},
        # peeling in the reference's source-by-source order (the default)
        {"name": "peel_sequential", "kind": "peel", "batched": False, "batch": 0, "beam": "none", "tiles": 128,
         "channels": 192, "timesteps": 4, "average": 16, "sources": 6, "passes": 1, "loops": 10},
        # the FEE beam's Jones at a source list's directions
        {"name": "fee_jones", "kind": "fee", "directions": 4600, "unique": 12, "channels": 384, "degree": 16},
        # training the warm start: one mini-batch forward and backward
        {"name": "mlp_gradients", "kind": "mlp", "batch": 4096, "hidden": 256},
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["direct", "direct", "tensor", "tensor", "host", "fee_predict", "dical", "dical", "prep", "peel",
                       "peel", "fee", "mlp"])
    if kind in ("direct", "tensor", "host", "fee_predict"):
        tiles, channels = rng.randint(17, 160), size(8, 400)
        # the largest sky that a drawn array may have, so that no drawn case
        # costs more than the largest listed one
        budget = (3.0e9 if kind == "direct" else 9.0e9) / (channels * tiles * tiles / 2)
        points = max(1, min(size(20, 4000), int(budget)))
        gaussians = min(size(1, 500), int(budget / 8)) if rng.random() < 0.7 else 0
        shapelets = min(size(1, 100), int(budget / 40)) if rng.random() < 0.7 else 0
        form = "direct" if kind == "direct" else "tensor"
        beam = "fee" if kind == "fee_predict" else rng.choice(["none", "analytic"])
        if kind == "direct" and rng.random() < 0.2:
            beam = "fee"
        c = _predict("", form, beam, tiles, channels, 1, points, gaussians, shapelets,
                     out="float64" if kind == "direct" and rng.random() < 0.4 else "float32", host=kind == "host",
                     unique=rng.randint(2, min(24, tiles)) if beam == "fee" else 0)
        del c["name"]
        return c
    if kind == "dical":
        tiles, nt = rng.randint(17, 144), rng.randint(1, 14)
        form = rng.choice(["plain", "collapsed", "collapsed_f32"])
        most = int(1.2e7 / (nt * tiles * (tiles - 1) / 2))
        return {"kind": "dical", "form": form, "tiles": tiles, "chanblocks": min(size(8, 500), max(8, most)),
                "timesteps": nt, "timeblocks": rng.randint(1, min(2, nt)), "max_iterations": rng.choice([30, 50]),
                "snr": round(rng.uniform(8.0, 60.0), 2)}
    if kind == "prep":
        avg = rng.choice([1, 2, 4])
        chanblocks = size(16, 200)
        return {"kind": "prep", "tiles": rng.randint(17, 140), "channels": chanblocks * avg,
                "timesteps": rng.randint(1, 8), "average": avg, "flagged": rng.randint(0, chanblocks // 8)}
    if kind == "peel":
        batched = rng.random() < 0.5
        avg = rng.choice([4, 8, 16])
        return {"kind": "peel", "batched": batched, "batch": 0, "beam": rng.choice(["none", "analytic"]),
                "tiles": rng.randint(33, 128), "channels": avg * rng.randint(2, 10), "timesteps": rng.randint(1, 6),
                "average": avg, "sources": rng.randint(1, 24 if batched else 6), "passes": rng.randint(1, 2),
                "loops": rng.randint(4, 10)}
    if kind == "fee":
        return {"kind": "fee", "directions": size(30, 6000), "unique": rng.randint(1, 20), "channels": size(16, 384),
                "degree": rng.randint(6, 18)}
    return {"kind": "mlp", "batch": size(300, 30000), "hidden": rng.choice([128, 256])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _freqs(channels):
    return CHANNEL0_HZ + np.arange(channels) * CHANNEL_HZ


def _lsts(timesteps):
    return PHASE_CENTRE[0] + np.arange(timesteps) * TIMESTEP_RAD


def _sky(case, seed):
    comps = synth.point_sky(case["points"], PHASE_CENTRE, 10.0, seed, curved_q_sigma=0.2) if case["points"] else []
    return comps + synth.gaussians_and_shapelets(case["gaussians"], case["shapelets"], PHASE_CENTRE, seed + 1)


def _fee_inputs(channels, tiles, unique, degree, seed):
    """Coefficients, channel frequencies, delays and amplitudes: one pointing,
    `unique` - 1 tiles with a dead dipole (or two) of their own."""
    freqs = _freqs(channels)
    nfile = int(math.ceil((freqs[-1] - freqs[0]) / 1.28e6)) + 2
    coeffs = synth.fee_coeffs((166.4e6 + np.arange(nfile) * 1.28e6).astype(np.uint32), degree, seed=seed)
    delays = np.tile(np.array([(d % 4) * 3 + (d // 4) for d in range(16)], np.uint32), (tiles, 1))
    for t in range(1, unique):
        delays[t, (t * 5) % 16] = 32
        if t > 15:
            delays[t, (t * 5 + 7) % 16] = 32
    return coeffs, freqs, delays, np.ones((tiles, 32))


def _prepare_predict(case, seed):
    sky = srclist.SkyModelArrays.from_components(_sky(case, seed))
    xyzs = synth.tiles_in_disk(case["tiles"], 750.0, seed + 2)
    freqs = _freqs(case["channels"])
    fee = None
    if case["beam"] == "fee":
        fee = FeeBeam(*_fee_inputs(case["channels"], case["tiles"], case["unique"], 12, seed + 3))
    modeller = SkyModeller(sky, xyzs, freqs, PHASE_CENTRE, LATITUDE, beam=case["beam"], form=case["form"], fee_beam=fee)
    nbl = case["tiles"] * (case["tiles"] - 1) // 2
    shape = (case["timesteps"], case["channels"], nbl, 8)
    if case["host"]:
        vis = torch.zeros(shape, dtype=torch.float32, pin_memory=True).numpy()
    else:
        vis = torch.zeros(shape, dtype=getattr(torch, case["out"]), device="cuda")
    return {"case": case, "modeller": modeller, "vis": vis, "lsts": _lsts(case["timesteps"])}


def _rand_gains(gen, chanblocks, tiles):
    """[chanblock][tile][2][2] complex128: amplitudes near 1, a phase per tile
    and polarisation that drifts over the band, and a little leakage."""
    def normal(*shape):
        return torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)

    band = torch.linspace(0.0, 1.0, chanblocks, dtype=torch.float64, device="cuda")[:, None]
    g = torch.zeros((chanblocks, tiles, 2, 2), dtype=torch.complex128, device="cuda")
    for k in range(2):
        g[:, :, k, k] = torch.polar((1.0 + 0.1 * normal(1, tiles)).expand(chanblocks, -1).clone(),
                                    0.6 * normal(1, tiles) + 0.3 * normal(1, tiles) * band)
        g[:, :, k, 1 - k] = 0.01 * torch.complex(normal(chanblocks, tiles), normal(chanblocks, tiles))
    return g


def _mul(a, b):
    """Products of 2 x 2 matrices over leading dimensions that broadcast."""
    return (a[..., :, :, None] * b[..., None, :, :]).sum(-2)


def _herm(a):
    return a.conj().transpose(-1, -2)


def _prepare_dical(case, seed):
    nt, nch, tiles = case["timesteps"], case["chanblocks"], case["tiles"]
    nbl = tiles * (tiles - 1) // 2
    gen = torch.Generator(device="cuda").manual_seed(seed)
    model = synth.polarised_model_device(nt, nch, nbl, gen)
    i, j = (torch.from_numpy(x).cuda() for x in np.triu_indices(tiles, 1))
    g = _rand_gains(gen, nch, tiles).to(torch.complex64)
    gp, gq = g[:, i], _herm(g[:, j])
    data = torch.empty_like(model)
    for t in range(nt):
        m = torch.view_as_complex(model[t].reshape(nch, nbl, 4, 2)).reshape(nch, nbl, 2, 2)
        d = torch.view_as_real(_mul(_mul(gp, m), gq).reshape(nch, nbl, 4)).reshape(nch, nbl, 8)
        noise = d.square().mean().sqrt() / case["snr"]
        data[t] = d + noise * torch.randn(d.shape, device="cuda", generator=gen)
    step = nt // case["timeblocks"]
    bounds = [(k * step, (k + 1) * step if k + 1 < case["timeblocks"] else nt) for k in range(case["timeblocks"])]
    return {"case": case, "data": data, "model": model, "timeblocks": bounds}


def _prepare_prep(case, seed):
    nt, nf, nbl = case["timesteps"], case["channels"], case["tiles"] * (case["tiles"] - 1) // 2
    gen = torch.Generator(device="cuda").manual_seed(seed)
    vis = torch.randn((nt, nf, nbl, 8), device="cuda", generator=gen)
    weights = torch.rand((nt, nf, nbl), device="cuda", generator=gen) * 20.0 - 3.0  # some samples flagged (< 0)
    chunks = nf // case["average"]
    flagged = sorted(int(k) for k in np.random.default_rng(seed).choice(chunks, case["flagged"], replace=False))
    model = torch.randn((1, chunks - case["flagged"], nbl, 8), device="cuda", generator=gen)
    baseline_weights = torch.rand(nbl, dtype=torch.float64, device="cuda", generator=gen)
    return {"case": case, "vis": vis, "weights": weights, "flagged": flagged, "model": model,
            "model_work": torch.empty_like(model), "baseline_weights": baseline_weights}


def _peel_inputs(case, seed):
    """Tile positions, bright point sources and their true offsets."""
    xyzs = synth.tiles_in_disk(case["tiles"], 750.0, seed + 2)
    comps = synth.point_sky(40 * case["sources"], PHASE_CENTRE, 10.0, seed, ref_freq=150e6)
    comps = sorted(comps, key=lambda c: -c.flux_type.fd.i)[: case["sources"]]
    rng = np.random.default_rng(seed + 3)
    truths = [(rng.normal(0.0, 2e-5), rng.normal(0.0, 2e-5), rng.uniform(0.9, 1.1)) for _ in comps]
    return xyzs, comps, truths


def _prepare_peel(case, seed):
    xyzs, comps, truths = _peel_inputs(case, seed)
    nt, nf, tiles = case["timesteps"], case["channels"], case["tiles"]
    nbl = tiles * (tiles - 1) // 2
    freqs, lsts = _freqs(nf), _lsts(nt)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    resid = 0.1 * torch.randn((nt, nf, nbl, 8), device="cuda", generator=gen)
    rc = torch.view_as_complex(resid.reshape(nt, nf, nbl, 4, 2))
    geo = _PeelGeometry(case, xyzs, comps)
    for s, truth in enumerate(truths):
        for t in range(nt):
            factor = (geo.iono(s, t, truth) - 1.0) * geo.rotation(s, t).conj()  # [nf][nbl]
            rc[t] += (geo.model[s, t][:, None, :] * factor[..., None]).to(torch.complex64)
    weights = torch.rand((nt, nf, nbl), device="cuda", generator=gen) * 8.0 + 0.1
    return {"case": case, "resid": resid, "work": torch.empty_like(resid), "weights": weights, "freqs": freqs,
            "xyzs": xyzs, "lsts": lsts, "average_lst": float(np.mean(lsts)),
            "sources": [srclist.SkyModelArrays.from_components([c]) for c in comps],
            "positions": [(c.ra, c.dec) for c in comps]}


def _prepare_fee(case, seed):
    coeffs, freqs, delays, amps = _fee_inputs(case["channels"], case["unique"], case["unique"], case["degree"], seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["directions"]
    az = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * (2.0 * math.pi)
    za = torch.acos(0.05 + 0.95 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen))
    return {"case": case, "beam": FeeBeam(coeffs, freqs, delays, amps), "az": az, "za": za}


def _mlp_params(case, seed):
    """Trained-like weights of the 40 -> hidden x 3 -> 8 network."""
    rng = np.random.default_rng(seed)
    dims = [IN_DIM, case["hidden"], case["hidden"], case["hidden"], OUT_DIM]
    parts = []
    for i, o in zip(dims[:-1], dims[1:]):
        parts += [rng.normal(0.0, math.sqrt(2.0 / i), (o, i)), rng.normal(0.0, 0.02, o)]
    return dims, [p.astype(np.float32) for p in parts]


def _prepare_mlp(case, seed):
    _, parts = _mlp_params(case, seed)
    net = WarmStartMLP(hidden=case["hidden"], num_hidden=3, seed=0)
    net.set_params(np.concatenate([p.ravel() for p in parts]))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((case["batch"], IN_DIM), device="cuda", generator=gen)
    t = x[:, CENTRE:CENTRE + OUT_DIM] + 0.1 * torch.randn((case["batch"], OUT_DIM), device="cuda", generator=gen)
    return {"case": case, "net": net, "x": x, "t": t.contiguous()}


def prepare(case, seed):
    return {"predict": _prepare_predict, "dical": _prepare_dical, "prep": _prepare_prep, "peel": _prepare_peel,
            "fee": _prepare_fee, "mlp": _prepare_mlp}[case["kind"]](case, seed)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "predict":
        vis, m = state["vis"], state["modeller"]
        if case["host"]:
            vis[:] = 0.0
            for t, lst in enumerate(state["lsts"]):
                m.model_timestep_with_host(lst, vis[t])
        else:
            vis.zero_()
            for t, lst in enumerate(state["lsts"]):
                m.model_timestep_with(lst, vis[t], return_uvws=False)
        return vis
    if kind == "dical":
        sols, results = cal.calibrate_timeblocks(state["data"], state["model"], state["timeblocks"],
                                                 max_iterations=case["max_iterations"], form=case["form"])
        counts = np.array([[[r.num_iterations, r.converged, r.num_failed] for r in tb] for tb in results], np.int64)
        return {"solutions": sols, "counts": counts}
    if kind == "prep":
        to, wto = cal.vis_average(state["vis"], state["weights"], state["model"].shape[1], state["flagged"])
        model = state["model_work"].copy_(state["model"])
        data = to[None].contiguous()
        cal.scale_by_weights(data, model, wto[None].contiguous(), state["baseline_weights"])
        return {"weights": wto, "data": data, "model": model}
    if kind == "peel":
        work = state["work"].copy_(state["resid"])
        consts = peel_mod.peel_timeblock(
            work, state["weights"], state["freqs"], state["xyzs"], state["lsts"], state["average_lst"], PHASE_CENTRE,
            state["sources"], state["positions"], [peel_mod.IonoConsts() for _ in state["sources"]], case["passes"],
            case["loops"], 1.0, case["average"], LATITUDE, beam=case["beam"], batched=case["batched"],
            batch_size=case["batch"])
        # fitted from single-precision averages of the visibilities
        fitted = np.array([[c.alpha, c.beta, c.gain] for c in consts], np.float32)
        return {"residual": work, "alpha_beta": fitted[:, :2].copy(), "gain": fitted[:, 2].copy()}
    if kind == "fee":
        return state["beam"].calc_jones(state["az"], state["za"], LATITUDE)
    loss, grads = state["net"].gradients(state["x"], state["t"])
    return {"loss": np.float32(loss), "gradients": grads}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "predict":
        nbl = case["tiles"] * (case["tiles"] - 1) // 2
        nvis = nbl * case["channels"] * case["timesteps"]
        comps = case["points"] + case["gaussians"] + case["shapelets"]
        size = 64 if case["out"] == "float64" else 32
        # a component's phasor from its tiles' factors (6), four complex
        # products with B S B^H, an envelope where it has one (the shapelets'
        # with its 6 x 6 basis products)
        per_tile = 64 if case["beam"] == "fee" else 0
        flops = nvis * ((38.0 + per_tile) * comps + 8.0 * case["gaussians"] + 120.0 * case["shapelets"])
        return {"bytes": nvis * size * (2 if case["host"] else 1) + 64.0 * comps * case["channels"], "flops": flops}
    if kind == "dical":
        nvis = case["timesteps"] * case["chanblocks"] * case["tiles"] * (case["tiles"] - 1) // 2
        nper = nvis // case["timesteps"] * case["timeblocks"]
        return {"bytes": 64.0 * nvis, "flops": 176.0 * nvis + 380.0 * 0.5 * case["max_iterations"] * nper}
    if kind == "prep":
        nbl, nt = case["tiles"] * (case["tiles"] - 1) // 2, case["timesteps"]
        used = case["channels"] // case["average"] - case["flagged"]
        return {"bytes": 36.0 * nbl * (nt * used * case["average"] + used) + 64.0 * nbl * used,
                "flops": 20.0 * nbl * nt * used * case["average"]}
    if kind == "peel":
        nvis = case["timesteps"] * case["channels"] * case["tiles"] * (case["tiles"] - 1) // 2
        per = case["sources"] * case["passes"]
        sweeps = case["passes"] * (1 if case["batched"] else case["sources"])
        return {"bytes": 100.0 * nvis * sweeps, "flops": 150.0 * nvis * per}
    if kind == "fee":
        sets = case["unique"] * (1 + int(case["channels"] * CHANNEL_HZ / 1.28e6))
        modes = case["degree"] * (case["degree"] + 2)
        return {"bytes": 64.0 * sets * (case["directions"] + modes), "flops": 56.0 * sets * case["directions"] * modes}
    h = case["hidden"]
    params = IN_DIM * h + 2 * h * h + h * OUT_DIM
    return {"bytes": 4.0 * (case["batch"] * (IN_DIM + OUT_DIM) + 2 * params),
            "flops": 2.0 * case["batch"] * (3 * params - IN_DIM * h)}


# ---------------------------------------------------------------------------
# The outputs in 64 bits
# ---------------------------------------------------------------------------
def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _tile_uvws(xyzs, lst, ra, dec):
    h = lst - ra
    s, c, sd, cd = math.sin(h), math.cos(h), math.sin(dec), math.cos(dec)
    x, y, z = xyzs[:, 0], xyzs[:, 1], xyzs[:, 2]
    return np.stack([s * x + c * y, -sd * c * x + sd * s * y + cd * z, cd * c * x - cd * s * y + sd * z], -1)


def _azel(ra, dec, lst):
    h = lst - ra
    sl, cl = math.sin(LATITUDE), math.cos(LATITUDE)
    x = -np.sin(h) * np.cos(dec)
    y = -np.cos(h) * np.cos(dec) * sl + np.sin(dec) * cl
    z = np.cos(h) * np.cos(dec) * cl + np.sin(dec) * sl
    return np.arctan2(x, y) % (2.0 * math.pi), np.arctan2(z, np.hypot(x, y))


def _analytic_jones(az, el, freq):
    """The dipole-array tile over a ground plane, [comp][2][2]."""
    k = 2.0 * math.pi * freq / VEL_C
    sza, cza, saz, caz = np.cos(el), np.sin(el), np.sin(az), np.cos(az)
    l, m = sza * saz, sza * caz
    af = 0.25 * (np.cos(k * 0.55 * l) + np.cos(k * 1.65 * l)) * (np.cos(k * 0.55 * m) + np.cos(k * 1.65 * m))
    amp = af * (1.0 - np.exp(-2j * k * 0.278 * cza)) / (2.0 * abs(math.sin(k * 0.278)))
    p01 = (cza - 1.0) * saz * caz
    return (amp * np.array([[cza * saz**2 + caz**2, p01], [p01, cza * caz**2 + saz**2]])).transpose(2, 0, 1)


def _legendre(nmax, theta):
    """{(n, m): (P_n^m / sin theta, dP_n^m / d theta)} for 0 <= m <= n, with the
    Condon-Shortley phase, from R_n^m = P_n^m / sin^m theta."""
    x, s = np.cos(theta), np.sin(theta)
    out, cols, lead = {}, {}, -1.0
    for m in range(1, nmax + 2):
        r = {m: np.full_like(x, lead), m + 1: x * (2 * m + 1) * lead}
        for n in range(m + 2, nmax + 2):
            r[n] = ((2 * n - 1) * x * r[n - 1] - (n + m - 1) * r[n - 2]) / (n - m)
        cols[m] = r
        lead *= -(2 * m + 1)
    for n in range(1, nmax + 1):
        out[n, 0] = (np.zeros_like(x), s * cols[1][n])
        for m in range(1, n + 1):
            r = cols[m]
            out[n, m] = (s ** (m - 1) * r[n], s ** (m - 1) * ((n - m + 1) * r[n + 1] - (n + 1) * x * r[n]))
    return out


def _fee_exact(coeffs, freqs, delays, amps, az, za):
    """Jones [tile][file frequency used][direction][2][2] of distinct tiles,
    zenith-normalised and rotated by the parallactic angle, and the column of
    every channel."""
    file_f = coeffs["freqs_hz"].astype(np.int64)
    closest = np.array([int(np.argmin(np.abs(file_f - int(round(f))))) for f in freqs])
    used = np.unique(closest)
    modes = coeffs["modes"]
    nmax = int(modes[2].max())
    legs, zen = _legendre(nmax, za), _legendre(nmax, np.zeros(1))

    def basis(leg, phi, theta):
        u = np.cos(theta)
        bt, bp = [], []
        for s, m, n in modes.T.tolist():
            a = abs(m)
            c = math.sqrt(0.5 * (2 * n + 1) * math.exp(math.lgamma(n - a + 1) - math.lgamma(n + a + 1)))
            c *= ((-1.0) ** m if m > 0 else 1.0) / math.sqrt(n * (n + 1))
            e = c * np.exp(1j * m * phi) * 1j**n
            p1sin, p1 = leg[n, a]
            if s == 1:
                bt.append(e * p1sin * -m)
                bp.append(1j * e * (-a * u * p1sin - p1))
            else:
                bt.append(e * (p1sin * a * u + p1))
                bp.append(1j * e * p1sin * m)
        return np.stack(bt), np.stack(bp)

    phi = 0.5 * math.pi - az
    bt, bp = basis(legs, phi, za)
    out = np.empty((len(delays), len(used), len(az), 2, 2), np.complex128)
    norm = np.empty((len(used), 2, 2))
    for k, fi in enumerate(used):
        q = coeffs["q"][fi, ..., 0] + 1j * coeffs["q"][fi, ..., 1]  # [pol][dipole][mode]
        for p, (ph_t, ph_p) in enumerate([(0.0, -0.5 * math.pi), (0.5 * math.pi, 0.0)]):
            qz = q[p].sum(0)
            norm[k, p, 0] = abs(qz @ basis(zen, np.array([ph_t]), np.zeros(1))[0])[0]
            norm[k, p, 1] = abs(qz @ basis(zen, np.array([ph_p]), np.zeros(1))[1])[0]
        for t in range(len(delays)):
            dead = delays[t] == 32
            w = np.where(dead, 0.0, 1.0) * np.exp(-2j * math.pi * float(file_f[fi]) * np.where(dead, 0, delays[t])
                                                  * 435e-12)
            for p in range(2):
                qt = (w * amps[t, 16 * p:16 * p + 16]) @ q[p]
                out[t, k, :, p, 0] = (qt @ bt) / norm[k, p, 0]
                out[t, k, :, p, 1] = -(qt @ bp) / norm[k, p, 1]
    el = 0.5 * math.pi - za
    sp, cp = math.sin(LATITUDE), math.cos(LATITUDE)
    x = -np.cos(az) * np.cos(el) * sp + np.sin(el) * cp
    y = -np.sin(az) * np.cos(el)
    z = np.cos(az) * np.cos(el) * cp + np.sin(el) * sp
    ha, dec = np.arctan2(y, x), np.arctan2(z, np.hypot(x, y))
    pa = np.arctan2(cp * np.sin(ha), sp * np.cos(dec) - cp * np.sin(dec) * np.cos(ha)) + 0.5 * math.pi
    rot = np.array([[np.cos(pa), np.sin(pa)], [-np.sin(pa), np.cos(pa)]]).transpose(2, 0, 1)
    return out @ rot, np.searchsorted(used, closest)


def _shapelet_basis(orders):
    """The tabulated basis values [order][10001] that the model interpolates."""
    x = np.linspace(-50.0, 50.0, 10001)
    h = [np.ones_like(x), 2.0 * x]
    for n in range(2, orders):
        h.append(2.0 * x * h[-1] - 2.0 * (n - 1) * h[-2])
    norm = [1.0 / math.sqrt(2.0**n * math.factorial(n)) for n in range(orders)]
    return _cuda(np.stack([np.exp(-0.5 * x * x) * norm[n] * h[n] for n in range(orders)]))


def _components(case, seed):
    comps = _sky(case, seed)
    ra = np.array([c.ra for c in comps])
    dec = np.array([c.dec for c in comps])
    pra, pdec = PHASE_CENTRE
    lmn = np.stack([np.cos(dec) * np.sin(ra - pra),
                    np.sin(dec) * math.cos(pdec) - np.cos(dec) * math.sin(pdec) * np.cos(ra - pra),
                    np.sin(dec) * math.sin(pdec) + np.cos(dec) * math.cos(pdec) * np.cos(ra - pra) - 1.0])
    return comps, ra, dec, _cuda(lmn)


def _stokes_i(comps, freq):
    r = np.array([freq / c.flux_type.fd.freq for c in comps])
    si = np.array([c.flux_type.si for c in comps])
    q = np.array([getattr(c.flux_type, "q", 0.0) for c in comps])
    return np.array([c.flux_type.fd.i for c in comps]) * r**si * np.exp(q * np.log(r) ** 2)


def _exact_predict(case, seed):
    comps, ra, dec, lmn = _components(case, seed)
    tiles, freqs, lsts = case["tiles"], _freqs(case["channels"]), _lsts(case["timesteps"])
    xyzs = synth.tiles_in_disk(tiles, 750.0, seed + 2)
    i, j = (torch.from_numpy(x).cuda() for x in np.triu_indices(tiles, 1))
    npt, ng, ns = case["points"], case["gaussians"], case["shapelets"]
    extended = [c.comp_type for c in comps[npt:]]
    maj, mnr, pa = (np.array([getattr(e, k) for e in extended]) for k in ("maj", "min", "pa"))
    fee = None
    if case["beam"] == "fee":
        fee = _fee_inputs(case["channels"], tiles, case["unique"], 12, seed + 3)
    if ns:
        basis = _shapelet_basis(6)
        coeff = np.zeros((ns, 6, 6), np.complex128)
        for k, e in enumerate(extended[ng:]):
            for co in e.coeffs:
                coeff[k, co.n1, co.n2] += co.value * 1j ** (co.n1 + co.n2)
        coeff = _cuda(coeff)
    vis = torch.zeros((len(lsts), len(freqs), i.numel(), 4), dtype=torch.complex128, device="cuda")
    for t, lst in enumerate(lsts):
        uvw = _cuda(_tile_uvws(xyzs, lst, *PHASE_CENTRE))
        uvw = uvw[i] - uvw[j]  # [bl][3] metres
        path = uvw @ lmn
        az, el = _azel(ra, dec, lst)
        if fee is not None:
            fee_j, col = _fee_exact(fee[0], freqs, fee[2][: case["unique"]], fee[3], az, 0.5 * math.pi - el)
            tile_row = torch.from_numpy(np.where(np.arange(tiles) < case["unique"], np.arange(tiles), 0)).cuda()
            fee_j = _cuda(fee_j)
        if ng:
            gp, gm = slice(0, ng), (math.pi / 2) ** 2 / math.log(2.0)
            sp, cp = _cuda(np.sin(pa[gp])), _cuda(np.cos(pa[gp]))
            kx, ky = uvw[:, :1] * sp + uvw[:, 1:2] * cp, uvw[:, :1] * cp - uvw[:, 1:2] * sp
            gexp = -gm * (_cuda(maj[gp] ** 2) * kx * kx + _cuda(mnr[gp] ** 2) * ky * ky)
        if ns:
            suv = np.stack([_tile_uvws(xyzs, lst, c.ra, c.dec)[:, :2] for c in comps[npt + ng:]], 1)  # [tile][comp][2]
            suv = _cuda(suv)
            suv = suv[i] - suv[j]
            sp, cp = _cuda(np.sin(pa[ng:])), _cuda(np.cos(pa[ng:]))
            scale = math.sqrt(math.pi**2 / (2.0 * math.log(2.0))) / 0.01
            sx = (suv[..., 0] * sp + suv[..., 1] * cp) * _cuda(maj[ng:] * scale)
            sy = (suv[..., 0] * cp - suv[..., 1] * sp) * _cuda(-mnr[ng:] * scale)
        for f, freq in enumerate(freqs):
            ool = freq / VEL_C
            arg = (2.0 * math.pi * ool) * path
            z = torch.complex(torch.cos(arg), torch.sin(arg))
            if ng:
                z[:, npt:npt + ng] *= torch.exp(gexp * ool**2)
            if ns:
                vals = []
                for s in (sx, sy):
                    pos = s * ool + 5000.0
                    k = pos.floor().clamp(0, 9999).long()
                    frac = pos - pos.floor()
                    lo = basis[:, k]
                    vals.append(lo + (basis[:, k + 1] - lo) * frac)  # [order][bl][comp]
                env = torch.zeros_like(z[:, npt + ng:])
                for n1 in range(6):
                    inner = sum(coeff[:, n1, n2] * vals[1][n2] for n2 in range(6))
                    env += vals[0][n1] * inner
                z[:, npt + ng:] *= env
            flux = _cuda(_stokes_i(comps, freq))
            if fee is None:
                b = np.tile(np.eye(2, dtype=np.complex128), (len(comps), 1, 1)) if case["beam"] == "none" else \
                    _analytic_jones(az, el, freq)
                w = _cuda(b @ b.conj().transpose(0, 2, 1)) * flux[:, None, None]
                vis[t, f] = z @ w.reshape(-1, 4)
            else:
                b = fee_j[:, int(col[f])]  # [unique][comp][2][2]
                z = z * flux
                # visibilities of every (row of unique beams) x (row of unique
                # beams) at once: baselines grouped by their tiles' beams
                key = tile_row[i] * case["unique"] + tile_row[j]
                for pair in torch.unique(key).tolist():
                    at = (key == pair).nonzero()[:, 0]
                    w = _mul(b[pair // case["unique"]], _herm(b[pair % case["unique"]]))
                    vis[t, f, at] = z[at] @ w.reshape(-1, 4)
    out = torch.view_as_real(vis).reshape(*vis.shape[:3], 8)
    return out.cpu().numpy() if case["host"] else out


def _exact_dical(case, seed):
    s = _prepare_dical(case, seed)
    tiles, nch = case["tiles"], case["chanblocks"]
    nbl = tiles * (tiles - 1) // 2
    i, j = (torch.from_numpy(x).cuda() for x in np.triu_indices(tiles, 1))
    out = np.empty((len(s["timeblocks"]), tiles, nch, 8))
    for k, (t0, t1) in enumerate(s["timeblocks"]):
        for c0 in range(0, nch, 64):
            c1 = min(nch, c0 + 64)
            n = c1 - c0
            x = torch.zeros((n, nbl, 4, 4), dtype=torch.complex128, device="cuda")
            c = torch.zeros_like(x)
            for t in range(t0, t1):
                d, m = (torch.view_as_complex(s[key][t, c0:c1].double().reshape(n, nbl, 4, 2)) for key in ("data", "model"))
                x += d[..., :, None] * m.conj()[..., None, :]
                c += m[..., :, None] * m.conj()[..., None, :]
            x, c = (v.reshape(n, nbl, 2, 2, 2, 2) for v in (x, c))  # [i][k][j][l] = sum a_ik conj(b_jl)
            g = torch.eye(2, dtype=torch.complex128, device="cuda").expand(n, tiles, 2, 2).clone()
            old = torch.zeros_like(g)
            live = torch.ones(n, dtype=torch.bool, device="cuda")
            prec = torch.full((n, tiles, 2, 2), 1e9, dtype=torch.float64, device="cuda")
            for it in range(1, case["max_iterations"] + 1):
                h = _mul(_herm(g), g)

                def sums(cov, a):
                    """Each baseline's two terms of cov with the tiles' matrices a
                    (the second conjugated)."""
                    return ((cov * a[:, j][:, :, None, :, None, :]).sum((3, 5)),
                            (cov * a[:, i].conj()[:, :, :, None, :, None]).sum((2, 4)))

                # tile 1: D (G_q M^H), (G_q M^H)^H (G_q M^H); tile 2: D^H (G_p M), (G_p M)^H (G_p M)
                t1s, t2s = sums(x, g)
                b1s, b2s = sums(c, h)
                top = torch.zeros_like(g).index_add_(1, i, t1s).index_add_(1, j, t2s.conj())
                bot = torch.zeros_like(g).index_add_(1, i, b1s).index_add_(1, j, b2s.conj())
                det = bot[..., 0, 0] * bot[..., 1, 1] - bot[..., 0, 1] * bot[..., 1, 0]
                inv = torch.stack([bot[..., 1, 1], -bot[..., 0, 1], -bot[..., 1, 0], bot[..., 0, 0]], -1)
                new = _mul(top, inv.reshape(n, tiles, 2, 2) / det[..., None, None])
                if it % 2 == 0:
                    step = (new - old).abs().square()
                    prec = torch.where(live[:, None, None, None], step, prec)
                    new = 0.5 * (new + old)
                g = torch.where(live[:, None, None, None], new, g)
                if it % 2 == 0:
                    live &= ~(prec < 1e-8).flatten(1).all(1)
                    if not live.any():
                        break
                old = g.clone()
            fine = (prec.flatten(1).max(1).values <= 1e-4)[:, None, None, None]
            g = torch.where(fine, g, torch.full_like(g, complex(math.nan, math.nan)))
            out[k, :, c0:c1] = torch.view_as_real(g.reshape(n, tiles, 4)).reshape(n, tiles, 8).transpose(0, 1).cpu().numpy()
    return {"solutions": out, "counts": None}


def _exact_prep(case, seed):
    s = _prepare_prep(case, seed)
    chunks = case["channels"] // case["average"]
    keep = [k for k in range(chunks) if k not in set(s["flagged"])]
    data, wts = torch.empty_like(s["model"], dtype=torch.float64), []
    for o, k in enumerate(keep):
        ch = slice(k * case["average"], (k + 1) * case["average"])
        v, w = s["vis"][:, ch].double().flatten(0, 1), s["weights"][:, ch].double().flatten(0, 1)
        pos = torch.where(w > 0, w, torch.zeros_like(w))
        total = pos.sum(0)
        mean = torch.where(total[:, None] > 0, (v * pos[..., None]).sum(0) / total.clamp(min=1e-300)[:, None], v.mean(0))
        wts.append(torch.where(total > 0, total, -w.abs().sum(0)))
        data[0, o] = mean
    w = torch.stack(wts)
    scale = torch.where(w > 0, w * s["baseline_weights"], torch.zeros_like(w))[None, ..., None]
    return {"weights": w, "data": data * scale, "model": s["model"].double() * scale}


class _PeelGeometry:
    """Phases of the peel's sources on every baseline, and their apparent
    Jones [source][timestep][channel][4] (a source alone at its own position
    has the same model on every baseline)."""

    def __init__(self, case, xyzs, comps):
        self.lam = _cuda(VEL_C / _freqs(case["channels"]))[:, None]
        i, j = np.triu_indices(case["tiles"], 1)
        lsts = _lsts(case["timesteps"])

        def bl(lst, ra, dec):
            u = _tile_uvws(xyzs, lst, ra, dec)
            return u[i] - u[j]

        centre = [bl(lst, *PHASE_CENTRE) for lst in lsts]
        self.uvw = [[_cuda(bl(lst, c.ra, c.dec).T) for lst in lsts] for c in comps]
        self.dw = [[_cuda(bl(lst, c.ra, c.dec)[:, 2] - centre[t][:, 2]) for t, lst in enumerate(lsts)] for c in comps]
        mean_lst = float(np.mean(lsts))
        self.uv_lo = [_cuda(bl(mean_lst, c.ra, c.dec).T) for c in comps]
        freqs = _freqs(case["channels"])
        model = np.zeros((len(comps), len(lsts), len(freqs), 2, 2), np.complex128)
        ra, dec = np.array([c.ra for c in comps]), np.array([c.dec for c in comps])
        for f, freq in enumerate(freqs):
            flux = _stokes_i(comps, freq)[:, None, None]
            for t, lst in enumerate(lsts):
                b = np.eye(2)[None] if case["beam"] == "none" else _analytic_jones(*_azel(ra, dec, lst), freq)
                model[:, t, f] = flux * (b @ b.conj().transpose(0, 2, 1))
        self.model = _cuda(model.reshape(len(comps), len(lsts), len(freqs), 4))

    def rotation(self, s, t):
        return torch.exp(-2j * math.pi * self.dw[s][t][None] / self.lam)

    def iono(self, s, t, consts):
        u, v, _ = self.uvw[s][t]
        return consts[2] * torch.exp(-2j * math.pi * (u * consts[0] + v * consts[1])[None] * self.lam)


def _exact_peel(case, seed):
    s = _prepare_peel(case, seed)
    xyzs, comps, _ = _peel_inputs(case, seed)
    geo = _PeelGeometry(case, xyzs, comps)
    nt, nf, avg = case["timesteps"], case["channels"], case["average"]
    nlo, ns = nf // avg, len(comps)
    nbl = geo.dw[0][0].numel()
    r = torch.view_as_complex(s["resid"].double().reshape(nt, nf, nbl, 4, 2))
    w = s["weights"].double()
    lam_lo = _cuda(VEL_C / s["freqs"].reshape(nlo, avg).mean(1))[:, None]
    wsum = w.reshape(nt, nlo, avg, nbl).sum((0, 2))
    consts = [[0.0, 0.0, 1.0] for _ in comps]
    batch = ns if case["batched"] and not case["batch"] else (case["batch"] or 1)
    for _ in range(case["passes"]):
        for b0 in range(0, ns, batch):
            group = range(b0, min(ns, b0 + batch))
            fitted = {}
            for k in group:
                d = torch.zeros((nlo, nbl), dtype=torch.complex128, device="cuda")
                m = torch.zeros_like(d)
                for t in range(nt):
                    src = (geo.model[k, t, :, 0] + geo.model[k, t, :, 3])[:, None] * geo.iono(k, t, consts[k])
                    obs = (r[t, ..., 0] + r[t, ..., 3]) * geo.rotation(k, t) + src
                    d += (obs * w[t]).reshape(nlo, avg, nbl).sum(1)
                    m += (src * w[t]).reshape(nlo, avg, nbl).sum(1)
                d, m = d / wsum, m / wsum
                u, v, _ = geo.uv_lo[k]
                a, b, g = 0.0, 0.0, 1.0
                for _ in range(case["loops"]):
                    mi = m * (g * torch.exp(-2j * math.pi * (u * a + v * b)[None] * lam_lo))
                    mr, mm = mi.real * (d.imag - mi.imag), mi.real**2
                    l2 = lam_lo**2
                    auu, auv, avv = ((wsum * mm * q * l2).sum().item() for q in (u * u, u * v, v * v))
                    au, av = ((wsum * mr * q * -lam_lo).sum().item() for q in (u, v))
                    vm, mms = (wsum * mi.real * d.real).sum().item(), (wsum * mm).sum().item()
                    den = 2.0 * math.pi * (auu * avv - auv * auv)
                    a, b, g = a + (au * avv - av * auv) / den, b + (av * auu - au * auv) / den, g * (vm / mms)
                    if g < 0.0:
                        break
                new = [consts[k][0] + a, consts[k][1] + b, consts[k][2] * g]
                if abs(new[0]) > 1e-3 or abs(new[1]) > 1e-3 or not 0.0 <= new[2] <= 1.5:
                    new = consts[k]
                fitted[k] = new
            for k in group:
                for t in range(nt):
                    change = (geo.iono(k, t, consts[k]) - geo.iono(k, t, fitted[k])) * geo.rotation(k, t).conj()
                    r[t] += geo.model[k, t][:, None, :] * change[..., None]
                consts[k] = fitted[k]
    c = np.array(consts)
    return {"residual": torch.view_as_real(r).reshape(nt, nf, nbl, 8), "alpha_beta": c[:, :2].copy(),
            "gain": c[:, 2].copy()}


def _exact_fee(case, seed):
    coeffs, freqs, delays, amps = _fee_inputs(case["channels"], case["unique"], case["unique"], case["degree"], seed)
    s = _prepare_fee(case, seed)
    j, _ = _fee_exact(coeffs, freqs, delays, amps, s["az"].cpu().numpy(), s["za"].cpu().numpy())
    return j.reshape(*j.shape[:3], 4).view(np.float64)


def _exact_mlp(case, seed):
    dims, parts = _mlp_params(case, seed)
    s = _prepare_mlp(case, seed)
    params = [torch.from_numpy(p).double().cuda().requires_grad_(True) for p in parts]
    x = s["x"].double()
    y = x
    for k in range(len(dims) - 1):
        y = y @ params[2 * k].T + params[2 * k + 1]
        if k + 2 < len(dims):
            y = torch.relu(y)
    loss = (y + x[:, CENTRE:CENTRE + OUT_DIM] - s["t"].double()).square().mean()
    grads = torch.autograd.grad(loss, params)
    return {"loss": np.float64(loss.item()), "gradients": torch.cat([g.flatten() for g in grads]).cpu().numpy()}


def exact(case, seed):
    return {"predict": _exact_predict, "dical": _exact_dical, "prep": _exact_prep, "peel": _exact_peel,
            "fee": _exact_fee, "mlp": _exact_mlp}[case["kind"]](case, seed)
