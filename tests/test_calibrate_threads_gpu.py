"""Calibrations of arrays of different sizes on several host threads: the
kernel's shared-memory opt-in is one per device, so a small array's call must
not have a large one's retry launch refused (csrc/calibrate.cu, opt_in_smem),
and the stream on which calls capture their graphs and the collapsed forms'
covariances are one per device too."""

import threading

import numpy as np
import pytest

from mwa_hyperdrive_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from mwa_hyperdrive_b200 import calibrate as cal  # noqa: E402


def problem(ntiles, nt, nch):
    """The middle chanblock starts from zero gains: it fails the first pass,
    is seeded from its neighbours and converges in the retry."""
    rng = np.random.default_rng(ntiles)
    model = synth.random_model(nt, nch, ntiles * (ntiles - 1) // 2, rng)
    data = synth.corrupt(model, synth.truth_gains(ntiles, nch, rng), rng, 30.0)
    start = torch.zeros((ntiles, nch, 8), dtype=torch.float64, device="cuda")
    start[..., 0] = start[..., 6] = 1.0
    start[:, nch // 2] = 0.0
    return torch.from_numpy(data).cuda(), torch.from_numpy(model).cuda(), start


def solve(p, stream, form="plain"):
    data, model, start = p
    with torch.cuda.stream(stream):
        dj = start.clone()
        res = cal.calibrate_timeblock(data, model, dj, (0, data.shape[0]), 40, 1e-8, 1e-4, form=form, stream=stream)
    stream.synchronize()
    return dj.cpu().numpy(), [(r.num_iterations, r.converged) for r in res]


def beside(large, small, solve, repeats):
    """`large` solved `repeats` times while a thread each solves the small
    problems over and over on a stream of its own."""
    torch.cuda.synchronize()
    stop, errors = threading.Event(), []

    def others(p):
        try:
            torch.cuda.set_device(0)
            stream = torch.cuda.Stream()
            while not stop.is_set():
                solve(p, stream)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=others, args=(p,)) for p in small]
    for t in threads:
        t.start()
    try:
        got = [solve(large, torch.cuda.Stream()) for _ in range(repeats)]
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors, errors
    return got


def test_retry_beside_smaller_arrays():
    large = problem(200, 2, 5)
    torch.cuda.synchronize()
    want, counts = solve(large, torch.cuda.Stream())
    assert all(c for _, c in counts)
    for dj, c in beside(large, [problem(n, 1, 3) for n in (5, 9, 17)], solve, 40):
        assert c == counts
        np.testing.assert_array_equal(dj, want)


def solve_timeblocks(p, stream):
    data, model, _ = p
    out, results = cal.calibrate_timeblocks(data, model, [(t, t + 1) for t in range(data.shape[0])], 24, 1e-8, 1e-4,
                                            stream=stream)
    return out, [[(r.num_iterations, r.converged) for r in tb] for tb in results]


def test_graphs_beside_each_other():
    large = problem(60, 3, 5)
    torch.cuda.synchronize()
    want, counts = solve_timeblocks(large, torch.cuda.Stream())
    for out, c in beside(large, [problem(n, 2, 3) for n in (5, 9, 17)], solve_timeblocks, 60):
        assert c == counts
        np.testing.assert_array_equal(out, want)


# the last size needs more covariances than the buffer holds
@pytest.mark.parametrize("form", ["collapsed", "collapsed_f32"])
def test_covariances_beside_each_other(form):
    def run(p, stream):
        return solve(p, stream, form)

    large = problem(100, 2, 5)
    torch.cuda.synchronize()
    want, counts = run(large, torch.cuda.Stream())
    for dj, c in beside(large, [problem(n, 1, 3) for n in (5, 40, 256)], run, 40):
        assert c == counts
        np.testing.assert_array_equal(dj, want)
