"""The FP64 phasor's polynomials (csrc/common.cuh, phasor_quarter_f64): the
constants the kernels hold and their accuracy, no GPU."""

import re
from pathlib import Path

import numpy as np

from mwa_hyperdrive_b200 import phasor_poly

SRC = Path(__file__).resolve().parents[1] / "mwa_hyperdrive_b200" / "csrc" / "common.cuh"


def test_kernel_holds_the_fitted_constants():
    vals = {name: float(v) for name, v in re.findall(r"(Q[SC]\d) = ([-+0-9.e]+)", SRC.read_text())}
    s, c = phasor_poly.fit64()
    for prefix, fitted in (("QS", s), ("QC", c)):
        held = np.array([vals[f"{prefix}{i}"] for i in range(fitted.size)])
        # printed to 18 digits; the last terms' own rounding moves them by ulps
        np.testing.assert_allclose(held, fitted, rtol=1e-9 if prefix == "QS" else 1e-9)
        np.testing.assert_allclose(held[:3], fitted[:3], rtol=4e-16)


def test_within_an_ulp():
    s, c = phasor_poly.fit64()
    r = np.linspace(-0.5, 0.5, 400_001)
    sn, cs = phasor_poly.evaluate_f64(r, s, c)
    x = r.astype(np.longdouble) * (np.longdouble("3.14159265358979323846264338327950288") / 2)
    ulp = 2.0**-52
    assert np.max(np.abs(sn - np.sin(x))) < ulp and np.max(np.abs(cs - np.cos(x))) < ulp
