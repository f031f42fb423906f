"""Far-field phases exp(-i k s) of a lossy medium where Im(k) s nears and leaves the
range of a double: the fields of given charges of a particle moved by s along the
direction carry the factor exp(-i k s), exactly up to exp(709), and beyond the range they
are infinite or NaN, not a finite number.

Tolerance: relative 1e-9 for the charges' own sum (FP64) and the argument k s of about
700, whose rounding gives 700 u ~ 1e-13."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

pytestmark = pytest.mark.gpu
EPS = (1.0 + 5.0j) ** 2
ENEI = 10.0


def fields(shift):
    v, f = shapes.trisphere(60, 1e-3)
    v = v + np.array([0.0, 0.0, shift])
    cp = m.comparticle([m.epsconst(EPS), m.epsconst(2.0)], [m.particle(v, f)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64"))
    rng = np.random.default_rng(1)
    n = cp.n
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)) * 1e-6
    sig = m.compstruct(cp, ENEI, sig1=c(n, 1), sig2=c(n, 1), h1=c(n, 3, 1), h2=c(n, 3, 1))
    far = m.spectrumret(medium=1).farfield(bem, sig, dir=[[0, 0, 1.0]])
    return far.e[0, :, 0], far.h[0, :, 0]


def test_growth_of_the_phase(gpu_lib):
    k = 2 * np.pi / ENEI * np.sqrt(complex(EPS))
    e0, h0 = fields(0.0)
    for x in (-600.0, -100.0, 300.0, 690.0, 705.0, 708.9):
        s = x / k.imag
        e, h = fields(s)
        with np.errstate(over="ignore"):
            want = np.exp(-1j * k * s)
        for a, b in ((e, e0), (h, h0)):
            big = np.abs(b) > 1e-3 * np.abs(b).max()
            assert np.all(np.abs(a[big] / (b[big] * want) - 1) < 1e-9), x
    for x in (715.0, 760.0, 1500.0, 3000.0, 1e6):
        e, h = fields(x / k.imag)
        assert not np.any(np.isfinite(e[np.abs(e0) > 1e-3 * np.abs(e0).max()])), x
