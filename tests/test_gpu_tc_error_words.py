"""Expired waits of the tensor-core pipelines inside sweeps: the error words of the
lanes, set by the host as an expired wait leaves them (no wait runs out), are reported
once by the next call whatever ran before it (first call, kept graph, a graph built for
another wavelength list, host-scheduled lanes), in both precisions, and the calls after
that give the results of the CUDA-core path."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

from test_gpu_parity import drude, rel

pytestmark = pytest.mark.gpu


def solver(prec, graph, diameter=20.0):
    v, f = shapes.trisphere(256, diameter)
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.particle(v, f)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision=prec))
    bem.set_option("sweep_graph", graph)
    return bem, m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])


@pytest.mark.parametrize("prec,tol", [("mixed", 1e-7), ("fp64", 1e-11)])
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("more", [False, True])
def test_reported_once_by_a_warm_call(gpu_lib, prec, tol, graph, more):
    bem, exc = solver(prec, graph)
    enei = np.linspace(500.0, 650.0, 5)
    ref = [bem.spectrum(exc, enei) for _ in range(2)][1]["ext"]
    bem.set_option("selftest_tc_error", 32)
    with pytest.raises(Exception, match="wait expired"):
        bem.spectrum(exc, np.linspace(500.0, 650.0, 25) if more else enei)
    for _ in range(2):
        assert rel(bem.spectrum(exc, enei)["ext"], ref) < tol


def test_reported_by_a_batch(gpu_lib):
    sets = [solver("mixed", 1, d) for d in (20.0, 30.0)]
    enei = np.linspace(500.0, 650.0, 4)
    items = [(b, e, enei) for b, e in sets]
    ref = [m.spectrum_batch(items) for _ in range(2)][1]
    sets[1][0].set_option("selftest_tc_error", 4)
    with pytest.raises(Exception, match="wait expired"):
        m.spectrum_batch(items)
    again = m.spectrum_batch(items)
    for a, b in zip(again, ref):
        assert rel(a["ext"], b["ext"]) < 1e-7
