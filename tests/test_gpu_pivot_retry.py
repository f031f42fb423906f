"""Mixed-precision solves of small particles whose 256-wide diagonal blocks, which
interchange no rows, leave a factorisation that does not contract (a rounded cube of a
nearly lossless metal with eps close to minus the water's): the call is run again with
64-wide pivoted blocks.  Every entry point that factors the matrices, one-graph and
host-scheduled sweeps, and a handle's results do not depend on the calls before.

Tolerance: a refinement that stops at its tolerance (1e-10 of the solution) leaves a
relative residual below it; one that stalls after ten steps was at 2e-10 to 9e-10.
The wavelengths are those at which the pivoted blocks converge within the ten steps."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

pytestmark = pytest.mark.gpu
TOL = 1e-10


def solver(eps=-2.0 + 1e-4j, graph=1):
    v, f = shapes.tricube(10, 20.0, shapes.rounding_to_e(20.0, 2.0))
    cp = m.comparticle([m.epsconst(1.77), m.epsconst(eps)], [m.particle(v, f)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="mixed"))
    bem.set_option("sweep_graph", graph)
    return cp, bem, m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])


@pytest.mark.parametrize("graph", [0, 1])
def test_sweep(gpu_lib, graph):
    cp, bem, exc = solver(graph=graph)
    first = bem.spectrum(exc, [550.0, 600.0])
    assert np.all(first["ir_resid"] < TOL)
    again = bem.spectrum(exc, [550.0, 600.0])
    assert np.all(again["ir_resid"] < TOL)
    other, _, _ = solver(-9.0 + 1.0j)
    good = m.bemsolver(other, m.bemoptions(precision="mixed"))
    ref = good.spectrum(exc, [550.0, 600.0])
    assert np.all(ref["ir_resid"] < TOL)
    assert np.array_equal(good.spectrum(exc, [550.0, 600.0])["ext"], ref["ext"])


def test_single_solve_and_potentials(gpu_lib):
    cp, bem, exc = solver()
    for _ in range(2):
        assert bem.mldivide(exc(cp, 600.0)).ir_resid < TOL
    dip = m.dipoleret(cp, [[0, 0, 18.0]])(cp, 600.0)
    a = bem.mldivide(dip)
    ref = m.bemsolver(cp, m.bemoptions(precision="fp64")).mldivide(dip)
    # the residual bound times the condition that the plane-wave solves show (1e5)
    assert np.max(np.abs(a.sig2 - ref.sig2)) < 1e5 * TOL * np.max(np.abs(ref.sig2))


def test_batch(gpu_lib):
    sets = [solver(), solver(-9.0 + 1.0j)]
    r = m.spectrum_batch([(b, e, [550.0, 600.0]) for _, b, e in sets])
    for q in r:
        assert np.all(q["ir_resid"] < TOL)


def test_better_of_both_is_kept(gpu_lib):
    """Two spheres of sizes 1 : 300, whose areas differ by 10^5 inside a block: neither
    converges in ten steps, the wide blocks end at a residual of 1e-8 and the pivoted
    ones above 1."""
    v, f = shapes.trisphere(144, 20.0)
    vb, fb = shapes.trisphere(144, 6000.0)
    drude = m.epsfun(lambda w: 10 - 9.065 ** 2 / (w * (w + 0.0708j)), "eV")
    cp = m.comparticle([m.epsconst(1.77), drude], [m.particle(v, f), m.particle(vb + [3012.0, 0, 0], fb)],
                       [[2, 1], [2, 1]], 1, 2)
    bem = m.bemsolver(cp, m.bemoptions(precision="mixed"))
    r = bem.spectrum(m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]]), [550.0, 600.0])
    assert np.all(r["ir_resid"] < 1e-4)


def test_gradient_and_iterative_solver(gpu_lib):
    """The other callers of the factorisation: the gradient's forward solve is run again
    as a sweep's is, and the iterative solver takes its dense preconditioner from either.
    Tolerance: the plane-wave solves' condition (1e5) times the refinement's 1e-10, and
    the iterative solver's own residual."""
    cp, bem, exc = solver()
    val, gv, _ = bem.cross_section_gradient(exc, 600.0, 0, "ext", "mixed")
    ref, rv, _ = bem.cross_section_gradient(exc, 600.0, 0, "ext", "fp64")
    assert abs(val - ref) < 1e5 * TOL * abs(ref)
    assert np.max(np.abs(gv - rv)) < 1e5 * TOL * np.max(np.abs(rv))
    it = m.bemsolver(cp, m.bemoptions(precision="mixed", iter={"tol": 1e-9}))
    for _ in range(2):
        it.mldivide(exc(cp, 600.0))
        assert it.info["flag"] == 0
