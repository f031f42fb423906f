"""External potentials of more than four columns (groups that share one
factorisation, mnpbem_solve_potentials_groups): every column has the bits it has
when its group is solved alone, and group sizes outside 1..4 are refused."""
import ctypes

import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import _lib

from test_gpu_parity import drude

pytestmark = pytest.mark.gpu
KEYS = ("phi1", "phi1p", "phi2", "phi2p", "a1", "a1p", "a2", "a2p")


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("ncol", [1, 5, 9])
def test_groups_equal_single_solves(gpu_lib, prec, ncol):
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.trisphere(144, 20.0)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision=prec))
    exc = m.dipoleret(cp, [[0, 0, 15.0], [0, 30.0, 0], [22.0, 3.0, 1.0]])(cp, 540.0)
    cut = lambda c0, c1: m.compstruct(cp, 540.0, **{k: np.asarray(getattr(exc, k))[..., c0:c1] for k in KEYS})
    sig = bem.mldivide(cut(0, ncol))
    for c0 in range(0, ncol, 4):
        one = bem.mldivide(cut(c0, min(ncol, c0 + 4)))
        for k in ("sig1", "sig2", "h1", "h2"):
            assert np.array_equal(getattr(sig, k)[..., c0:c0 + 4], getattr(one, k)), (k, c0)


@pytest.mark.parametrize("npol", [0, 5])
def test_group_size_refused(gpu_lib, npol):
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.trisphere(32, 10.0)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions())
    pots, sols = (_lib.Potentials * 2)(), (_lib.Solution * 2)()
    pots[0].npol, pots[1].npol = 1, npol
    em = np.ascontiguousarray(cp.eps_media(540.0)[0])
    st = gpu_lib.mnpbem_solve_potentials_groups(bem._h, pots, 2, 540.0,
                                                em.view(np.float64).ctypes.data_as(_lib.c_double_p), em.size,
                                                _lib.MIXED, None, sols)
    with pytest.raises(Exception):
        _lib.check(st)
