"""rho1 and the transition rho1 at every orbital count and at hole-space sizes
around the kernel's tiles of 32 configurations (one, a few lanes of one tile,
one tile more than the blocks take at once), against the oracle's definition
(orc.density, flat t1[k + l*M]; onebodyMatrix.h:190-251) at the repository's 1e-12."""
import numpy as np
import pytest
import torch

import mcpi_b200 as mc
from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("M", range(1, 17))
@pytest.mark.parametrize("N", [1, 2, 4])
def test_rho1_every_orbital_count(orc, N, M):
    phi, psi = mc.random_problem(N, M, 11)[0], mc.random_problem(N, M, 12)[0]
    sp = mc.FockSpace(N, M)
    for tables in (False, True):          # decoded and packed occupations
        if tables:
            sp.set_integrals(*mc.lieb_integrals(M, 1.0))
        r = sp.rho1(psi).cpu().numpy()
        assert rel(r, orc.density(N, M, 1, psi, psi).reshape(M, M).T) <= TOL
        assert np.array_equal(np.triu(r, 1), np.conj(np.tril(r, -1)).T)
        assert rel(sp.trans_rho1(phi, psi).cpu().numpy(), orc.density(N, M, 1, phi, psi).reshape(M, M).T) <= TOL
    sp.close()


@pytest.mark.parametrize("N,M", [(33, 2), (64, 2), (7, 5), (12, 4), (9, 6), (8, 8), (10, 7)])
def test_rho1_tile_edges(orc, N, M):
    phi, psi = mc.random_problem(N, M, 21)[0], mc.random_problem(N, M, 22)[0]
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 1.0))
    assert rel(sp.rho1(psi).cpu().numpy(), orc.density(N, M, 1, psi, psi).reshape(M, M).T) <= TOL
    t = sp.trans_rho1(phi, psi)
    assert rel(t.cpu().numpy(), orc.density(N, M, 1, phi, psi).reshape(M, M).T) <= TOL
    assert torch.equal(t, sp.trans_rho1(phi, psi))        # fixed summation order
    sp.close()
