"""The last sum of the densities on both sides of eight partial sums, where that
of rho2 changes its kernel: rho2 of one state (tiles of 64 configurations at M <= 10, of
32 above twelve orbitals), of two states (32), and rho1 of both (256
configurations per block at M = 3), against the oracle's definition
(twobodyMatrix.h:991-1487, onebodyMatrix.h:190-251) at the repository's 1e-12."""
import pytest

import mcpi_b200 as mc
from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12


# blocks of rho2, t2: 8, 16; 9, 17; 4, 8; 5, 9; one of each; 5; 15 and 1 at M = 16 and 13
@pytest.mark.parametrize("N,M", [(32, 3), (33, 3), (23, 3), (24, 3), (2, 5), (4, 16), (5, 13), (2, 16)])
def test_rho2_partial_counts(orc, N, M):
    phi, psi = mc.random_problem(N, M, 51)[0], mc.random_problem(N, M, 52)[0]
    sp = mc.FockSpace(N, M)
    for got, a in ((sp.rho2(psi), psi), (sp.trans_rho2(phi, psi), phi)):
        assert rel(got.cpu().numpy().reshape(-1), orc.density(N, M, 2, a, psi)) <= TOL
    sp.close()


@pytest.mark.parametrize("N,M", [(63, 3), (64, 3), (1, 3), (5, 16), (4, 12)])
def test_rho1_partial_counts(orc, N, M):
    phi, psi = mc.random_problem(N, M, 53)[0], mc.random_problem(N, M, 54)[0]
    sp = mc.FockSpace(N, M)
    for got, a in ((sp.rho1(psi), psi), (sp.trans_rho1(phi, psi), phi)):
        assert rel(got.cpu().numpy(), orc.density(N, M, 1, a, psi).reshape(M, M).T) <= TOL
    sp.close()
