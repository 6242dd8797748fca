"""H.psi where one orbital holds more than 256 bosons: the occupations that the
pair-creation kernels keep per row must not wrap there. Spaces of two to four
orbitals around 256 particles, in every form of kernel 2 (contact, shared
tables, registers, fused), against the oracle's restatement of the reference
(hamiltonianMatrix.h:891-1425, applyHconf_XX) at the repository's 1e-12."""
import numpy as np
import pytest

import mcpi_b200 as mc
from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12


def finite_range(M, g):
    """A finite-range interaction on a ring in plane waves: momentum blocks that are no outer products."""
    Ho, _ = mc.lieb_integrals(M, g)
    i = np.arange(M)
    l, q, s, k = np.meshgrid(i, i, i, i, indexing="ij")
    v = lambda p: np.exp(-0.06 * p.astype(float) ** 2)
    return Ho, np.where(k + s == q + l, 0.5 * g * (v(k - l) + v(k - q)), 0.0).reshape(-1).astype(np.complex128)


CASES = [(N, M, kind) for N, M in [(300, 1), (256, 2), (257, 2), (258, 2), (300, 2), (600, 2), (260, 3)]
         for kind in ("lieb", "range", "random")] + [(258, 4, "lieb")]


@pytest.mark.parametrize("N,M,kind", CASES)
def test_more_than_256_bosons_in_an_orbital(orc, N, M, kind):
    C, Ho, Hint = mc.random_problem(N, M, 7)
    if kind == "lieb":
        Ho, Hint = mc.lieb_integrals(M, 2.5)
    elif kind == "range":
        Ho, Hint = finite_range(M, 1.5)
    ref = orc.apply_h(N, M, C, Ho, Hint, mode=2)
    for opts in ({}, {mc.OPT_CREATE_FORM: 1}, {mc.OPT_FUSED_HPSI: 1}):
        sp = mc.FockSpace(N, M)
        for o, v in opts.items():
            sp.set_option(o, v)
        sp.set_integrals(Ho, Hint)
        assert rel(sp.apply_h(C).cpu().numpy(), ref) <= TOL, opts
        sp.close()
