"""The one-launch Lanczos of small spaces (mcpi_lanczos / mcpi_ground with real
momentum-block integrals, up to eleven orbitals) takes every sum in the order
of the launch sequence (MCPI_OPT_DIRECT_HPSI = 1 keeps that), so alpha, beta,
the basis and the Ritz vector are the same bit for bit: at odd row counts, row
counts around the 32-, 256- and 1,024-row units of the sums, fewer and more
basis vectors than a staged chunk of 64, and after a breakdown. E0 is checked
against the oracle (groundStateLieb.c:348-471) at the repository's 1e-10."""
import numpy as np
import pytest
import torch

import mcpi_b200 as mc

pytestmark = pytest.mark.gpu


def gauss_integrals(M, g):
    """A finite-range interaction on a ring in plane waves: real momentum blocks."""
    Ho, _ = mc.lieb_integrals(M, g)
    i = np.arange(M)
    l, q, s, k = np.meshgrid(i, i, i, i, indexing="ij")
    v = lambda p: np.exp(-0.06 * p.astype(float) ** 2)
    return Ho, np.where(k + s == q + l, 0.5 * g * (v(k - l) + v(k - q)), 0.0).reshape(-1).astype(np.complex128)


# (rows: 21, 41, 255, 256, 3003, 1287, 220, 1001, 1330, 8008, 11440)
@pytest.mark.parametrize("N,M,lm,kind", [(5, 3, 8, "lieb"), (40, 2, 12, "lieb"), (21, 3, 40, "lieb"),
                                         (3, 9, 33, "gauss"), (5, 11, 375, "lieb"), (8, 6, 64, "gauss"),
                                         (9, 4, 66, "lieb"), (10, 5, 65, "gauss"), (18, 4, 150, "lieb"),
                                         (6, 11, 100, "gauss"), (7, 10, 150, "lieb"), (2, 2, 8, "lieb")])
def test_small_lanczos_is_the_launch_sequence_bit_for_bit(N, M, lm, kind):
    Ho, Hint = gauss_integrals(M, 1.5) if kind == "gauss" else mc.lieb_integrals(M, 4.0)
    C0 = mc.random_problem(N, M, 23)[0]
    runs = []
    for direct in (1, 2, 2):
        sp = mc.FockSpace(N, M)
        sp.set_option(mc.OPT_DIRECT_HPSI, direct)
        sp.set_integrals(Ho, Hint)
        it, a, b, V = sp.lanczos(C0, lm)
        E, psi, itg = sp.ground(C0, lm)
        n = max(it, 1)
        runs.append((it, a[:n], b[:max(n - 1, 0)], V[:n].cpu().numpy(), E, psi.cpu().numpy(), itg))
        sp.close()
    for x in runs[1:]:
        assert x[0] == runs[0][0] and x[6] == runs[0][6] and x[4] == runs[0][4]
        for k in (1, 2, 3, 5):
            assert np.array_equal(x[k], runs[0][k]), (N, M, k)


def test_small_lanczos_against_oracle(orc):
    N, M, lm = 5, 7, 57
    Ho, Hint = mc.lieb_integrals(M, 10.0)
    C0 = orc.perf_inputs(N, M)[0]
    Eo, po, ito = orc.ground(N, M, Ho, Hint, C0, lm, mode=2)
    sp = mc.FockSpace(N, M)
    sp.set_integrals(Ho, Hint)
    for _ in range(2):                                     # the second solve reuses the workspaces
        E, psi, it = sp.ground(C0, lm)
        assert it == ito and abs(E - Eo) <= 1e-10 * max(1.0, abs(Eo))
    sp.close()


def test_small_lanczos_first_step_breakdown():
    # a Fock state is an eigenvector of the non-interacting gas
    N, M = 6, 7
    Ho, Hint = mc.lieb_integrals(M, 0.0)
    sp = mc.FockSpace(N, M)
    sp.set_integrals(Ho, Hint)
    C0 = np.zeros(sp.nc, np.complex128)
    C0[17] = 1.0
    it, a, _, _ = sp.lanczos(C0, 20)
    assert it == 0 and abs(a[0] - np.dot(mc.IndexToFock(17, N, M), Ho.diagonal())) <= 1e-10 * abs(a[0])
    sp.close()
