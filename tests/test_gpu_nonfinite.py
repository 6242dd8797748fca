"""Infinite amplitudes in rho1 and the transition rho1. An entry is a sum of
products with positive weights, so with positive amplitudes one infinite
amplitude makes exactly the entries that use it infinite, and leaves the rest
at their finite values (onebodyMatrix.h:190-251). No lane of a partly filled
tile may turn them into NaN: hole spaces of 35, 78, 126 and 1,287
configurations against the kernel's tiles of 32, with the infinite amplitude
reached from the first and from the last hole configuration."""
import numpy as np
import pytest

import mcpi_b200 as mc
from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(4, 5), (3, 12), (6, 5), (9, 6)])
@pytest.mark.parametrize("tables", [False, True])
def test_rho1_with_one_infinite_amplitude(orc, N, M, tables):
    rng = np.random.default_rng(N * 100 + M)
    nc, nc1 = mc.nc_of(N, M), mc.nc_of(N - 1, M)
    assert nc1 % 32
    phi = rng.uniform(0.5, 1.5, nc).astype(np.complex128)
    sp = mc.FockSpace(N, M)
    if tables:
        sp.set_integrals(*mc.lieb_integrals(M, 1.0))
    for h in (0, nc1 - 1):
        for orb in (0, M - 1):
            v = mc.IndexToFock(h, N - 1, M)
            v[orb] += 1
            psi = rng.uniform(0.5, 1.5, nc).astype(np.complex128)
            finite = psi.copy()
            finite[mc.FockToIndex(N, M, v)] = 0.0
            psi[mc.FockToIndex(N, M, v)] = np.inf
            held = v > 0
            for got, ref, inf in (
                    (sp.rho1(psi), orc.density(N, M, 1, finite, finite), held[:, None] | held[None, :]),
                    (sp.trans_rho1(phi, psi), orc.density(N, M, 1, phi, finite), np.tile(held, (M, 1)))):
                re = got.cpu().numpy().real
                assert np.array_equal(np.isposinf(re), inf), (h, orb)
                ref = ref.reshape(M, M).T.real
                assert rel(re[~inf], ref[~inf]) <= 1e-12
    sp.close()
