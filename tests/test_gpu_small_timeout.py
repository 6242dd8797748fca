"""The bounded grid barriers of the one-launch Lanczos (mcpi_lanczos of a small
space): with one block held back (MCPI_OPT_TEST_STALL_GATHER) the others give
up after the limit and the solve returns MCPI_ERR_TIMEOUT; the next solve of the
same space is right again. One tile of rows, a few, and more than there are blocks."""
import numpy as np
import pytest

import mcpi_b200 as mc

pytestmark = pytest.mark.gpu
ERR_TIMEOUT = 7


@pytest.mark.parametrize("N,M,lm", [(8, 2, 9), (5, 7, 30), (6, 10, 50)])
def test_barrier_timeout_and_recovery(N, M, lm):
    C0 = mc.random_problem(N, M, 31)[0]
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 3.0))
    it, a, b, _ = sp.lanczos(C0, lm)
    sp.set_option(mc.OPT_WAIT_LIMIT_KCYCLES, 500)          # about 0.3 ms per wait
    sp.set_option(mc.OPT_TEST_STALL_GATHER, 1)
    for call in (lambda: sp.lanczos(C0, lm), lambda: sp.ground(C0, lm)):
        with pytest.raises(mc.MCPIError) as e:
            call()
        assert e.value.status == ERR_TIMEOUT
    sp.set_option(mc.OPT_TEST_STALL_GATHER, 0)
    sp.set_option(mc.OPT_WAIT_LIMIT_KCYCLES, 0)
    it2, a2, b2, _ = sp.lanczos(C0, lm)
    assert it2 == it and np.array_equal(a2, a) and np.array_equal(b2, b)
    sp.close()
