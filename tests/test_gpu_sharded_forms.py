"""A sharded Lanczos on one rank is mcpi_lanczos bit for bit also where a solve
and a single H.psi take different forms: contact interactions of an odd number
of plane waves, where the recurrence amplifies rounding to order one and the
solve's form therefore decides the Ritz vector's sign -- with the direct form in
the solve (M = 11 from 180,000 rows) and the pair kernels (M = 13, 15) -- and
where both take the contact form (M = 10, 12). Row blocks of several ranks
follow the same rule, so there a row of H.psi does not depend on their number.
The plain row range keeps the form of the whole call."""
import socket

import numpy as np
import pytest
import torch
import torch.distributed as dist

import mcpi_b200 as mc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def one_rank():
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1)
    yield
    dist.destroy_process_group()


@pytest.mark.parametrize("N,M,lm", [(10, 11, 24), (5, 13, 40), (4, 15, 40), (5, 12, 40), (12, 10, 24)])
def test_one_rank_is_the_single_solve(one_rank, N, M, lm):
    from mcpi_b200.distributed import ShardedLanczos
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 5.0))
    C0 = torch.from_numpy(mc.random_problem(N, M, 104)[0]).cuda()
    sl = ShardedLanczos(sp.nc, lambda v: sp.apply_h_rows(v, sl.r0, sl.r1), torch.device("cuda"))
    it, alpha, beta, V = sl.lanczos(C0.clone(), lm)
    it1, alpha1, beta1, V1 = sp.lanczos(C0, lm)
    assert it == it1 == lm
    assert np.array_equal(alpha, alpha1) and np.array_equal(beta[:lm - 1], beta1[:lm - 1])
    assert torch.equal(V, V1)
    # outside the solve the row range is the whole call's again
    assert torch.equal(sp.apply_h_rows(C0, 0, sp.nc), sp.apply_h(C0))
    sp.close()


@pytest.mark.parametrize("N,M", [(10, 11), (5, 13), (4, 15)])
def test_rows_of_a_solve_do_not_depend_on_the_ranks(N, M):
    from mcpi_b200.distributed import row_block, solve_rows
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 5.0))
    x = torch.from_numpy(mc.random_problem(N, M, 105)[0]).cuda()
    with solve_rows():
        whole = sp.apply_h_rows(x, 0, sp.nc)
        for W in (2, 3):
            parts = [sp.apply_h_rows(x, *row_block(sp.nc, W, r)) for r in range(W)]
            assert torch.equal(torch.cat(parts), whole)
    sp.close()
