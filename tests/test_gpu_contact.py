"""The contact form of H.psi (momentum blocks that are outer products, as a
contact interaction gives): one pair sum per total momentum instead of one per
creation pair. It is the default where it is the fastest form (every M >= 12;
larger spaces below), so small spaces of many orbitals are checked against the
oracle's restatement of the reference (hamiltonianMatrix.h:891-1425,
applyHconf_XX) and larger ones against the direct form
(MCPI_OPT_DIRECT_HPSI = 1), which sums the same terms in another order. A sum
of at most 136 pairs of terms, each a product of a few rounded factors, is
within 1e-13 of the other order's; the bound is the repository's 1e-12."""
import numpy as np
import pytest
import torch

import mcpi_b200 as mc
from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _state(nc, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn(nc, dtype=torch.complex128, device="cuda", generator=gen)
    return x / torch.linalg.vector_norm(x)


def _two_launches(sp, x):
    return sp.apply_h_profile(x, reps=1)[1] > 0.0


def scaled_contact(M, g, seed):
    """Contact integrals with a real factor per orbital, Hint[k,s,q,l] times
    f_k f_s f_q f_l: outer products whose factors all differ."""
    f = np.random.default_rng(seed).uniform(0.5, 2.0, M)
    Ho, Hint = mc.lieb_integrals(M, g)
    t = Hint.reshape(M, M, M, M) * np.einsum("l,q,s,k->lqsk", f, f, f, f)
    return Ho, t.reshape(-1)


@pytest.mark.parametrize("N,M,kind", [(2, 12, "lieb"), (5, 12, "lieb"), (4, 13, "lieb"), (3, 16, "lieb"),
                                      (70, 2, "lieb"), (66, 3, "lieb"), (5, 14, "zero"), (4, 15, "scaled")])
def test_contact_against_oracle(orc, N, M, kind):
    Ho, Hint = scaled_contact(M, 1.5, N) if kind == "scaled" else mc.lieb_integrals(M, 0.0 if kind == "zero" else 2.5)
    C = mc.random_problem(N, M, 5)[0]
    sp = mc.FockSpace(N, M)
    sp.set_integrals(Ho, Hint)
    ref = orc.apply_h(N, M, C, Ho, Hint, mode=2)
    full = sp.apply_h(C)
    assert rel(full.cpu().numpy(), ref) <= TOL
    assert rel(sp.apply_h_adjoint(C).cpu().numpy(), ref) <= TOL     # Hermitian integrals
    nc = sp.nc
    for r0, r1 in [(0, nc), (0, 1), (nc - 1, nc), (nc // 3, nc // 3 + min(257, nc // 3)), (nc // 2, nc)]:
        assert torch.equal(sp.apply_h_rows(C, r0, r1), full[r0:r1]), (r0, r1)
    sp.close()


@pytest.mark.parametrize("N,M", [(12, 10), (14, 10), (10, 11), (13, 11), (9, 13), (20, 8), (16, 9)])
def test_contact_against_direct(N, M):
    Ho, Hint = mc.lieb_integrals(M, 1.0)
    sp = mc.FockSpace(N, M)
    sp.set_integrals(Ho, Hint)
    x = _state(sp.nc, N * 100 + M)
    got = sp.apply_h(x)
    part = sp.apply_h_rows(x, sp.nc // 3, sp.nc // 2)
    sp.set_option(mc.OPT_DIRECT_HPSI, 1)
    ref = sp.apply_h(x)
    norm = torch.linalg.vector_norm(ref)
    assert float(torch.linalg.vector_norm(got - ref) / norm) <= TOL
    assert float(torch.linalg.vector_norm(part - ref[sp.nc // 3:sp.nc // 2]) / norm) <= TOL
    sp.close()


def test_near_contact_blocks_keep_the_direct_form():
    # one block value off by 1e-12: no outer product within rounding, so the
    # value has to be applied as it is
    N, M = 14, 10
    Ho, Hint = mc.lieb_integrals(M, 1.0)
    sp = mc.FockSpace(N, M)
    sp.set_integrals(Ho, Hint)
    x = _state(sp.nc, 3)
    assert _two_launches(sp, x)
    t = Hint.reshape(M, M, M, M).copy()
    t[4, 4, 4, 4] *= 1.0 + 1e-12
    sp.set_integrals(Ho, t.reshape(-1))
    assert not _two_launches(sp, x)
    sp.close()


def test_contact_calls_on_two_streams_do_not_mix():
    # the calls share one intermediate: each must see its own, whatever the
    # streams do
    N, M = 14, 10
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 1.0))
    xs = [_state(sp.nc, 40 + k) for k in range(2)]
    refs = [sp.apply_h(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[] for _ in range(2)]
    for _ in range(20):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                outs[k].append(sp.apply_h(xs[k]))
    torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(o, refs[k]) for o in outs[k])
    sp.close()


def test_capture_uses_the_direct_form():
    # a captured call may run beside calls outside its graph: it takes the form
    # that has no scratch, and matches the contact form to rounding
    N, M = 14, 10
    sp = mc.FockSpace(N, M)
    sp.set_integrals(*mc.lieb_integrals(M, 1.0))
    x = _state(sp.nc, 9)
    ref, out = sp.apply_h(x), torch.empty_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sp.apply_h(x, out)
    g.replay()
    torch.cuda.synchronize()
    assert float(torch.linalg.vector_norm(out - ref) / torch.linalg.vector_norm(ref)) <= TOL
    del g
    sp.close()


def test_batched_contact_groups_follow_their_integrals():
    # groups of M = 10, 11, 12 take the contact form; one member with another
    # interaction moves its group to the direct or two-kernel form at the next
    # run, and back. E0 against single solves at the repository's 1e-10.
    lm = 40
    members = [(6, 10), (4, 10), (5, 11), (7, 11), (3, 12), (5, 12), (6, 7)]
    i = np.arange(16)

    def finite_range(M, g):
        Ho, _ = mc.lieb_integrals(M, g)
        l, q, s, k = np.meshgrid(i[:M], i[:M], i[:M], i[:M], indexing="ij")
        v = lambda p: np.exp(-0.06 * p.astype(float) ** 2)
        return Ho, np.where(k + s == q + l, 0.5 * g * (v(k - l) + v(k - q)), 0.0).reshape(-1).astype(np.complex128)

    contact = [mc.lieb_integrals(M, 0.5 + 0.7 * x) for x, (N, M) in enumerate(members)]
    other = [finite_range(M, 1.5) for N, M in members]
    starts = [mc.random_problem(N, M, 60 + x)[0] for x, (N, M) in enumerate(members)]

    def singles(ints):
        out = []
        for (N, M), (Ho, Hint), C in zip(members, ints, starts):
            sp = mc.FockSpace(N, M)
            sp.set_option(mc.OPT_DIRECT_HPSI, 1)
            sp.set_integrals(Ho, Hint)
            out.append(sp.ground(C, lm)[0])
            sp.close()
        return np.array(out)

    b = mc.Batch(members, lm)
    for x in range(len(members)):
        b.set_integrals(x, *contact[x])
        b.set_start(x, starts[x])
    mixed = list(contact)
    for changed in ([], [1, 3, 5], [1, 3, 5]):
        for x in changed:
            mixed[x] = other[x] if mixed[x] is contact[x] else contact[x]
            b.set_integrals(x, *mixed[x])
        E, it = b.run()
        ref = singles(mixed)
        assert (it == lm).all()
        assert np.abs(E - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
    b.close()
