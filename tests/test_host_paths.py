"""Host code of the library without a GPU (tests/fake_cuda.py): a launch that
fails fails the call it belongs to."""
import ctypes as ct

import numpy as np
import pytest

import fake_cuda
import mcpi_b200 as mc
from fake_cuda import ERR_CUDA, ERR_NOMEM, OK


@pytest.fixture(scope="session")
def fake_so(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def fake(fake_so):
    f = fake_cuda.Fake(fake_so)
    f.reset()
    yield f
    f.reset()


def every_launch_counts(fake, make, call, most=24):
    """Fails each launch of a call in turn, on a fresh space (whose first call
    also builds what the space keeps) and on a used one: the call has to report
    it, and the next call has to run clean and whole."""
    s = make()
    first = fake.kernels(lambda: call(s))
    warm = fake.kernels(lambda: call(s))
    assert warm
    for k in range(min(len(warm), most)):
        fake.L.fake_fail_launch(k)
        assert call(s) == ERR_CUDA, k
        assert fake.kernels(lambda: call(s)) == warm, k
    s.close()
    for k in range(min(len(first), most)):
        s = make()
        fake.L.fake_fail_launch(k)
        assert call(s) == ERR_CUDA, k
        assert set(warm) <= set(fake.kernels(lambda: call(s))) <= set(first) | set(warm), k
        assert fake.kernels(lambda: call(s)) == warm, k
        s.close()


CALLS = {
    "apply_h": lambda s: s.apply_h(), "adjoint": lambda s: s.apply_h_adjoint(),
    "rho1": lambda s: s.density(1), "rho2": lambda s: s.density(2), "t1": lambda s: s.density(1, False),
    "t2": lambda s: s.density(2, False), "rows": lambda s: s.rows(1, s.nc - 1), "dot": lambda s: s.dot(),
    "lanczos": lambda s: s.lanczos(9), "ground": lambda s: s.ground(9), "lowmem": lambda s: s.ground(5, True)}


# (options, shared memory a block may take): every form of H.psi, and the
# densities' forms by the orbital count
@pytest.mark.parametrize("N,M,kind,opts,optin", [
    (5, 6, "lieb", {}, 0), (5, 6, "lieb", {mc.OPT_DIRECT_HPSI: 0}, 0), (5, 6, "lieb", {mc.OPT_CREATE_FORM: 1}, 0),
    (5, 6, "lieb", {mc.OPT_DIRECT_HPSI: 0, mc.OPT_FUSED_HPSI: 1}, 0),
    (5, 6, "lieb", {mc.OPT_NO_MOMENTUM_KERNEL: 1}, 0), (5, 6, "random", {}, 0),
    (5, 6, "random", {mc.OPT_NO_GEMM_KERNEL: 1}, 0), (4, 10, "random", {}, 120000),
    (3, 13, "lieb", {}, 0), (3, 16, "random", {}, 0), (70, 2, "lieb", {}, 0)])
@pytest.mark.parametrize("call", CALLS)
def test_a_failed_launch_fails_its_call(fake, N, M, kind, opts, optin, call):
    if optin:
        fake.L.fake_optin(optin)
    if call == "rows" and opts.get(mc.OPT_CREATE_FORM):
        return                                            # row ranges need the default pair-creation form
    _, Ho, Hint = mc.random_problem(N, M, 3)

    def make():
        s = fake.space(N, M)
        for o, v in opts.items():
            s.option(o, v)
        assert s.set_integrals(*((Ho, Hint) if kind == "random" else mc.lieb_integrals(M, 1.0))) == OK
        return s

    every_launch_counts(fake, make, CALLS[call])


def test_a_failed_launch_fails_the_batch(fake):
    b = fake.batch([(4, 7), (5, 7), (3, 10), (4, 10), (3, 12)], 5, mc.lieb_integrals)
    n = len(fake.kernels(b.run))
    b.close()
    for k in range(0, n, 3):
        b = fake.batch([(4, 7), (5, 7), (3, 10), (4, 10), (3, 12)], 5, mc.lieb_integrals)
        fake.L.fake_fail_launch(k)
        assert b.run() == ERR_CUDA, k
        b.close()


def test_a_failed_table_launch_leaves_no_table(fake):
    # mcpi_set_integrals packs the occupations of two spaces, the first rho1 of a third
    for k in range(2):
        s = fake.space(5, 6)
        fake.L.fake_fail_launch(k)
        assert s.set_integrals(*mc.lieb_integrals(6, 1.0)) == ERR_CUDA
        again = fake.kernels(lambda: s.set_integrals(*mc.lieb_integrals(6, 1.0)))
        assert len([n for n in again if "k_pack_occ" in n]) == 2
        fake.L.fake_fail_launch(0)
        assert s.density(1) == ERR_CUDA
        assert len([n for n in fake.kernels(lambda: s.density(1)) if "k_pack_occ" in n]) == 1
        s.close()


def forms(kernels):
    """The forms of H.psi among the launched kernels."""
    known = {"k_contact_sum": "contact", "k_hpsi_direct": "direct", "k_pair_create": "pairs", "k_hpsi_fused": "fused"}
    return {f for k, f in known.items() for n in kernels if k in n}


@pytest.mark.parametrize("lowmem", [False, True])
def test_a_solve_keeps_one_form_when_memory_runs_out(fake, lowmem):
    # N=12, M=10: contact form with an S from the pool. Whichever of its requests
    # the pool turns down, once or for good, all H.psi of a solve take one form.
    s = fake.space(12, 10)
    assert s.set_integrals(*mc.lieb_integrals(10, 1.0)) == OK
    solve = (lambda: s.ground(6, True)) if lowmem else (lambda: s.lanczos(6))
    assert forms(fake.kernels(solve)) == {"contact"}
    for for_good in (0, 1):
        for k in range(12):
            fake.L.fake_fail_pool(k, for_good)
            got = forms(fake.kernels(solve))
            assert got == {"direct" if k == 0 else "contact"}, (for_good, k)
            fake.L.fake_fail_pool(-1, 0)
    s.close()


# (N, M, form of a single H.psi, form of a solve, form of a part of a solve's rows)
@pytest.mark.parametrize("N,M,single,solve,part", [
    (10, 11, "contact", "direct", "direct"), (5, 13, "contact", "pairs", "pairs"), (4, 15, "contact", "pairs", "pairs"),
    (5, 12, "contact", "contact", "contact"), (12, 10, "contact", "contact", "direct"), (6, 9, "direct", "direct", "direct")])
def test_rows_of_a_solve_take_its_form(fake, N, M, single, solve, part):
    s = fake.space(N, M)
    assert s.set_integrals(*mc.lieb_integrals(M, 1.0)) == OK
    s.option(mc.OPT_FUSED_HPSI, 0)
    rows = lambda e, r0, r1: forms(fake.kernels(lambda: s.rows(r0, r1, e)))
    assert forms(fake.kernels(s.apply_h)) == {single} == rows("mcpi_apply_h_rows", 0, s.nc)
    if s.nc > 13000:                       # smaller ones may take the one-launch Lanczos
        assert forms(fake.kernels(lambda: s.lanczos(3))) == {solve}
    assert forms(fake.kernels(lambda: s.ground(3, True))) == {solve}
    assert rows("mcpi_shard_apply_h", 0, s.nc) == {solve}
    assert rows("mcpi_shard_apply_h", 5, s.nc // 2) == {part}
    s.close()


def test_solve_rows_is_per_thread_and_nests():
    import threading
    from mcpi_b200 import _rows
    from mcpi_b200.distributed import solve_rows
    seen = []
    with solve_rows():
        with solve_rows():
            pass
        seen.append(_rows.solve)
        t = threading.Thread(target=lambda: seen.append(getattr(_rows, "solve", False)))
        t.start()
        t.join()
        try:
            with solve_rows():
                raise KeyError
        except KeyError:
            pass
        seen.append(_rows.solve)
    assert seen == [True, False, True] and not _rows.solve


class Held:
    """A space of 13 bosons in 10 orbitals with one H.psi queued: the pool holds
    its S, 51 MB, freed on the stream but not seen to be. On the device then no
    more than `room` bytes are left beside it."""

    def __init__(self, fake, room):
        self.s = fake.space(13, 10)
        assert self.s.set_integrals(*mc.lieb_integrals(10, 1.0)) == OK
        self.fake, self.room = fake, room

    def __enter__(self):
        assert forms(self.fake.kernels(self.s.apply_h)) == {"contact"}
        assert self.fake.L.fake_pool_held() > 50e6
        self.fake.L.fake_headroom(self.room)
        return self

    def __exit__(self, *exc):
        self.fake.reset()
        self.s.close()


def alloc(s, n):
    p = ct.c_void_p()
    rc = s.L.mcpi_alloc(s.h, ct.c_size_t(n), ct.byref(p))
    if rc == OK:
        s.L.mcpi_free(s.h, p)
    return rc


def packs(kernels):
    return len([n for n in kernels if "k_pack_occ" in n])


def test_pool_memory_goes_to_an_allocation(fake):
    with Held(fake, 1 << 20) as h:
        assert alloc(h.s, 40 << 20) == OK and fake.L.fake_pool_held() == 0
        assert alloc(h.s, 80 << 20) == ERR_NOMEM              # more than there is stays refused
        assert forms(fake.kernels(h.s.apply_h)) == {"contact"}


def test_pool_memory_goes_to_the_tables(fake):
    t = fake.space(11, 11)                                     # occupations 2.8 and 0.7 MB, rho1's 1.5 MB
    with Held(fake, 1 << 20):
        assert packs(fake.kernels(lambda: t.set_integrals(*mc.lieb_integrals(11, 1.0)))) == 2
    assert t.density(2) == OK                                  # the partial sums, not counted here
    with Held(fake, 1 << 20):
        assert packs(fake.kernels(lambda: t.density(1))) == 1
    n = ct.c_int64()
    with Held(fake, 1 << 20):
        assert t.L.mcpi_two_map_size(t.h, 1, ct.byref(n)) == OK
    t.close()


def test_pool_memory_goes_to_an_operator_and_a_space(fake):
    _, Ho, Hint = mc.random_problem(4, 12, 3)
    t = fake.space(4, 12)                                      # dense pair matrices, 97 kB each
    with Held(fake, 40 << 10):
        assert t.set_integrals(Ho, Hint) == OK
    t.close()
    with Held(fake, 64):
        u = fake.space(4, 4)
        u.close()


def test_pool_memory_goes_to_a_batch(fake):
    # arena 36 MB with the contact form's intermediates, 21 MB without
    members = [(10, 10), (10, 10)]
    with Held(fake, 30 << 20):
        b = fake.batch(members, 5, mc.lieb_integrals)
        assert b.rc == OK and any("k_batch_contact" in n for n in fake.kernels(b.run))
        b.close()


def test_a_batch_leaves_room_for_its_tables(fake):
    # With room for the larger arena but not for what the batch still needs
    # after it, the batch takes the smaller arena and runs the direct form.
    members, later = [(10, 10), (10, 10)], 2 * ((1 << 20) + 8 * (92378 + 24310))
    b = fake.batch(members, 5, mc.lieb_integrals)
    n = ct.c_size_t()
    b.L.mcpi_batch_arena_bytes(b.h, ct.byref(n))
    b.close()
    for room, contact in ((n.value + later + (1 << 20), True), (n.value + (1 << 16), False)):
        fake.L.fake_headroom(room)
        b = fake.batch(members, 5, mc.lieb_integrals)
        assert b.rc == OK
        assert any("k_batch_contact" in k for k in fake.kernels(b.run)) == contact
        b.close()
        fake.reset()


@pytest.mark.parametrize("N,M,lm,one", [(2, 2, 7, False), (2, 2, 8, True), (5, 11, 23, False), (5, 11, 24, True),
                                        (9, 7, 39, False), (9, 7, 40, True), (12, 6, 400, False), (6, 11, 400, False),
                                        (9, 7, 2048, True), (2, 2, 2049, False)])
def test_which_solves_take_one_launch(fake, N, M, lm, one):
    s = fake.space(N, M)                   # 3, 3,003, 5,005, 6,188 and 8,008 rows
    assert s.set_integrals(*mc.lieb_integrals(M, 1.0)) == OK
    assert any("k_small_lanczos" in k for k in fake.kernels(lambda: s.lanczos(lm))) == one
    s.close()


# 92,378 and 48,620 rows at M = 10, 92,378 and 43,758 at M = 11, 1,365 at M = 12
@pytest.mark.parametrize("members,contact", [
    ([(10, 10)], False), ([(10, 10), (9, 10)], True), ([(4, 10)] * 19, False), ([(4, 10)] * 20, True),
    ([(9, 11)], False), ([(9, 11), (5, 11), (5, 11)], True), ([(3, 11)] * 14, False), ([(3, 11)] * 15, True),
    ([(4, 12)], True), ([(10, 9)] * 3, False)])
def test_which_batches_take_the_contact_form(fake, members, contact):
    b = fake.batch(members, 4, mc.lieb_integrals)
    assert b.rc == OK
    assert any("k_batch_contact" in k for k in fake.kernels(b.run)) == contact
    b.close()


def scaled_contact(M, g, f):
    """Contact integrals with a real factor per orbital."""
    Ho, Hint = mc.lieb_integrals(M, g)
    return Ho, (Hint.reshape(M, M, M, M) * np.einsum("l,q,s,k->lqsk", f, f, f, f)).reshape(-1)


def test_the_contact_form_takes_exact_products_only(fake):
    M = 12
    for f, exact in ((np.ones(M), True), (2.0 ** np.arange(-6, 6), True), (-np.ones(M), True),
                     (np.random.default_rng(1).uniform(0.5, 2.0, M), False)):
        s = fake.space(4, M)
        assert s.set_integrals(*scaled_contact(M, 0.7, f)) == OK
        assert forms(fake.kernels(s.apply_h)) == {"contact" if exact else "pairs"}
        assert forms(fake.kernels(s.apply_h_adjoint)) == {"contact" if exact else "pairs"}
        s.close()


def test_tables_are_written_before_another_stream_can_read_them(fake):
    s = fake.space(6, 7)
    assert not fake.unfinished(lambda: s.set_integrals(*mc.lieb_integrals(7, 1.0)))
    fake.L.fake_capture(1)                 # a captured call writes no table that an eager one would read
    assert packs(fake.kernels(lambda: s.density(1))) == 0
    fake.L.fake_capture(0)
    first = fake.kernels(lambda: s.density(1))
    assert packs(first) == 1
    s.close()
    s = fake.space(6, 7)
    assert s.set_integrals(*mc.lieb_integrals(7, 1.0)) == OK
    assert packs(fake.unfinished(lambda: s.density(1))) == 0
    s.close()


def test_calls_without_pool_memory_take_the_direct_form(fake):
    s = fake.space(12, 10)
    assert s.set_integrals(*mc.lieb_integrals(10, 1.0)) == OK
    for call in (s.apply_h, s.apply_h_adjoint, lambda: s.rows(0, s.nc)):
        for got, refused in (("contact", False), ("direct", True), ("contact", False)):
            fake.L.fake_fail_pool(0 if refused else -1, 0)
            assert forms(fake.kernels(call)) == {got}
    t = fake.space(13, 10)
    fake.L.fake_headroom(1 << 20)          # its S takes 51 MB, the pool holds 28
    assert t.set_integrals(*mc.lieb_integrals(10, 1.0)) == OK
    assert forms(fake.kernels(t.apply_h)) == {"direct"}
    t.close()
    s.close()


@pytest.mark.parametrize("N,form", [(18, "contact"), (19, "direct")])
def test_the_contact_scratch_is_at_most_2_gib(fake, N, form):
    s = fake.space(N, 11)                  # S of 1.8 and 2.8 GB
    assert s.set_integrals(*mc.lieb_integrals(11, 1.0)) == OK
    assert forms(fake.kernels(s.apply_h)) == {form}
    s.close()
