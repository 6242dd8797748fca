"""Batches in the contact form with ten and eleven orbitals (from 131,072 and
98,304 rows together, or with as few launches as the direct form): E0 against
single solves in the direct form at the repository's 1e-10, members of very
different sizes, and one member's integrals changed in between."""
import numpy as np
import pytest

import mcpi_b200 as mc
from test_gpu_many_bosons import finite_range

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [[(10, 10), (9, 10), (2, 10)], [(9, 11), (6, 11), (2, 11)], [(3, 10)] * 20,
                                     [(3, 11)] * 30 + [(4, 12)]])
def test_batched_contact_form(members):
    lm = 24
    b = mc.Batch(members, lm)
    ints = [mc.lieb_integrals(M, 0.5 + 0.3 * x) for x, (N, M) in enumerate(members)]
    starts = [mc.random_problem(N, M, 80 + x)[0] for x, (N, M) in enumerate(members)]
    for change in (None, finite_range, mc.lieb_integrals):
        if change:
            ints[1] = change(members[1][1], 1.7)
        ref = []
        for x, ((N, M), (Ho, Hint), C) in enumerate(zip(members, ints, starts)):
            b.set_integrals(x, Ho, Hint)
            b.set_start(x, C)
            sp = mc.FockSpace(N, M)
            sp.set_option(mc.OPT_DIRECT_HPSI, 1)
            sp.set_integrals(Ho, Hint)
            ref.append(sp.ground(C, lm)[0])
            sp.close()
        E, it = b.run()
        assert np.abs(E - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
    b.close()
