"""The one-launch Lanczos near the largest spaces it takes (5,500 rows), where
blocks hold more than one tile of 32 rows, and at the fewest steps there: alpha,
beta, the basis and the Ritz vector are the launch sequence's bit for bit."""
import pytest

from test_gpu_small_lanczos import test_small_lanczos_is_the_launch_sequence_bit_for_bit as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,lm,kind", [(6, 10, 60, "lieb"), (9, 7, 40, "gauss"), (15, 5, 120, "lieb"),
                                         (11, 6, 35, "gauss"), (26, 4, 70, "lieb")])
def test_largest_spaces(N, M, lm, kind):
    check(N, M, lm, kind)
