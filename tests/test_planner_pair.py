"""The learned planner where packed-pair kernels exist (complex64 2^15..2^24):
the model has no features for them and they are the choice, as they are
without a planner (host only: no kernel runs)."""
import ctypes

import pytest

import algofft
from algofft import planner as P


def _choose(prec, n, batch, real):
    buf = ctypes.create_string_buffer(128)
    algofft.check(algofft.lib().gfft_planner_choose(prec, n, batch, 1, real, buf, 128))
    return buf.value.decode()


@pytest.mark.parametrize("n", [1 << k for k in range(15, 25)])
def test_learned_choice_is_the_packed_pair_variant(n):
    P.Model.load(P.DEFAULT_MODEL).install()
    for batch in (0, 1, 64):
        for real in (0, 1):
            tok = _choose(0, n, batch, real)
            assert tok.endswith("-pair") and tok in algofft.Variants(n)
