"""The product sumcheck at the sizes where its rounds change form: wholly in one
block (up to 2^9 points), launched rounds before it, and fixes with the
challenge's table from 2^16 (three polynomials) or 2^18 pairs on; and every round
launched, down to the last, under a long pending transcript.  Every output and the transcript against the oracle, on values with zero, all-ones and
repeated entries among uniform ones."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [(k, n) for k in (2, 3) for n in (1, 2, 5, 6, 8, 9, 10, 11, 12)] + [(3, 17), (3, 18),
                                                                                                  (2, 19), (2, 20)])
def test_every_round_form_matches_the_oracle(built_lib, k, n):
    _check(built_lib, k, n, bytes(range(40)))


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 6, 7, 8, 11])
def test_launched_rounds_match_the_oracle(built_lib, k, n):
    _check(built_lib, k, n, bytes(range(250)) * 40)


def _check(bg, k, n, past):
    polys = rand.random_elems(k << n, 8800 + 32 * k + n)
    polys[::7] = 0
    polys[3::11] = 255
    polys[5::13] = polys[1]
    claim = rand.random_elems(1, 17 * n + k)
    ch = bg.GenericChallenger.keccak256()
    ch.observe(past)
    got = bg.prove_sumcheck(k, polys, claim, ch.clone())
    want = O.sumcheck_prove(k, n, polys, claim, ch.state())
    for a, b in zip(got, want):
        assert np.array_equal(np.asarray(a).reshape(-1), np.asarray(b).reshape(-1))
