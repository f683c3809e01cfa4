"""Sumcheck passes over Gram matrices (sum_check, src/subroutines/
fast_norm_check.rs:135-320) against the CPU oracle, bit-exact, where the passes
change: one tile, the first length with a second tensor-core pass, the largest
bytes, moduli at both ends of the range, and a run longer than one segment."""
import numpy as np
import pytest

from helpers import nc_challenges, rand_mod
from salsaa_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(gpu_lib, cuda):
    from salsaa_b200 import api as A
    return A


@pytest.mark.parametrize("rows,n,d,q,top", [
    (1, 1 << 12, 128, P.Q0, False),   # one tile
    (1, 1 << 12, 128, P.Q0, True),
    (3, 1 << 13, 64, P.Q62, False),   # 62-bit modulus
    (2, 1 << 13, 64, P.Q62, True),
    (5, 1 << 16, 256, P.Q1, False),
    (2, 1 << 13, 16, (1 << 47) + 5, True),  # a modulus just above 2^47
    (3, 1 << 22, 128, P.Q0, False),   # two tensor-core passes
    (8, 1 << 21, 128, P.Q0, False),   # as many rows as the Gram room takes
])
def test_sumcheck_gram(api, oracle, rows, n, d, q, top):
    w = np.full((rows, n), q - 1, dtype=np.uint64) if top else rand_mod(np.random.default_rng(n + rows), (rows, n), q)
    claims, polys = api.sum_check(api.to_dev(w), d, q, 7, 2)
    claims, polys = api.to_host(claims), api.to_host(polys)
    nr = n.bit_length() - 1
    for rep in range(2):
        cs = nc_challenges(7, 2, rep, nr, q)
        for k in range(rows):
            claim, want, _ = oracle.sumcheck(w[k], q, cs)
            assert int(claims[k]) == claim
            assert np.array_equal(polys[rep, :, k], want), (rep, k)


def test_sumcheck_gram_segments(api, cuda):
    """A constant vector folds to itself: round t has the polynomial (h v^2, 0, 0)."""
    q, n = P.Q0, 1 << 28
    w = cuda.full((1, n), q - 1, dtype=cuda.int64, device="cuda")
    claims, polys = api.sum_check(w, 128, q, 7, 2)
    assert int(api.to_host(claims)[0]) == n % q
    polys = api.to_host(polys)
    nr = n.bit_length() - 1
    want = np.array([[(n >> (t + 1)) % q, 0, 0] for t in range(nr)], dtype=np.uint64)
    for rep in range(2):
        assert np.array_equal(polys[rep, :, 0], want)
