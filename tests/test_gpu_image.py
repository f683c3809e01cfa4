"""Key rows over byte images of the witness (the tensor-core commitment path of
parallel_dot_series_matrix, src/arithmetic.rs:459-505) against the CPU oracle,
bit-exact, where the tiling changes: one 64-element chunk, several key blocks
stacked or sharing key tiles, the largest key and row counts, extreme values."""
import numpy as np
import pytest

from helpers import rand_mod
from salsaa_b200 import params as P

pytestmark = pytest.mark.gpu
Q = {128: P.Q0, 256: P.Q1, 512: P.Q2}


@pytest.fixture(scope="module")
def api(gpu_lib, cuda):
    from salsaa_b200 import api as A
    return A


@pytest.mark.parametrize("d,ms,width,wit_len,rows,top", [
    (128, 12, 64, 128, 1, False),        # one chunk, narrower than the key block
    (128, 12, 1 << 17, 1 << 17, 1, False),  # eight key blocks stacked, two accumulators
    (128, 12, 1 << 16, 1 << 16, 3, False),  # two key blocks stacked, two accumulators
    (128, 12, 1 << 14, 1 << 15, 9, True),   # the widest tile, every byte at its largest
    (128, 13, 1 << 15, 1 << 15, 4, False),  # more than 12 key rows: one accumulator
    (128, 18, 1 << 14, 1 << 14, 9, True),   # the largest key table
    (128, 1, 1 << 14, 1 << 14, 2, False),   # one key row
    (256, 7, 1 << 15, 1 << 15, 3, False),
    (256, 16, 1 << 9, 1 << 10, 8, True),
    (512, 4, 1 << 14, 1 << 14, 5, False),
    (512, 3, 128, 128, 7, True),
])
def test_commit_image(api, oracle, d, ms, width, wit_len, rows, top):
    q = Q[d]
    p = P.make_params(d, q, ms, wit_len, 1)
    w = (np.full((rows, width, d), q - 1, dtype=np.uint64) if top
         else rand_mod(np.random.default_rng(width + rows), (rows, width, d), q))
    want = oracle.commit_ck(p, 9, w)
    ctx = api.Context(p, crs_seed=9)
    got = api.to_host(ctx.parallel_dot_series_matrix(api.to_dev(w)))
    assert np.array_equal(got, want)
