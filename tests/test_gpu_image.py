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


@pytest.mark.parametrize("d,ms,width,rows,lo,hi,odd", [
    (128, 12, 1 << 14, 1, -128, 128, None),   # every value that fits a byte
    (128, 4, 64, 3, -128, 128, None),         # the fewest elements
    (128, 4, 1 << 14, 2, -1, 2, 128),         # ternary but for one value past the byte, late in the rows
    (128, 4, 1 << 14, 2, -1, 2, -129),
    (256, 7, 1 << 13, 2, -128, 128, None),
    (256, 3, 1 << 13, 1, -128, -127, None),   # all at the lower end: the largest sums
    (256, 3, 1 << 13, 1, -1, 2, 128),
    (128, 3, 1 << 13, 1, -128, -127, None),
    (128, 3, 1 << 15, 4, -128, 128, None),    # tens of items per CTA: every ring of the pipeline wraps
    (256, 3, 1 << 14, 4, -128, 128, None),
])
def test_commit_short_values(api, oracle, d, ms, width, rows, lo, hi, odd):
    """Short witnesses go through the byte transform on the tensor cores; one
    value outside [-128, 127] sends the whole witness to the FP64 transform."""
    q = Q[d]
    p = P.make_params(d, q, ms, max(width, 128), 1)
    v = np.random.default_rng(width + rows).integers(lo, hi, size=(rows, width, d))
    if odd is not None:
        v[-1, -5, d - 3] = odd
    w = np.where(v < 0, q + v, v).astype(np.uint64)
    want = oracle.commit_ck(p, 2, w)
    ctx = api.Context(p, crs_seed=2)
    got = api.to_host(ctx.parallel_dot_series_matrix(api.to_dev(w)))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("d,folding,rounds,log_wit,bound", [
    (128, False, 3, 14, 1),         # the relation's ternary witness
    (128, False, 3, 14, 127),       # the largest that stays short in round 0; digits above 7 bits later
    (128, False, 3, 14, 128),       # round 0 wide, later rounds on their own sizes
    (128, False, 5, 16, 1),         # more statement rows than one tensor-core pass holds
    (128, False, 2, 13, 40000),     # every round wide, the projected row beyond two limbs
    (128, True, 1, 12, 1),
    (128, True, 1, 12, 127),
    (128, True, 1, 12, 5000),
    (256, False, 2, 13, 1),
    (256, False, 2, 13, 200),
    (256, True, 1, 11, 127),
])
def test_prove_short_and_wide(api, oracle, d, folding, rounds, log_wit, bound):
    """A proof's rounds take the byte steps while the witness is short and the
    word steps once it is not; the bytes are the oracle's either way."""
    q = Q[d]
    p = P.make_params(d, q, 3, 1 << log_wit, rounds, folding)
    v = np.random.default_rng(bound + d).integers(-bound, bound + 1, size=(p.init_wit_rep, p.wit_len, d))
    w = np.where(v < 0, q + v, v).astype(np.uint64)
    rc, want, _ = oracle.prove(p, 5, 6, witness=w)
    assert rc == 0
    ctx = api.Context(p, crs_seed=5)
    got = ctx.prove(6, witness=w)
    assert np.array_equal(got, want)
    pr = api.Prover(ctx)
    pr.set_overlap()
    pr.set_graph()
    import torch
    dw, out = api.to_dev(w), torch.zeros(ctx.proof_bytes, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        pr.enqueue(6, out, dw)
        pr.sync()
        assert np.array_equal(out.cpu().numpy(), want)
    pr.close()


@pytest.mark.parametrize("d,rows,width,lo,hi,odd", [
    (128, 1, 1 << 16, -128, 128, None),   # more chunks than CTAs: both accumulators and every ring wrap
    (128, 8, 1 << 13, -128, -127, None),  # long chunks, a part of the output rows per CTA, the largest sums
    (256, 3, 768 * 5, -128, 128, None),
    (512, 2, 512, -1, 2, 128),            # one value past the byte
    (128, 4, 4096, -1, 2, -129),
])
def test_project_tiles(api, oracle, d, rows, width, lo, hi, odd):
    """Projection of word rows through byte tiles, or exactly when a value does not fit."""
    from helpers import proj_challenge
    q = Q[d]
    v = np.random.default_rng(width + d).integers(lo, hi, size=(rows, width, d))
    if odd is not None:
        v[-1, -3, d - 5] = odd
    w = np.where(v < 0, q + v, v).astype(np.uint64)
    iz, sg = proj_challenge(5, 2, rows * 256)
    want = oracle.project(w, q, iz, sg)
    assert np.array_equal(api.to_host(api.project(api.to_dev(w), q, 5, 2)), want)


@pytest.mark.parametrize("d,rows,width,lo,hi,c_hi,odd", [
    (128, 8, 8193, -31, 32, 1, None),      # ternary challenges, one element past a tile
    (128, 8, 8255, -128, -127, 127, None),  # the largest sums, one element short of a tile
    (128, 4, 16385, -128, 128, 127, 128),  # a row value past the byte: the transforms
    (128, 4, 16400, -1, 2, 128, None),     # a challenge past it
    (128, 1, 1 << 16, -128, 128, 1, None),
    (256, 8, 4097, -128, 128, 1, None),
    (256, 8, 4100, -1, 2, 1, -129),
])
def test_fold_tiles(api, oracle, d, rows, width, lo, hi, c_hi, odd):
    """Long folds of word rows through byte tiles, or the transforms when a value does not fit."""
    q = Q[d]
    rng = np.random.default_rng(width + d)
    v = rng.integers(lo, hi, size=(rows, width, d))
    if odd is not None:
        v[-1, -1, d - 5] = odd
    cv = rng.integers(-c_hi, c_hi + 1, size=(rows, d)) if c_hi != 127 else np.full((rows, d), 127)
    cv[0, 1] = c_hi
    w, c = (np.where(x < 0, q + x, x).astype(np.uint64) for x in (v, cv))
    got = api.to_host(api.fold(api.to_dev(w), q, api.to_dev(c)))
    assert np.array_equal(got, oracle.fold(w, q, c))


def near_short(q):
    """Residues far from zero whose low 32 bits look like a short value's."""
    hi = (q >> 32) << 32
    return [(1 << 32) - 32896, (1 << 32) - 129, (1 << 32) - 128, (1 << 32) - 1, 1 << 32, (1 << 32) + 1, hi, hi + 0x7880,
            q - (1 << 32), q - (1 << 32) + 1, q >> 1, (q >> 1) + 1]


@pytest.mark.parametrize("d", [128, 256])
def test_values_near_short(api, oracle, d):
    """One such residue among ternary values, and (proofs) alone, so that the
    projected row holds it and its negative: everything is the oracle's."""
    q = Q[d]
    p = P.make_params(d, q, 3, 1 << 13, 2)
    ctx, pc = api.Context(p, crs_seed=5), P.make_params(d, q, 3, 128, 1)
    rng = np.random.default_rng(d)
    A = rand_mod(rng, (3, 128, d), q)
    key, small = api.DenseKey(api.to_dev(A), q), api.Context(pc, crs_seed=5)
    tern = rng.integers(-1, 2, size=(1, 1 << 13, d))
    tern = np.where(tern < 0, q + tern, tern).astype(np.uint64)
    for v in near_short(q):
        w = tern[:, :128].copy()
        w[0, 77, 9] = v
        assert np.array_equal(api.to_host(small.parallel_dot_series_matrix(api.to_dev(w))), oracle.commit_ck(pc, 5, w)), v
        assert np.array_equal(api.to_host(key.commit(api.to_dev(w))), oracle.dense_commit(A, w, q)), v
        for base in (tern, np.zeros_like(tern)):
            w = base.copy()
            w[0, 4321, 3] = v
            rc, want, _ = oracle.prove(p, 5, 6, witness=w)
            assert rc == 0
            assert np.array_equal(ctx.prove(6, witness=w), want), (v, int(base.any()))
    key.close()


@pytest.mark.parametrize("d,folding,log_wit,rounds", [(128, False, 13, 2), (128, True, 12, 1), (256, False, 13, 2),
                                                      (512, False, 13, 2)])
def test_prove_word_aligned_witness(api, oracle, cuda, d, folding, log_wit, rounds):
    """A device witness on any word boundary gives the oracle's proof, by
    direct launches and by graph replay, and stays as it was."""
    q = Q[d]
    p = P.make_params(d, q, 3, 1 << log_wit, rounds, folding)
    v = np.random.default_rng(d).integers(-1, 2, size=(p.init_wit_rep, p.wit_len, d))
    w = np.where(v < 0, q + v, v).astype(np.uint64)
    rc, want, _ = oracle.prove(p, 5, 6, witness=w)
    assert rc == 0
    ctx = api.Context(p, crs_seed=5)
    dw = api.to_dev(np.concatenate([[0], w.reshape(-1)]))[1:]
    assert dw.data_ptr() % 16 == 8
    out = cuda.zeros(ctx.proof_bytes, dtype=cuda.uint8, device="cuda")
    for graph in (False, True):
        pr = api.Prover(ctx)
        pr.set_graph(graph)
        for _ in range(2):
            out.zero_()
            cuda.cuda.synchronize()
            pr.enqueue(6, out, dw)
            pr.sync()
            assert np.array_equal(out.cpu().numpy(), want)
        pr.close()
    assert np.array_equal(api.to_host(dw), w.reshape(-1))


def test_commits_of_many_threads(api, oracle):
    """Host threads whose launches need different amounts of shared memory."""
    import ctypes
    import threading
    import torch
    from salsaa_b200 import lib
    q, p = P.Q0, P.make_params(128, P.Q0, 12, 1 << 9, 1)
    ctx = api.Context(p, crs_seed=5)
    wants, errors = {}, []
    for rows in (1, 9):
        w = rand_mod(np.random.default_rng(rows), (rows, 1 << 9, 128), q)
        wants[rows] = (w, oracle.commit_ck(p, 5, w))

    def work(rows):
        w, want = wants[rows]
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            dw, out = api.to_dev(w), api.dev_empty((12, rows, 128))
            for _ in range(1000):
                rc = lib().salsaa_commit(ctx.h, api._p(dw), rows, 1 << 9, api._p(out), ctypes.c_void_p(s.cuda_stream))
                if rc:
                    errors.append((rows, rc))
                    return
            if not np.array_equal(api.to_host(out), want):
                errors.append((rows, "wrong"))

    threads = [threading.Thread(target=work, args=(r,)) for r in (1, 9) * 4]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
