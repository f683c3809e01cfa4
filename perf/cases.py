"""The measured workloads of the SALSAA prover: its whole proofs and its steps.

Every case goes through the package's public interface (salsaa_b200.api) the
way a host program calls it: device-resident inputs, results in device
buffers, and the objects such a program keeps (a context with its CRS tables,
proof slots, a dense key) made once beforehand.  Values are what the protocol
meets: ternary witnesses, short decomposition digits, uniform residues for
transforms and keys.  All outputs are whole numbers: residues in [0, q) or
proof bytes.

Kinds of case:
  ntt             batched negacyclic transform, either direction, the protocol's
                  incomplete form (50-bit primes) or the full form (62-bit prime)
  poly_mul        batched negacyclic products (forward, pointwise, inverse)
  commit          commitment-key rows times witness rows
  sum_check       both repetitions of the norm-check sumcheck
  sum_check_batch many sumchecks of uneven lengths in one call
  project         the ternary projection of a split witness
  fold_decompose  the end of a round: fold the rows, then split into digits
  dense           C = A * W with a dense key
  prove           whole proofs: SNARK or folding step, one or several in flight
"""
import math

import torch

from salsaa_b200 import api
from salsaa_b200 import params as P

MODULUS = {128: P.Q0, 256: P.Q1, 512: P.Q2}
# commitment-key rows of the parameter sets A0, A1, A2
KEY_ROWS = {128: 12, 256: 7, 512: 4}
LARGEST = 1 << 26  # coefficients of the largest witness, that of A0


def listed():
    return [
        # the smallest call: one column of ring elements back from evaluation form
        {"name": "ntt_small", "kind": "ntt", "n": 64, "q62": True, "incomplete": False, "inverse": True, "count": 48},
        # the A0 witness to slot form, the protocol's own transform
        {"name": "ntt_d128", "kind": "ntt", "n": 128, "q62": False, "incomplete": True, "inverse": False,
         "count": 1 << 19},
        # the transform microbenchmark at the 62-bit prime: forward, pointwise, inverse; a ragged batch
        {"name": "poly_mul_n256", "kind": "poly_mul", "n": 256, "count": 60001},
        # the first message of a folding step: 4 witness rows under 12 key rows (F0)
        {"name": "commit_f0", "kind": "commit", "d": 128, "rows": 4, "width": 1 << 17, "log_wit": 17},
        # the norm check of 2^24 coefficients
        {"name": "sum_check_2e24", "kind": "sum_check", "d": 128, "rows": 1, "log_n": 24, "digits": False},
        # 64 uneven instances between 2^16 and 2^22
        {"name": "sum_check_batch64", "kind": "sum_check_batch", "count": 64, "log_min": 16, "log_max": 22},
        # the projection of a middle round: 8 rows of digits after the split
        {"name": "project_8rows", "kind": "project", "d": 128, "rows": 8, "width": 1 << 15, "digits": True},
        # the end of a middle round, with a width that is no power of two
        {"name": "fold_decompose", "kind": "fold_decompose", "d": 128, "rows": 8, "width": 20001, "parts": 2},
        # the dense Ajtai commitment: 16 x 2^16 key, 8 columns of base-16 digits
        {"name": "dense_r8", "kind": "dense", "d": 128, "n": 16, "m": 1 << 16, "r": 8, "base": 16},
        # a small proof, where the launches count
        {"name": "prove_small", "kind": "prove", "d": 128, "rows": 4, "log_wit": 13, "rounds": 2, "folding": False,
         "in_flight": 1, "graph": False, "overlap": False},
        # the headline: one A0 proof, at the settings for low latency
        {"name": "prove_a0", "kind": "prove", "d": 128, "rows": 12, "log_wit": 19, "rounds": 8, "folding": False,
         "in_flight": 1, "graph": True, "overlap": True},
        # a service's folding steps (F0), four of them in flight
        {"name": "prove_f0_x4", "kind": "prove", "d": 128, "rows": 12, "log_wit": 17, "rounds": 1, "folding": True,
         "in_flight": 4, "graph": False, "overlap": False},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ntt", "poly_mul", "commit", "sum_check", "sum_check_batch", "project", "fold_decompose",
                       "dense", "prove", "prove"])
    if kind == "ntt":
        q62 = rng.random() < 0.4
        n = rng.choice([64, 128, 256, 1024] if q62 else [128, 256, 512])
        return {"kind": kind, "n": n, "q62": q62, "incomplete": not q62, "inverse": rng.random() < 0.5,
                "count": max(1, _log_uniform(rng, 1 << 11, LARGEST) // n)}
    if kind == "poly_mul":
        n = rng.choice([64, 128, 256, 1024])
        return {"kind": kind, "n": n, "count": max(1, _log_uniform(rng, 1 << 12, LARGEST // 2) // n)}
    if kind == "commit":
        d = rng.choice([128, 256, 512])
        rows = rng.randint(1, 9)
        lw = rng.randint(9, (LARGEST // (d * rows)).bit_length() - 1)
        return {"kind": kind, "d": d, "rows": rows, "width": 1 << lw, "log_wit": max(lw, 13)}
    if kind == "sum_check":
        rows = rng.randint(1, 4)
        return {"kind": kind, "d": rng.choice([128, 256, 512]), "rows": rows,
                "log_n": rng.randint(12, (LARGEST // rows).bit_length() - 1), "digits": rng.random() < 0.5}
    if kind == "sum_check_batch":
        lo = rng.randint(12, 16)
        return {"kind": kind, "count": rng.randint(8, 64), "log_min": lo, "log_max": rng.randint(lo + 2, 22)}
    if kind == "project":
        d, rows = rng.choice([128, 256, 512]), rng.choice([2, 4, 8])
        chunk = rows * 256
        return {"kind": kind, "d": d, "rows": rows,
                "width": chunk * max(1, _log_uniform(rng, 1 << 20, LARGEST) // (chunk * rows * d)),
                "digits": rng.random() < 0.7}
    if kind == "fold_decompose":
        d, rows = rng.choice([128, 256, 512]), rng.choice([2, 4, 8])
        return {"kind": kind, "d": d, "rows": rows, "width": _log_uniform(rng, 1 << 17, LARGEST) // (rows * d),
                "parts": rng.choice([2, 2, 3])}
    if kind == "dense":
        return {"kind": kind, "d": 128, "n": rng.choice([8, 16]), "m": 1 << rng.randint(12, 16),
                "r": rng.choice([1, 2, 5, 8]), "base": rng.choice([2, 16])}
    d = rng.choice([128, 128, 256, 512])
    tuned = rng.random() < 0.5
    if rng.random() < 0.4:
        return {"kind": kind, "d": 128, "rows": rng.choice([12, 13]), "log_wit": rng.randint(11, 17), "rounds": 1,
                "folding": True, "in_flight": rng.randint(1, 4), "graph": tuned, "overlap": tuned}
    lw = rng.randint(13, 20 - d.bit_length() + 7)
    return {"kind": kind, "d": d, "rows": KEY_ROWS[d], "log_wit": lw, "rounds": rng.randint(1, min(8, lw - 11)),
            "folding": False, "in_flight": rng.randint(1, 4) if lw <= 16 else 1, "graph": tuned, "overlap": tuned}


# ---- inputs --------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(shape, q, gen):
    return torch.randint(0, q, shape, dtype=torch.int64, device="cuda", generator=gen)


def _centred(shape, lo, hi, q, gen):
    """Values uniform in [lo, hi) as residues mod q."""
    w = torch.randint(lo, hi, shape, dtype=torch.int64, device="cuda", generator=gen)
    return w.add_((w < 0) * q)


def _ternary(shape, q, gen):
    """P(0) = 1/2, P(1) = P(-1) = 1/4, as residues mod q."""
    w = torch.randint(0, 4, shape, dtype=torch.int8, device="cuda", generator=gen)
    return ((w == 2).to(torch.int64)).add_((w == 3) * (q - 1))


def _short(shape, digits, q, gen):
    return _centred(shape, -31, 32, q, gen) if digits else _ternary(shape, q, gen)


def _batch_logs(case):
    """Lengths spread over the range, the same for every seed."""
    span = case["log_max"] - case["log_min"] + 1
    return [case["log_min"] + (5 * i + i // span) % span for i in range(case["count"])]


def prepare(case, seed):
    gen, kind = _gen(seed), case["kind"]
    s = {"kind": kind, "case": case, "seed": int(seed)}
    if kind in ("ntt", "poly_mul"):
        n = case["n"]
        s["q"] = q = P.Q62 if kind == "poly_mul" or case["q62"] else MODULUS[n]
        s["x"] = _uniform((case["count"], n), q, gen)
        s["out"] = api.dev_empty((case["count"], n))
        if kind == "poly_mul":
            s["y"] = _uniform((case["count"], n), q, gen)
    elif kind == "commit":
        d = case["d"]
        q = MODULUS[d]
        s["ctx"] = api.Context(P.make_params(d, q, KEY_ROWS[d], 1 << case["log_wit"], 1), seed & 0xFFFF)
        s["w"] = _ternary((case["rows"], case["width"], d), q, gen)
    elif kind == "sum_check":
        s["q"] = q = MODULUS[case["d"]]
        s["w"] = _short((case["rows"], 1 << case["log_n"]), case["digits"], q, gen)
    elif kind == "sum_check_batch":
        s["q"] = P.Q0
        s["vecs"] = [_ternary((1 << k,), P.Q0, gen) for k in _batch_logs(case)]
    elif kind == "project":
        s["q"] = q = MODULUS[case["d"]]
        s["w"] = _short((case["rows"], case["width"], case["d"]), case["digits"], q, gen)
    elif kind == "fold_decompose":
        s["q"] = q = MODULUS[case["d"]]
        s["w"] = _centred((case["rows"], case["width"], case["d"]), -31, 32, q, gen)
        s["c"] = _centred((case["rows"], case["d"]), -1, 2, q, gen)
    elif kind == "dense":
        half = case["base"] // 2
        s["q"] = q = MODULUS[case["d"]]
        s["key"] = api.DenseKey(_uniform((case["n"], case["m"], case["d"]), q, gen), q)
        s["w"] = _centred((case["r"], case["m"], case["d"]), -half, half, q, gen)
        s["slot"] = api.dev_empty(s["w"].shape)
        s["out"] = api.dev_empty((case["n"], case["r"], case["d"]))
    elif kind == "prove":
        d = case["d"]
        p = P.make_params(d, MODULUS[d], case["rows"], 1 << case["log_wit"], case["rounds"], case["folding"])
        s["ctx"] = ctx = api.Context(p, seed & 0xFFFF)
        s["slots"] = []
        for _ in range(case["in_flight"]):
            pr = api.Prover(ctx)
            pr.set_overlap(case["overlap"])
            pr.set_graph(case["graph"])
            w = _ternary((p.init_wit_rep, p.wit_len, d), p.q, gen)
            s["slots"].append((pr, w, torch.empty(ctx.proof_bytes, dtype=torch.uint8, device="cuda")))
    else:
        raise ValueError("unknown kind %r" % kind)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, case, seed = s["kind"], s["case"], s["seed"]
    if kind == "ntt":
        return api.ntt(s["x"], case["n"], s["q"], inverse=case["inverse"], incomplete=case["incomplete"],
                       out=s["out"])
    if kind == "poly_mul":
        return api.poly_mul(s["x"], s["y"], case["n"], s["q"], out=s["out"])
    if kind == "commit":
        return s["ctx"].parallel_dot_series_matrix(s["w"])
    if kind == "sum_check":
        return api.sum_check(s["w"], case["d"], s["q"], seed, 1)
    if kind == "sum_check_batch":
        claims, polys = api.sum_check_batch(s["vecs"], s["q"], seed, 1)
        return [claims, torch.cat(polys)]
    if kind == "project":
        return api.project(s["w"], s["q"], seed, 1)
    if kind == "fold_decompose":
        folded = api.fold(s["w"], s["q"], s["c"])
        digits, radix = api.decompose_matrix_by_chunks(folded[None], s["q"], case["parts"])
        return [folded, digits, radix]
    if kind == "dense":
        return s["key"].commit(s["w"], out=s["out"], w_slot=s["slot"])
    for i, (pr, w, proof) in enumerate(s["slots"]):
        pr.enqueue(seed * 64 + i, proof, w)
    for pr, _, _ in s["slots"]:
        pr.sync()
    return [proof for _, _, proof in s["slots"]]


def _transform_ops(words, n):
    """A butterfly is a product and two sums on two words."""
    return 1.5 * words * math.log2(n)


def work(case):
    """Bytes: the inputs once and the outputs once.  flops: products and sums
    mod q that the step is defined by."""
    kind = case["kind"]
    if kind in ("ntt", "poly_mul"):
        n, words = case["n"], case["count"] * case["n"]
        if kind == "poly_mul":
            return {"bytes": 24 * words, "flops": 3 * _transform_ops(words, n) + words}
        return {"bytes": 16 * words, "flops": _transform_ops(words, n // 2 if case["incomplete"] else n)}
    if kind == "commit":
        d, words = case["d"], case["rows"] * case["width"] * case["d"]
        ms = KEY_ROWS[d]
        return {"bytes": 8 * (words + ms * d + ms * case["rows"] * d),
                "flops": 4 * ms * words + _transform_ops(words, d // 2)}
    if kind == "sum_check":
        words = case["rows"] << case["log_n"]
        # each of the two repetitions halves its vector round by round: three products and a fold per pair
        return {"bytes": 8 * words + 8 * case["rows"] * (1 + 6 * case["log_n"]), "flops": 2 * 8 * words}
    if kind == "sum_check_batch":
        logs = _batch_logs(case)
        words = sum(1 << k for k in logs)
        return {"bytes": 8 * words + 8 * sum(1 + 3 * k for k in logs), "flops": 8 * words}
    if kind == "project":
        out = case["width"] * case["d"]
        return {"bytes": 8 * (case["rows"] + 1) * out, "flops": case["rows"] * 256 * out}
    if kind == "fold_decompose":
        out, rows, d = case["width"] * case["d"], case["rows"], case["d"]
        return {"bytes": 8 * (rows * (out + d) + out + case["parts"] * out),
                "flops": 4 * rows * out + (rows + 1) * _transform_ops(out, d // 2)}
    if kind == "dense":
        n, m, r, d = case["n"], case["m"], case["r"], case["d"]
        return {"bytes": 8 * d * (n * m + m * r + n * r), "flops": 4 * n * m * r * d}
    # prove: the witness in, the proof out; the commitments of every round
    d, rows, width = case["d"], case["rows"], 1 << case["log_wit"]
    p = P.make_params(d, MODULUS[d], rows, width, case["rounds"], case["folding"])
    k, ops = p.init_wit_rep, 0
    for rd in range(case["rounds"]):
        if not case["folding"] and rd:
            k *= 2
        ops += 4 * rows * (k + 0.5) * width * d + 16 * k * width * d
        k, width = 2, width if case["folding"] else width // 2
    words = p.init_wit_rep * p.wit_len * d
    return {"bytes": case["in_flight"] * (8 * words + api.proof_size(p)), "flops": case["in_flight"] * ops}


def exact(case, seed):
    """None: every output is an array of residues or bytes, right only when equal."""
    return None
