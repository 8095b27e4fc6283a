"""The work a prover has this library do, as cases that can be timed and compared.

A case is one call (or the few calls that belong together) through bc_ntt's public entry
points, at the sizes a proof system uses them: columns of 2^3 to 2^24 Goldilocks words, 1 to
256 of them, low-degree extensions by 2, 4 or 8.  Inputs are uniform in [0, p), the
distribution of trace columns after blinding; every output is a field element in canonical
form, a whole number, so two correct implementations agree bit for bit.
"""
import math
import os
import random
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "era-boojum-cuda_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bc_ntt  # noqa: E402

P = bc_ntt.P

# Words that one drawn case may write: an eighth of what the largest listed case writes.
DRAW_WORDS = 1 << 27


def listed():
    return [
        # one short column: a public-input or boundary polynomial, where the call itself is the cost
        {"name": "ntt_1x2e10", "kind": "ntt", "log_n": 10, "cols": 1, "gap": 0, "mode": "forward", "log_ext": 0},
        # a small forward transform, the benchmark's latency workload
        {"name": "ntt_16x2e16", "kind": "ntt", "log_n": 16, "cols": 16, "gap": 0, "mode": "forward", "log_ext": 0},
        # monomial form of an odd number of trace columns, in place
        {"name": "intt_33x2e19", "kind": "ntt", "log_n": 19, "cols": 33, "gap": 0, "mode": "inverse_in_place", "log_ext": 0},
        # one coset of a quotient's domain, columns inside a larger matrix at odd distances
        {"name": "coset_70x2e20", "kind": "ntt", "log_n": 20, "cols": 70, "gap": 5, "mode": "forward", "log_ext": 2},
        # an extension of a small circuit
        {"name": "lde_16x2e13_b4", "kind": "lde", "log_n": 13, "cols": 16, "log_b": 2, "layout": "coset_major"},
        # a mid-sized circuit with an odd column count, each column's cosets side by side
        {"name": "lde_93x2e18_b8", "kind": "lde", "log_n": 18, "cols": 93, "log_b": 3, "layout": "column_major"},
        # the benchmark's workload: the trace of a large circuit
        {"name": "lde_128x2e22_b2", "kind": "lde", "log_n": 22, "cols": 128, "log_b": 1, "layout": "coset_major"},
        # the longest columns the reference takes
        {"name": "lde_10x2e24_b2", "kind": "lde", "log_n": 24, "cols": 10, "log_b": 1, "layout": "coset_major"},
        # many small circuits of uneven size, extended by one persistent launch
        {"name": "batch_192", "kind": "batch", "jobs": 192, "lo": 10, "hi": 16, "max_cols": 8, "shapes": 11},
        # columns in pinned host memory, extensions back to pinned host memory
        {"name": "host_16x2e20_b2", "kind": "host", "log_n": 20, "cols": 16, "log_b": 1},
        # requests of a proving service on device-resident columns
        {"name": "serve_96", "kind": "serve", "jobs": 96, "lo": 10, "hi": 16, "max_cols": 16, "shapes": 23},
        # openings: all columns evaluated at one point of the quadratic extension
        {"name": "open_64x2e20", "kind": "open", "log_n": 20, "cols": 64},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choices(["ntt", "lde", "batch", "host", "serve", "open"], [4, 6, 1, 1, 1, 1])[0]
    if kind == "ntt":
        log_n = rng.randint(3, 24)
        cols = _log_int(rng, 1, max(1, min(256, DRAW_WORDS >> log_n)))
        mode = rng.choice(["forward", "inverse", "inverse_in_place", "forward_in_place", "forward_b2n"])
        return {"kind": kind, "log_n": log_n, "cols": cols, "gap": rng.choice([0, 0, 2, 7, 64]), "mode": mode,
                "log_ext": rng.choice([0, 1, 2, 3])}
    if kind == "lde":
        log_b = rng.randint(1, 3)
        log_n = rng.randint(6, 24)
        cols = _log_int(rng, 1, max(1, min(256, DRAW_WORDS >> (log_n + log_b))))
        return {"kind": kind, "log_n": log_n, "cols": cols, "log_b": log_b,
                "layout": rng.choice(["coset_major", "column_major"])}
    if kind in ("batch", "serve"):
        lo = rng.randint(8, 12)
        return {"kind": kind, "jobs": _log_int(rng, 16, 192), "lo": lo, "hi": lo + rng.randint(2, 5),
                "max_cols": rng.randint(2, 12), "shapes": rng.randrange(1 << 20)}
    if kind == "host":
        log_n = rng.randint(14, 20)
        return {"kind": kind, "log_n": log_n, "cols": _log_int(rng, 1, min(64, 1 << (24 - log_n))), "log_b": rng.randint(1, 2)}
    log_n = rng.randint(8, 22)
    return {"kind": kind, "log_n": log_n, "cols": _log_int(rng, 1, min(128, 1 << (27 - log_n)))}


def _shapes(case):
    """(log_n, cols, log_blowup) of a batch's jobs or a service's requests."""
    rng = random.Random(case["shapes"])
    return [(rng.randint(case["lo"], case["hi"]), rng.randint(1, case["max_cols"]), rng.randint(1, 2))
            for _ in range(case["jobs"])]


def _words(count, seed, device="cuda"):
    """`count` words uniform in [0, p), as int64."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (count,), dtype=torch.int64, device="cuda", generator=g)
    x = torch.where((x < 0) & (x >= -(2**32 - 1)), x & (2**32 - 1), x)  # words >= p, one in 2^32
    return x if device == "cuda" else x.cpu().pin_memory()


_server = None


def _ready():
    """What a program does once: the tables, and the plan table tuned for this GPU."""
    if not _ready.done:
        bc_ntt.Context.create()
        bc_ntt.load_tuned_plans()
        _ready.done = True


_ready.done = False


def prepare(case, seed):
    global _server
    _ready()
    kind = case["kind"]
    s = {"case": case}
    if kind == "ntt":
        s["stride"] = (1 << case["log_n"]) + case["gap"]
        s["in"] = _words(s["stride"] * case["cols"], seed)
        if not case["mode"].endswith("in_place"):
            s["out"] = torch.zeros_like(s["in"])
    elif kind == "lde":
        s["in"] = _words(case["cols"] << case["log_n"], seed)
        s["out"] = torch.empty(case["cols"] << (case["log_n"] + case["log_b"]), dtype=torch.int64, device="cuda")
    elif kind in ("batch", "serve"):
        shapes = _shapes(case)
        s["in"] = _words(sum(c << n for n, c, _ in shapes), seed)
        s["out"] = torch.empty(sum(c << (n + b) for n, c, b in shapes), dtype=torch.int64, device="cuda")
        jobs, i, o = [], 0, 0
        for n, c, b in shapes:
            jobs.append((s["in"][i:i + (c << n)], s["out"][o:o + (c << (n + b))], n, c, b))
            i, o = i + (c << n), o + (c << (n + b))
        if kind == "batch":
            s["plan"] = bc_ntt.LdeBatch(jobs)
        else:
            s["jobs"] = jobs
            if _server is None:  # one server for the process
                _server = bc_ntt.LdeServer(256 << 20, slots=2)
    elif kind == "host":
        s["in"] = _words(case["cols"] << case["log_n"], seed, "cpu")
        s["out"] = torch.empty(case["cols"] << (case["log_n"] + case["log_b"]), dtype=torch.int64, pin_memory=True)
        s["workspace"] = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    else:
        n = 1 << case["log_n"]
        s["ys"] = _words(case["cols"] << case["log_n"], seed)
        s["x"] = _words(2, seed + 1)
        s["cf"] = torch.empty(2, dtype=torch.int64, device="cuda")
        s["coeffs"] = torch.empty(2 * n, dtype=torch.int64, device="cuda")
        words, _ = bc_ntt.get_batch_eval_temp_storage_sizes(bc_ntt.EVAL_BASE_AT_EXT, n, case["cols"])
        s["temp"] = torch.empty(max(1, words), dtype=torch.int64, device="cuda")
        s["evals"] = torch.empty(2 * case["cols"], dtype=torch.int64, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ntt":
        log_n, cols, mode, e = case["log_n"], case["cols"], case["mode"], case["log_ext"]
        k = (1 << e) - 1  # the last coset; without an extension the plain domain
        bitrev, inverse = mode.startswith("inverse") or mode == "forward_b2n", mode.startswith("inverse")
        if mode.endswith("in_place"):
            bc_ntt.batch_ntt_in_place(s["in"], log_n, cols, 0, s["stride"], bitrev, inverse, e, k)
            return s["in"]
        bc_ntt.batch_ntt_out_of_place(s["in"], s["out"], log_n, cols, 0, 0, s["stride"], s["stride"], bitrev, inverse,
                                      e, k)
        return s["out"]
    if kind == "lde":
        n = 1 << case["log_n"]
        if case["layout"] == "coset_major":
            bc_ntt.lde(s["in"], s["out"], case["log_n"], case["cols"], case["log_b"])
        else:
            bc_ntt.lde(s["in"], s["out"], case["log_n"], case["cols"], case["log_b"], n, n << case["log_b"], n)
        return s["out"]
    if kind == "batch":
        s["plan"].run()
        return s["out"]
    if kind == "serve":
        ids = [_server.submit_device(*j) for j in s["jobs"]]
        for i in ids:
            _server.wait(i)
            _server.release(i)
        return s["out"]
    if kind == "host":
        bc_ntt.lde_host(s["in"], s["out"], case["log_n"], case["cols"], case["log_b"], s["workspace"])
        return s["out"]
    n = 1 << case["log_n"]
    # values of a coset in bit-reversed order, as an extension leaves them
    bc_ntt.precompute_lagrange_coeffs(s["x"], s["cf"], 7, s["coeffs"], True, ext=True)
    bc_ntt.batch_eval(bc_ntt.EVAL_BASE_AT_EXT, s["ys"], n, case["cols"], s["coeffs"], s["temp"], None, s["evals"])
    return {"coeffs": s["coeffs"], "evals": s["evals"]}


def work(case):
    """Words in and out once; a butterfly as one product, one sum and one difference in the field."""
    kind = case["kind"]
    if kind == "ntt":
        words = case["cols"] << case["log_n"]
        return {"bytes": 16 * words, "flops": 3 * (words // 2) * case["log_n"] + (words if case["log_ext"] else 0)}
    if kind == "open":
        n = 1 << case["log_n"]
        # two products and two sums a value; some ten products a coefficient of the extension
        return {"bytes": 8 * (n * case["cols"] + 2 * n + 2 * case["cols"]), "flops": 4 * n * case["cols"] + 20 * n}
    shapes = [(case["log_n"], case["cols"], case["log_b"])] if kind in ("lde", "host") else _shapes(case)
    b = f = 0
    for n, c, lb in shapes:
        words = c << n
        b += 8 * words * (1 + (1 << lb))
        f += 3 * (words // 2) * n * (1 + (1 << lb)) + words
    return {"bytes": b, "flops": f}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """No floating output to compare: every word is exact already, and compared as it is."""
    return None
