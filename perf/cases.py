"""The work a user has this framework do, as timed cases.

A case names a public entry point and its sizes; ``prepare`` makes what the
caller has in hand before the call, ``run`` is one call as a program makes it,
with everything it returns.  All arithmetic is exact (GF(2^32), GF(2^128),
BLAKE3, SHA-256), so outputs are whole numbers and bytes.
"""
import importlib
import math

import numpy as np
import torch

lg = importlib.import_module("ligerito-rust_b200")

QUERIES = 148


def listed():
    return [
        # One proof of the smallest generated config: all launches and latency.
        {"name": "prove16", "op": "prove", "log": 16, "cols": 6, "input": "device"},
        # The 2^20 config of the command-line program, its polynomial in
        # ordinary (pageable) host memory, as a program that just read or made
        # it has it.
        {"name": "prove20-host", "op": "prove", "log": 20, "cols": 6, "input": "pageable"},
        # The 2^24 headline config, the polynomial already on the device.
        {"name": "prove24", "op": "prove", "log": 24, "cols": 6, "input": "device"},
        # The same from pinned host memory: the end-to-end form of the
        # headline benchmark.
        {"name": "prove24-pinned", "op": "prove", "log": 24, "cols": 6, "input": "pinned"},
        # The largest proof of the benchmark.
        {"name": "prove28", "op": "prove", "log": 28, "cols": 6, "input": "device"},
        # A batch of equal small proofs in one call, as a proving service
        # groups its queue; an odd count.
        {"name": "lockstep18x23", "op": "lockstep", "log": 18, "cols": 6, "count": 23},
        # The other direction: verifying a 2^24 proof from its bytes.
        {"name": "verify24", "op": "verify", "log": 24, "cols": 6},
        # One commitment of a matrix of a program's own: few long columns, a
        # count that is no power of two.
        {"name": "commit14x40", "op": "commit", "log_m": 14, "n": 40},
        # The batched transform of the FFT benchmark, and the inverse on a
        # ragged batch of shorter vectors.
        {"name": "fft20x64", "op": "fft", "log": 20, "batch": 64},
        {"name": "ifft13x130", "op": "ifft", "log": 13, "batch": 130},
        # A multilinear polynomial evaluated in its top variables, more than
        # one launch takes.
        {"name": "partial22k9", "op": "partial", "log": 22, "k": 9},
        # A verifier's or a custom protocol's induced basis polynomial from an
        # opening of 64-word rows.
        {"name": "induce16", "op": "induce", "log": 16, "nch": 6, "queries": QUERIES},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    given = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in given:
            return case


def _draw(rng):
    op = rng.choice(2 * ["prove", "prove", "lockstep", "verify", "commit", "encode", "fft", "ifft", "partial",
                         "induce"] + ["eval013", "gf128"])
    if op == "prove":
        log = rng.randint(16, 26)
        return {"op": op, "log": log, "cols": rng.randint(4, min(7, log - 10)),
                "input": rng.choice(["device", "pageable", "pinned"])}
    if op == "lockstep":
        log = rng.randint(16, 21)
        return {"op": op, "log": log, "cols": rng.randint(4, min(7, log - 10)),
                "count": _log_uniform(rng, 2, min(64, 1 << (24 - log)))}
    if op == "verify":
        log = rng.randint(16, 25)
        return {"op": op, "log": log, "cols": rng.randint(4, min(7, log - 10))}
    if op in ("commit", "encode"):
        log_m = rng.randint(5, 18)
        return {"op": op, "log_m": log_m, "n": _log_uniform(rng, 1, min(256, 1 << (25 - log_m)))}
    if op in ("fft", "ifft"):
        log = rng.randint(1, 22)
        return {"op": op, "log": log, "batch": _log_uniform(rng, 1, 1 << min(16, 26 - log))}
    if op == "partial":
        log = rng.randint(4, 26)
        return {"op": op, "log": log, "k": rng.randint(1, min(12, log))}
    if op == "eval013":
        return {"op": op, "log": rng.randint(1, 25)}
    if op == "induce":
        return {"op": op, "log": rng.randint(6, 20), "nch": rng.randint(3, 7),
                "queries": rng.choice([QUERIES, rng.randint(1, 256)])}
    return {"op": op, "n": _log_uniform(rng, 1, 1 << 22)}


def _config(case):
    """The generated config of 2^log coefficients; with another number of
    first columns (2^cols), the same pattern of 16-column steps after it."""
    log, cols = case["log"], case["cols"]
    if cols == 6:
        return lg.config_for_size(log)
    dims, left = [], log - cols
    while not dims or left - 4 >= 10:
        left -= 4
        dims.append((1 << left, 16))
    return lg.ProverConfig(recursive_steps=len(dims), initial_dims=(1 << (log - cols), 1 << cols), dims=dims,
                           initial_k=cols, ks=[4] * len(dims))


def _words(gen, n):
    """n uniform 32-bit field elements on the device."""
    return torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=gen)


def _host_words(rng, n):
    return rng.integers(0, 1 << 32, size=n, dtype=np.uint32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    op = case["op"]
    s = {"op": op, "ctx": lg.default_context()}
    if op == "prove":
        s["cfg"] = _config(case)
        poly = _words(gen, 1 << case["log"])
        if case["input"] == "pinned":
            s["keep"] = poly.cpu().pin_memory()
            poly = s["keep"].numpy().view(np.uint32)
        elif case["input"] == "pageable":
            poly = poly.cpu().numpy().view(np.uint32)
        s["poly"], s["record"] = poly, np.zeros(_record_size(s["cfg"]), np.uint8)
    elif op == "lockstep":
        s["cfg"] = _config(case)
        s["records"] = np.zeros((case["count"], _record_size(s["cfg"])), np.uint8)
        s["polys"] = _words(gen, case["count"] << case["log"]).view(case["count"], -1)
    elif op == "verify":
        cfg = _config(case)
        s["proof"] = lg.prover(cfg, _words(gen, 1 << case["log"]), s["ctx"]).to_bytes()
        s["cfg"] = lg.verifier_config_for(cfg)
    elif op in ("commit", "encode"):
        s["log_m"], s["n"] = case["log_m"], case["n"]
        s["poly"] = _words(gen, case["n"] << case["log_m"])
    elif op in ("fft", "ifft"):
        s["log"] = case["log"]
        s["data"] = _words(gen, case["batch"] << case["log"])
    elif op == "partial":
        s["evals"], s["rs"] = _words(gen, 1 << case["log"]), _host_words(rng, case["k"])
    elif op == "eval013":
        s["f"], s["g"] = _words(gen, 1 << case["log"]), _words(gen, 1 << case["log"])
    elif op == "induce":
        s["log"], nq = case["log"], case["queries"]
        s["rows"] = _host_words(rng, nq << case["nch"]).reshape(nq, -1)
        s["challenges"] = [int(x) for x in _host_words(rng, case["nch"])]
        s["queries"] = np.sort(rng.choice(4 << max(case["log"], 8), size=nq, replace=False)).tolist()
        s["alpha"] = int(_host_words(rng, 1)[0])
    elif op == "gf128":
        s["a"], s["b"] = (_words(gen, 4 * case["n"]).view(torch.int64).view(-1, 2) for _ in range(2))
    torch.cuda.synchronize()  # the inputs are there before the call
    return s


def _record_size(cfg):
    """An upper bound of a config's proof bytes (their number varies with the
    queries: each opening carries as many Merkle nodes as they need)."""
    dims = [cfg.initial_dims] + list(cfg.dims)
    rows = sum(QUERIES * (4 + 4 * n) + QUERIES * (m.bit_length() + 1) * 36 + 64 for m, n in dims)
    left = (cfg.dims[-1][0] << _log2(cfg.dims[-1][1])) >> cfg.ks[-1]
    return 256 + rows + 36 * len(dims) + 4 * left + 12 * (sum(cfg.ks) + 2 * len(dims))


def _log2(x):
    return x.bit_length() - 1


def _record(proof, out):
    """The proof's bytes in the caller's fixed-size record, as a program that
    stores or sends proofs keeps them."""
    b = proof.to_bytes()
    out[:len(b)] = np.frombuffer(b, dtype=np.uint8)
    out[len(b):] = 0
    return out


def run(s):
    op, ctx = s["op"], s["ctx"]
    if op == "prove":
        return _record(lg.prover(s["cfg"], s["poly"], ctx), s["record"])
    if op == "lockstep":
        return [_record(p, r) for p, r in zip(lg.prove_lockstep(s["cfg"], s["polys"], ctx), s["records"])]
    if op == "verify":
        # the outcome, and the commitment root that it stands for
        return lg.verifier(s["cfg"], s["proof"], ctx), np.frombuffer(s["proof"], np.uint8, 32, 16)
    if op == "commit":
        encoded, tree, root = lg.ligero_commit(s["poly"], s["log_m"], s["n"], ctx)
        return encoded, tree, np.frombuffer(root, dtype=np.uint8)
    if op == "encode":
        return lg.encode_cols(s["poly"], s["log_m"], s["n"], ctx)
    if op == "fft":
        lg.fft(s["data"], s["log"], ctx)
        return s["data"]
    if op == "ifft":
        lg.ifft(s["data"], s["log"], ctx)
        return s["data"]
    if op == "partial":
        return lg.partial_eval(s["evals"], s["rs"], ctx)
    if op == "eval013":
        return list(lg.eval_013_product(s["f"], s["g"], ctx))
    if op == "induce":
        basis, total = lg.induce_sumcheck_poly(s["log"], s["rows"], s["challenges"], s["queries"], s["alpha"], ctx)
        return basis, total
    return lg.gf128_mul(s["a"], s["b"], ctx)


def exact(case, seed):
    """Outputs are whole numbers and bytes, none of them rounded."""
    return None


def _fft_products(points):
    """Field products of an additive FFT: one a butterfly and stage."""
    return points // 2 * max(1, points.bit_length() - 1)


def _commit_work(log_m, n):
    """Bytes and field products of encoding n columns of 2^log_m and hashing the tree."""
    m = 1 << log_m
    return 4 * n * m + 16 * n * m + 32 * (8 * m - 1), n * m + 4 * n * _fft_products(m)


def _prove_work(case):
    """A proof reads its polynomial and writes some hundred KB; its products
    are those of the first commitment and the fold (the rest is a few percent)."""
    log, cols = case["log"], case["cols"]
    return 4 << log, _commit_work(log - cols, 1 << cols)[1] + (1 << log)


def work(case):
    """Bytes: inputs read once, outputs written once.  flops: field products."""
    op = case["op"]
    if op == "prove":
        b, p = _prove_work(case)
    elif op == "lockstep":
        b, p = (x * case["count"] for x in _prove_work(case))
    elif op == "verify":
        # the proof (148 rows and their siblings, and the later steps'), and
        # the first opening's induced basis polynomial
        b, p = QUERIES * ((4 << case["cols"]) + 32 * (case["log"] - 4)) * 2, QUERIES << (case["log"] - case["cols"])
    elif op == "commit":
        b, p = _commit_work(case["log_m"], case["n"])
    elif op == "encode":
        b, p = 20 * case["n"] << case["log_m"], _commit_work(case["log_m"], case["n"])[1]
    elif op in ("fft", "ifft"):
        b, p = 8 * case["batch"] << case["log"], case["batch"] * _fft_products(1 << case["log"])
    elif op == "partial":
        b, p = (4 << case["log"]) + (4 << (case["log"] - case["k"])), 1 << case["log"]
    elif op == "eval013":
        b, p = 8 << case["log"], 3 << (case["log"] - 1)
    elif op == "induce":
        b, p = (4 << case["log"]) + (4 * case["queries"] << case["nch"]), case["queries"] << case["log"]
    else:
        b, p = 48 * case["n"], case["n"]
    return {"bytes": b, "flops": p}
