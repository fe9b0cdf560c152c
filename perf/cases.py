"""The measured workloads of the sumcheck prover.

Each case is one call, or one short sequence of calls, of the public Python
API (`effsc_gpu`) as a program that proves, verifies or folds makes it: the
prover, batch or server such a program keeps is made in `prepare`, the
transcript, the proof and the read-back of its results are in `run`.  Tables
are seeded uniform Goldilocks values, the distribution of committed or
randomly combined polynomials.  Every output is a field element or a vector
of them, in whole 64-bit words.
"""
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "efficient-sumcheck_gb300"))
import effsc_gpu as E  # noqa: E402

KINDS = {"ml": E.ML, "ip": E.IP}
HOOK = bytes(range(32))     # the 32 bytes a caller absorbs per round (config 3's hook)


def listed():
    return [
        # the smallest proof: a dozen rounds, all of it launch and transcript latency
        {"name": "ip_n12", "do": "proof", "kind": "ip", "order": "msb", "field": 3, "len": 1 << 12, "rounds": 12},
        # a base-field multilinear claim of the ordinary size (2^20 evaluations)
        {"name": "ml_n20_fp", "do": "proof", "kind": "ml", "order": "msb", "field": 1, "len": 1 << 20, "rounds": 20},
        # the headline: an inner product of two 2^26 tables, extension challenges
        {"name": "ip_n26", "do": "proof", "kind": "ip", "order": "msb", "field": 3, "len": 1 << 26, "rounds": 26},
        # the same relation for a caller that binds the low variable first
        {"name": "ip_lsb_n24", "do": "proof", "kind": "ip", "order": "lsb", "field": 3, "len": 1 << 24, "rounds": 24},
        # a zero-check eq * f * g, stopped after 16 rounds with a per-round hook; the folded tables go on to the next step
        {"name": "coef_eqfg_n24", "do": "coef", "vars": 24, "rounds": 16, "hook": True},
        # the same claim through the factored eq prover
        {"name": "eqf_n24", "do": "eqf", "vars": 24, "rounds": 16, "hook": True},
        # one GKR layer with 2^12 gates
        {"name": "gkr_k12", "do": "gkr", "k": 12},
        # the trait's own round loop, the transcript and hook on the host, tables of no power of two
        {"name": "rounds_ip_len1000003", "do": "rounds", "kind": "ip", "order": "msb", "field": 3, "len": 1000003,
         "rounds": 20},
        # a cohort of uneven proofs as one graph
        {"name": "batch_ip128", "do": "batch", "kind": "ip", "count": 128, "low": 10, "high": 22},
        # a burst of mixed requests with their tables in host memory
        {"name": "serve_48", "do": "serve", "count": 48, "low": 14, "high": 20},
        # the other direction: the verifier's replay of a cohort's proofs
        {"name": "verify_256", "do": "verify", "count": 256, "degree": 2, "low": 10, "high": 22},
        # folding 2^20 committed polynomials of degree 7
        {"name": "pg_fold_n20", "do": "fold", "levels": 20, "width": 8, "field": 1},
    ]


def draw(rng):
    do = rng.choice(("proof", "proof", "proof", "coef", "eqf", "gkr", "rounds", "batch", "serve", "verify", "fold"))
    if do in ("proof", "rounds"):
        kind, order = rng.choice(("ip", "ip", "ml")), rng.choice(("msb", "lsb"))
        v = rng.randint(10, 25 if do == "proof" else 20)
        n = 1 << v
        if order == "msb" and rng.random() < (0.2 if do == "proof" else 0.6):
            n = rng.randint((1 << (v - 1)) + 1, 1 << v)     # any length: the upper half is padded with zeros
        field = rng.choice((3, 3, 1))
        c = {"do": do, "kind": kind, "order": order, "field": field, "len": n,
             "rounds": v if rng.random() < 0.7 else rng.randint(max(4, v // 2), v)}
        if field == 3 and v <= 23 and rng.random() < 0.25:
            c["ext"] = True                                  # tables of extension elements
        return c
    if do in ("coef", "eqf"):
        v = rng.randint(12, 23)
        return {"do": do, "vars": v, "rounds": rng.randint(v // 2, v), "hook": rng.random() < 0.5}
    if do == "gkr":
        return {"do": do, "k": rng.randint(5, 11)}
    if do == "batch":
        low = rng.randint(8, 12)
        return {"do": do, "kind": rng.choice(("ip", "ml")), "count": int(2 ** rng.uniform(3, 7.5)), "low": low,
                "high": low + rng.randint(1, 9)}
    if do == "serve":
        low = rng.randint(12, 16)
        return {"do": do, "count": int(2 ** rng.uniform(2, 6)), "low": low, "high": low + rng.randint(1, 4)}
    if do == "verify":
        low = rng.randint(6, 16)
        return {"do": do, "count": int(2 ** rng.uniform(0, 10)), "degree": rng.choice((1, 2, 3)), "low": low,
                "high": low + rng.randint(0, 10)}
    return {"do": do, "levels": rng.randint(8, 20), "width": rng.randint(2, 12), "field": rng.choice((1, 3))}


def _words(gen, *shape):
    """Uniform canonical residues mod p = 2^64 - 2^32 + 1 as int64 words on the GPU."""
    lo = torch.randint(0, 1 << 32, shape, generator=gen, device="cuda", dtype=torch.int64)
    hi = torch.randint(0, 1 << 32, shape, generator=gen, device="cuda", dtype=torch.int64)
    x = (hi << 32) | lo
    return torch.where((hi == 0xFFFFFFFF) & (lo > 0), lo - 1, x)     # the words above p wrap


def _host(t):
    return t.cpu().numpy().view(np.uint64)


def _prover_class(kind, order):
    return {("ml", "msb"): E.MultilinearProver, ("ml", "lsb"): E.MultilinearProverLSB,
            ("ip", "msb"): E.InnerProductProver, ("ip", "lsb"): E.InnerProductProverLSB}[kind, order]


def _sizes(case):
    """The number of variables of each proof of a cohort: part of the case, uniform on low..high."""
    rng = random.Random("%d %d %d" % (case["count"], case["low"], case["high"]))
    return [rng.randint(case["low"], case["high"]) for _ in range(case["count"])]


def _serve_kind(i):
    return "ml" if i % 10 in (2, 5, 8) else "ip"       # 30 % multilinear


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    do = case["do"]
    s = dict(case, label=b"cases/%d" % seed)
    if do in ("proof", "rounds"):
        nc = 3 if case.get("ext") else 1
        count = 2 if case["kind"] == "ip" else 1
        s["tables"] = [_words(gen, nc, case["len"]) for _ in range(count)]      # component-major, resident on the GPU
        cls = _prover_class(case["kind"], case["order"])
        torch.cuda.synchronize()
        s["prover"] = cls.from_device([t.data_ptr() for t in s["tables"]], [case["len"]] * count, [nc] * count,
                                      field=case["field"])
    elif do == "coef":
        n = 1 << case["vars"]
        eq = torch.from_numpy(E.build_eq_table(_host(_words(gen, case["vars"], 3))).view(np.int64))
        s["tables"] = [eq.cuda().t().contiguous(), _words(gen, n), _words(gen, n)]
        torch.cuda.synchronize()
        s["prover"] = E.CoefficientProver.from_device([t.data_ptr() for t in s["tables"]], [n] * 3, [3, 1, 1])
    elif do == "eqf":
        s["prover"] = E.EqFactoredProver(_host(_words(gen, case["vars"], 3)), _host(_words(gen, 1 << case["vars"])))
    elif do == "gkr":
        n = 1 << case["k"]
        s["prover"] = E.GkrProver(_host(_words(gen, n * n)), _host(_words(gen, n * n)), _host(_words(gen, n)))
    elif do == "batch":
        nv = _sizes(case)
        count = 2 if case["kind"] == "ip" else 1
        seeds = [[E.table_seed(seed, count * i + j) for j in range(count)] for i in range(len(nv))]
        s["batch"] = E.Batch(KINDS[case["kind"]], nv, seeds=seeds)
    elif do == "serve":
        nv = _sizes(case)
        s["server"] = E.Server(64 << 30, max_active=64)
        s["requests"] = []
        for i, v in enumerate(nv):
            kind = _serve_kind(i)
            s["requests"].append((KINDS[kind], v, list(_host(_words(gen, 2 if kind == "ip" else 1, 1 << v)))))
    elif do == "verify":
        nv = _sizes(case)
        s["claims"] = _host(_words(gen, len(nv), 3))
        s["polys"] = [_host(_words(gen, v, case["degree"], 3)) for v in nv]
        s["transcripts"] = [E.Transcript.keccak(E.FP3, b"cases/%d/%d" % (seed, i)) for i in range(len(nv))]
    else:
        f, n = case["field"], 1 << case["levels"]
        s["polys"] = _words(gen, n, case["width"], f)
        ab = _host(_words(gen, case["levels"], 2, f))
        s["pairs"] = [(ab[i, 0], ab[i, 1]) for i in range(case["levels"])]
    return s


def _out(*arrays):
    return [np.ascontiguousarray(a).view(np.int64) for a in arrays]


def _proof(p):
    return _out(p.round_polys, p.challenges, p.final_value)


def run(s):
    do = s["do"]
    if do == "proof":
        pr = s["prover"]
        pr.reset()
        return _proof(pr.prove(s["rounds"], E.Transcript.keccak(s["field"], s["label"])))
    if do in ("coef", "eqf"):
        pr = s["prover"]
        pr.reset()
        proof = pr.prove(s["rounds"], E.Transcript.keccak(E.FP3, s["label"]), hook=HOOK if s["hook"] else b"")
        # what the caller's next step reads: the folded tables
        return _proof(proof) + _out(*[pr.table(i) for i in range(3)])
    if do == "gkr":
        pr = s["prover"]
        pr.reset()
        proof = pr.prove(2 * s["k"], E.Transcript.keccak(E.FP3, s["label"]))
        return _proof(proof) + _out(pr.claimed_w_values())
    if do == "rounds":
        pr = s["prover"]
        pr.reset()
        return _proof(E.sumcheck(pr, s["rounds"], E.Transcript.keccak(s["field"], s["label"]),
                                 lambda _round, t: t.absorb(HOOK)))
    if do == "batch":
        b = s["batch"]
        return _out(*b.prove_raw([E.Transcript.keccak(E.FP3, s["label"] + b"/%d" % i) for i in range(len(b))]))
    if do == "serve":
        srv = s["server"]
        ids = [srv.submit(kind, v, E.Transcript.keccak(E.FP3, s["label"] + b"/%d" % i), tables=tables)
               for i, (kind, v, tables) in enumerate(s["requests"])]
        got = srv.drain()
        proofs = [got[i][0] for i in ids]
        return _out(np.concatenate([p.round_polys.reshape(-1) for p in proofs]),
                    np.concatenate([p.challenges.reshape(-1) for p in proofs]),
                    np.stack([p.final_value for p in proofs]))
    if do == "verify":
        fin, ch = E.sumcheck_verify_batch(s["claims"], s["degree"], s["polys"], s["transcripts"], hook=HOOK)
        return _out(fin, np.concatenate(ch))
    return _out(E.protogalaxy_fold_raw(s["pairs"], s["polys"].data_ptr(), 1 << s["levels"], s["width"],
                                       field=s["field"]))


def exact(case, seed):
    """Every output is an element of the field, in whole words: the values are
    exact or wrong, and compared word for word."""
    return None


def work(case):
    """The input words, read once each, and the words of the proof."""
    do = case["do"]
    if do in ("proof", "rounds"):
        tables, d = (2, 2) if case["kind"] == "ip" else (1, 1)
        words = tables * case["len"] * (3 if case.get("ext") else 1) + (case["rounds"] * (d + 1) + 1) * case["field"]
    elif do == "coef":
        words = 5 * (1 << case["vars"]) + 12 * case["rounds"] + 9 * (1 << (case["vars"] - case["rounds"]))
    elif do == "eqf":
        words = (1 << case["vars"]) + 9 * case["rounds"] + 3 * (1 << (case["vars"] - case["rounds"]))
    elif do == "gkr":
        words = 2 * (1 << (2 * case["k"])) + (1 << case["k"]) + 18 * case["k"]
    elif do in ("batch", "serve"):
        words = 0
        for i, v in enumerate(_sizes(case)):
            two = _serve_kind(i) == "ip" if do == "serve" else case["kind"] == "ip"
            words += ((2 if two else 1) << v) + v * (9 if two else 6) + 3
    elif do == "verify":
        words = sum(_sizes(case)) * (3 * case["degree"] + 3) + 6 * case["count"]
    else:
        words = (1 << case["levels"]) * case["width"] * case["field"]
    return {"bytes": 8.0 * words, "flops": 0.0}
