"""The work that is timed: what a PLONK prover has this library do, call by call.

Every case goes through the Python front end (``ppfr``), as a user's program
calls it: polynomials are ``(n, 4)`` int64 tensors of canonical BLS12-381 Fr
elements in Montgomery form, uniformly random (blinded wires, challenges and
commitment scalars are), and the tables, commitment keys and plans that such a
program keeps between calls are made in ``prepare``.

Sizes: circuits of 2^8 .. 2^22 rows and their extended domains up to 2^24,
the range of the repository's benchmark and tests.
"""
import importlib
import math

import torch

ppfr = importlib.import_module("ppopp26-artifact_gb300").ppfr

MUL = 256  # 32-bit multiply instructions of one Fr multiplication (two halves of 8 x 8 product + reduction)
FQ_MUL = 576  # the same for the base field (12 limbs)


def listed():
    return [
        # a small circuit's transform: one call's latency is all that counts
        {"name": "ntt_2p12", "kind": "ntt", "lg": 12, "inverse": False},
        # evaluations back to coefficients at an ordinary circuit size
        {"name": "intt_2p18", "kind": "ntt", "lg": 18, "inverse": True},
        # the headline transform: a large circuit (or a 4x extended 2^22 domain)
        {"name": "ntt_2p24", "kind": "ntt", "lg": 24, "inverse": False},
        # coset extension of a wire polynomial held as coefficients
        {"name": "lde_coeffs_2p20_x4", "kind": "lde", "lg": 20, "lam": 2, "evals": False},
        # coset extension from evaluations to the 8x quotient domain
        {"name": "lde_evals_2p21_x8", "kind": "lde", "lg": 21, "lam": 3, "evals": True},
        # a polynomial that lives in page-locked host memory
        {"name": "ntt_host_2p22", "kind": "host", "lg": 22, "inverse": False},
        # the copy-constraint accumulator z of a 2^20-row circuit
        {"name": "gp_perm_2p20", "kind": "perm", "lg": 20},
        # the stand-alone operators on one ragged polynomial: running product,
        # opening value and opening quotient
        {"name": "scans_1000003", "kind": "scans", "n": 1000003},
        # quotient terms over an extended domain (permutation + gates)
        {"name": "quotient_2p20", "kind": "quotient", "n": 1 << 20},
        # a one-off commitment: variable-base multi-scalar multiplication
        {"name": "msm_200003", "kind": "msm", "n": 200003, "fixed": False},
        # commitments to the prover's own key, window tables kept in HBM
        {"name": "msm_fixed_2p20", "kind": "msm", "n": 1 << 20, "fixed": True},
        # many circuits' polynomials of mixed sizes queued as one plan
        {"name": "batch_32_mixed", "kind": "batch", "count": 32, "min_lg": 10, "max_lg": 18, "graph": False},
    ]


def _size(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "lde", "lde", "host", "perm", "scans", "scans", "quotient", "msm", "msm", "batch"])
    if kind == "ntt":
        return {"kind": kind, "lg": rng.randint(8, 24), "inverse": rng.random() < 0.5}
    if kind == "lde":
        lam = rng.randint(1, 3)
        return {"kind": kind, "lg": rng.randint(8, 24 - lam), "lam": lam, "evals": rng.random() < 0.5}
    if kind == "host":
        return {"kind": kind, "lg": rng.randint(10, 22), "inverse": rng.random() < 0.5}
    if kind == "perm":
        return {"kind": kind, "lg": rng.randint(8, 21)}
    if kind == "scans":
        return {"kind": kind, "n": _size(rng, 250, 1 << 22) | 1}
    if kind == "quotient":
        return {"kind": kind, "n": _size(rng, 1 << 10, 1 << 21)}
    if kind == "msm":
        return {"kind": kind, "n": _size(rng, 250, 1 << 18), "fixed": rng.random() < 0.5}
    lo = rng.randint(8, 12)
    return {"kind": kind, "count": rng.randint(6, 48), "min_lg": lo, "max_lg": rng.randint(lo + 1, 17),
            "graph": rng.random() < 0.5}


def _batch_jobs(case):
    """(kind, lg, lam) of every polynomial: two transforms for each extension,
    a grand product now and then, sizes cycling through the range."""
    jobs = []
    for i in range(case["count"]):
        lg = case["min_lg"] + (i * 5) % (case["max_lg"] - case["min_lg"] + 1)
        kind = (ppfr.JOB_NTT, ppfr.JOB_INTT, ppfr.JOB_LDE_COEFFS, ppfr.JOB_NTT, ppfr.JOB_INTT,
                ppfr.JOB_LDE_EVALS, ppfr.JOB_NTT, ppfr.JOB_GP)[i % 8]
        jobs.append((kind, lg, 2 if kind in (ppfr.JOB_LDE_COEFFS, ppfr.JOB_LDE_EVALS) else 0))
    return jobs


def _small_mont(k):
    """k in Montgomery form as a one-element tensor."""
    x = torch.zeros((1, 4), dtype=torch.int64, device="cuda")
    x[0, 0] = k
    return ppfr.to_mont(x)


def prepare(case, seed):
    made = [0]

    def rand(n):
        made[0] += 1
        return ppfr.random_fr(n, seed * 1000 + made[0])

    kind = case["kind"]
    s = {"kind": kind}
    if kind == "ntt":
        ppfr.prepare(case["lg"], case["inverse"])
        n = 1 << case["lg"]
        s |= {"x": rand(n), "out": ppfr.empty(n), "inverse": case["inverse"]}
    elif kind == "lde":
        if case["evals"]:
            ppfr.prepare(case["lg"], True)
        ppfr.prepare(case["lg"] + case["lam"])
        s |= {"x": rand(1 << case["lg"]), "out": ppfr.empty(1 << (case["lg"] + case["lam"])), "lam": case["lam"],
              "mode": ppfr.LDE_EVALS if case["evals"] else ppfr.LDE_COEFFS}
    elif kind == "host":
        ppfr.prepare(case["lg"], case["inverse"])
        n = 1 << case["lg"]
        x = ppfr.empty_pinned(n)
        x.copy_(rand(n))
        s |= {"x": x, "out": ppfr.empty_pinned(n), "inverse": case["inverse"]}
    elif kind == "perm":
        n = 1 << case["lg"]
        s |= {"w": [rand(n) for _ in range(3)], "sigma": [rand(n) for _ in range(3)], "params": rand(5),
              "out": ppfr.empty(n)}
    elif kind == "scans":
        s |= {"x": rand(case["n"]), "z": rand(1)}
    elif kind == "quotient":
        n = case["n"]
        gate_v = {name: rand(n) for name in ppfr.GATE_VECTORS}
        gate_s = {name: rand(1) for name in ppfr.GATE_SCALARS}
        for name, k in (("one", 1), ("two", 2), ("three", 3), ("four", 4), ("nine", 9), ("eighteen", 18),
                        ("eightyone", 81), ("eightythree", 83)):
            gate_s[name] = _small_mont(k)
        wires = [gate_v[name] for name in ("a_val", "b_val", "c_val", "d_val")]
        s |= {"gate_v": gate_v, "gate_s": gate_s, "gate_out": ppfr.empty(n), "perm_out": ppfr.empty(n),
              "perm": dict(x=rand(n), w=wires, z=rand(n), z_next=rand(n), sigma=[rand(n) for _ in range(4)],
                           mod=rand(n), l1=rand(n), alpha=rand(1), beta=rand(1), gamma=rand(1),
                           k=[rand(1) for _ in range(3)], one=gate_s["one"])}
    elif kind == "msm":
        points = ppfr.g1_mul_gen(rand(case["n"]))
        s |= {"scalars": rand(case["n"]), "out": torch.empty((3, 6), dtype=torch.int64, device="cuda")}
        s["key" if case["fixed"] else "points"] = ppfr.MsmBases(points) if case["fixed"] else points
    elif kind == "batch":
        jobs = []
        for job, lg, lam in _batch_jobs(case):
            jobs.append((job, rand(1 << lg), ppfr.empty(1 << (lg + lam)), lam))
        s |= {"plan": ppfr.Batch(jobs), "outs": [j[2] for j in jobs]}
        if case["graph"]:
            s["plan"].capture()
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["kind"]
    if kind == "ntt":
        return ppfr.ntt(s["x"], s["inverse"], out=s["out"])
    if kind == "lde":
        return ppfr.lde(s["x"], s["lam"], s["mode"], out=s["out"])
    if kind == "host":
        return ppfr.ntt_host(s["x"], s["inverse"], out=s["out"])
    if kind == "perm":
        return ppfr.gp_perm(s["w"], s["sigma"], s["params"], out=s["out"])
    if kind == "scans":
        # the running product and the quotient are made in place, of copies
        return (ppfr.gp_prefix_(s["x"].clone()), ppfr.evaluate(s["x"], s["z"]),
                ppfr.div_xplusc_(s["x"].clone(), s["z"]))
    if kind == "quotient":
        return (ppfr.quotient_permutation(**s["perm"], out=s["perm_out"]),
                ppfr.gate_constraint(s["gate_v"], s["gate_s"], 5, out=s["gate_out"]))
    if kind == "msm":
        if "key" in s:
            return s["key"].msm(s["scalars"], out=s["out"])
        return ppfr.msm_g1(s["points"], s["scalars"], out=s["out"])
    s["plan"].run()
    return s["outs"]


def _transform(n):
    return n // 2 * (n.bit_length() - 1)


def work(case):
    """Bytes read and written once, and 32-bit multiplications (as flops) of
    the operators' textbook counts."""
    kind = case["kind"]
    if kind in ("ntt", "host"):
        n = 1 << case["lg"]
        return {"bytes": 64 * n, "flops": MUL * (_transform(n) + (n if case["inverse"] else 0))}
    if kind == "lde":
        n, ext = 1 << case["lg"], 1 << case["lam"]
        mm = ext * _transform(n) + n + (_transform(n) + n if case["evals"] else 0)
        return {"bytes": 32 * n * (1 + ext), "flops": MUL * mm}
    if kind == "perm":
        n = 1 << case["lg"]
        return {"bytes": 7 * 32 * n, "flops": MUL * 16 * n}
    if kind == "scans":
        n = case["n"]
        return {"bytes": 5 * 32 * n, "flops": MUL * 3 * n}
    if kind == "quotient":
        n = case["n"]
        return {"bytes": 33 * 32 * n, "flops": MUL * (18 + 81) * n}
    if kind == "msm":
        # bucket method with signed 16-bit windows: one mixed addition (about
        # ten base-field multiplications) per scalar and window
        n = case["n"]
        return {"bytes": 128 * n, "flops": FQ_MUL * 10 * 16 * n}
    total = {"bytes": 0, "flops": 0}
    for job, lg, lam in _batch_jobs(case):
        n = 1 << lg
        if job == ppfr.JOB_GP:
            w = {"bytes": 64 * n, "flops": MUL * n}
        elif lam:
            w = work({"kind": "lde", "lg": lg, "lam": lam, "evals": job == ppfr.JOB_LDE_EVALS})
        else:
            w = work({"kind": "ntt", "lg": lg, "inverse": job == ppfr.JOB_INTT})
        total = {k: total[k] + w[k] for k in total}
    return total


def exact(case, seed):
    """Every output is a whole number (an element of a finite field or of a
    curve over one), so none has a value in 64-bit floating point."""
    return None
