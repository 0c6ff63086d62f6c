"""The calls that programs on this framework spend their time in, at the sizes they make them.

The kinds of call, each through the package's public entry points:

* ``apply``    K X on device buffers (``KinshipOperator.apply_device`` / ``apply_device_f32``): one
               vector inside a CG step, a block of probes, a randomized-SVD sketch;
* ``half``     the GenotypeMatrix half-passes Z^T X and Z V on host arrays;
* ``pcg``      block conjugate gradients on (sigma2_g K + sigma2_e I) X = B;
* ``lowrank``  the whole low-rank REML null model and scan on resident genotypes;
* ``aireml``   the matrix-free AI-REML (CG solves, Hutchinson probes, Lanczos log-determinant);
* ``open``     .bed bytes in host memory to a resident matrix, its statistics and an operator over
               a cohort and a set of variants.

Genotypes are Hardy-Weinberg draws with minor allele frequencies U(maf, 0.5) and missing calls at
random, as the package's synthetic cohorts have them; right-hand sides are N(0, 1) as probes,
sketches and residuals are.
"""
import numpy as np
import torch

import cosmicscanner_b200 as cs

COVARIATES = 3  # intercept, N(0, 1), Bernoulli(0.5)


def listed():
    return [
        # one CG step's product on the small single-trait configuration: a call of microseconds,
        # of which a solver makes thousands
        {"name": "vector_small", "kind": "apply", "n": 2000, "m": 10000, "k": 1,
         "precision": "fp64", "f32": False, "subset": False, "missing": 0.01, "maf": 0.05},
        # the same product on the headline cohort
        {"name": "vector", "kind": "apply", "n": 50000, "m": 100000, "k": 1,
         "precision": "fp64", "f32": False, "subset": False, "missing": 0.02, "maf": 0.05},
        # an AI-REML block on the headline cohort: y, 3 covariates and 30 probes
        {"name": "probes", "kind": "apply", "n": 50000, "m": 100000, "k": 34,
         "precision": "mixed", "f32": False, "subset": False, "missing": 0.02, "maf": 0.05},
        # the sketch of the low-rank null model (rank 256 + 10) on the headline cohort: the
        # largest call, and most of the time of a whole job
        {"name": "sketch", "kind": "apply", "n": 50000, "m": 100000, "k": 266,
         "precision": "mixed", "f32": False, "subset": False, "missing": 0.02, "maf": 0.05},
        # the sketch in the plain FP64 form, the default precision, over a cohort's subset with
        # ragged sizes and rarer variants
        {"name": "sketch_fp64", "kind": "apply", "n": 20011, "m": 30007, "k": 266,
         "precision": "fp64", "f32": False, "subset": True, "missing": 0.01, "maf": 0.01},
        # a caller that keeps its vectors in single precision, a block of middle width
        {"name": "block_f32", "kind": "apply", "n": 31001, "m": 52003, "k": 96,
         "precision": "mixed", "f32": True, "subset": False, "missing": 0.02, "maf": 0.05},
        # scores and effects of a few traits: both half-passes on host arrays, FP64
        {"name": "half_passes", "kind": "half", "n": 20011, "m": 30007, "k": 8,
         "precision": "fp64", "subset": True, "missing": 0.01, "maf": 0.01},
        # a mixed-model solve for one phenotype, the reference's MatrixFreePCG call
        {"name": "pcg_one", "kind": "pcg", "n": 5003, "m": 20011, "k": 1, "precision": "fp64",
         "tol": 1e-8, "missing": 0.01, "maf": 0.05},
        # a block solve as AI-REML makes them
        {"name": "pcg_block", "kind": "pcg", "n": 20000, "m": 40000, "k": 34,
         "precision": "mixed", "tol": 1e-6, "missing": 0.02, "maf": 0.05},
        # the headline job: null model and scan of every SNP
        {"name": "lowrank_job", "kind": "lowrank", "n": 50000, "m": 100000, "rank": 256,
         "missing": 0.02, "maf": 0.05},
        # AI-REML iterations on the small single-trait configuration
        {"name": "aireml_small", "kind": "aireml", "n": 2000, "m": 10000, "probes": 30,
         "iters": 8, "missing": 0.01, "maf": 0.05},
        # a cohort made resident, with an operator over a subset of it
        {"name": "open_cohort", "kind": "open", "n": 20011, "m": 30007, "missing": 0.01,
         "maf": 0.01},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    """Sizes over the logarithm of 1,500..50,000 samples and 4,000..100,000 SNPs, odd ones
    included; widths over 1..266."""
    kind = rng.choice(["apply", "apply", "apply", "apply", "half", "pcg", "lowrank", "aireml", "open"])
    c = {"kind": kind, "n": _log_int(rng, 1500, 50000), "m": _log_int(rng, 4000, 100000),
         "missing": round(rng.uniform(0.002, 0.03), 4), "maf": rng.choice([0.01, 0.05])}
    if kind == "apply":
        c["k"] = _log_int(rng, 1, 266)
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["f32"] = c["precision"] == "mixed" and rng.random() < 0.25
        c["subset"] = rng.random() < 0.3
        if c["precision"] == "fp64" and c["k"] > 4:
            c["n"], c["m"] = min(c["n"], 20011), min(c["m"], 30007)
    elif kind == "half":
        c.update(n=min(c["n"], 20011), m=min(c["m"], 30007), k=rng.randint(1, 16),
                 precision=rng.choice(["fp64", "mixed"]), subset=rng.random() < 0.5)
    elif kind == "pcg":
        # exact() factorises an n x n matrix
        c.update(n=min(c["n"], 12000), m=min(c["m"], 40000), k=_log_int(rng, 1, 40),
                 precision=rng.choice(["fp64", "mixed"]))
        c["tol"] = 1e-8 if c["precision"] == "fp64" else 1e-6
    elif kind == "lowrank":
        c["rank"] = rng.randint(40, 256)
    elif kind == "aireml":
        c.update(n=min(c["n"], 6000), m=min(c["m"], 20000), probes=rng.randint(15, 40),
                 iters=rng.randint(4, 8))
    else:
        c.update(n=min(c["n"], 20011), m=min(c["m"], 30007))
    return c


# ---------------------------------------------------------------- inputs

def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + stream)


def _codes(case, seed):
    """PLINK 2-bit codes (00: two A1, 01: missing, 10: one, 11: none), SNP-major, in row blocks."""
    n, m, miss = case["n"], case["m"], case["missing"]
    gen = _generator(seed, 1)
    maf = torch.rand(m, 1, generator=gen, device="cuda") * (0.5 - case["maf"]) + case["maf"]
    two = miss + (1 - miss) * maf * maf
    one = two + (1 - miss) * 2 * maf * (1 - maf)
    n4 = 4 * ((n + 3) // 4)
    step = max(1, (1 << 28) // n4)
    for r in range(0, m, step):
        u = torch.rand(min(step, m - r), n4, generator=gen, device="cuda")
        code = (u < miss).to(torch.uint8)
        code += 3
        code -= (u < one[r:r + step]).to(torch.uint8)
        code -= 2 * (u < two[r:r + step]).to(torch.uint8)
        del u
        yield r, code


def _bed(case, seed):
    """A .bed file's bytes in host memory."""
    n, m = case["n"], case["m"]
    rows = torch.empty(m, (n + 3) // 4, dtype=torch.uint8, device="cuda")
    for r, code in _codes(case, seed):
        q = code.view(code.shape[0], -1, 4)
        rows[r:r + code.shape[0]] = q[..., 0] | (q[..., 1] << 2) | (q[..., 2] << 4) | (q[..., 3] << 6)
    bed = np.empty(3 + rows.numel(), dtype=np.uint8)
    bed[:3] = (0x6C, 0x1B, 0x01)
    torch.from_numpy(bed)[3:].copy_(rows.view(-1))
    return bed


def _selection(case, seed):
    """Nine tenths of the samples and of the variants, in order."""
    rng = np.random.default_rng([int(seed), 2])
    keep = np.sort(rng.choice(case["n"], case["n"] * 9 // 10, replace=False)).astype(np.int32)
    variants = np.sort(rng.choice(case["m"], case["m"] * 9 // 10, replace=False)).astype(np.int32)
    return keep, variants


def _used(case):
    """Samples and variants of the operator."""
    n, m = case["n"], case["m"]
    return (n * 9 // 10, m * 9 // 10) if case.get("subset") or case["kind"] == "open" else (n, m)


def _operator(case, seed):
    g = cs.Genotypes.from_bed_bytes(_bed(case, seed), case["n"], case["m"])
    return cs.KinshipOperator(g, *(_selection(case, seed) if case.get("subset") else (None, None)))


def _normal(case, seed, stream, *shape):
    return torch.randn(*shape, generator=_generator(seed, stream), device="cuda", dtype=torch.float64)


def _phenotype(case, seed):
    """y and X as a user holds them: host arrays, h2 about 0.4 from the first 200 SNPs."""
    n = case["n"]
    effects = _normal(case, seed, 5, 200)
    _, code = next(iter(_codes(case, seed)))
    dosage = torch.tensor([2.0, 0.0, 1.0, 0.0], device="cuda", dtype=torch.float64)[code[:200, :n].long()]
    g = effects @ (dosage - dosage.mean(1, keepdim=True))
    g = (g - g.mean()) / g.std() * 0.4 ** 0.5
    rng = np.random.default_rng([int(seed), 3])
    X = np.column_stack([np.ones(n), rng.standard_normal(n), rng.integers(0, 2, n)])
    y = g.cpu().numpy() + 0.5 * X[:, 1] + rng.standard_normal(n) * 0.6 ** 0.5
    return y, X


def prepare(case, seed):
    kind = case["kind"]
    if kind == "open":
        keep, variants = _selection(case, seed)
        return {"case": case, "bed": _bed(case, seed), "keep": keep, "variants": variants}
    if kind == "lowrank":
        y, X = _phenotype(case, seed)
        g = cs.Genotypes.from_bed_bytes(_bed(case, seed), case["n"], case["m"])
        return {"case": case, "g": g, "y": y, "X": X}
    op = _operator(case, seed)
    n, m = _used(case)
    if kind == "apply":
        X = _normal(case, seed, 3, case["k"], n)  # column-major n x k
        if case["f32"]:
            X = X.float()
        return {"case": case, "op": op, "X": X, "Y": torch.empty_like(X)}
    if kind == "half":
        X = _normal(case, seed, 3, case["k"], n).cpu().numpy().T
        V = _normal(case, seed, 4, case["k"], m).cpu().numpy().T
        return {"case": case, "op": op, "X": X, "V": V}
    if kind == "pcg":
        B = _normal(case, seed, 3, case["k"], n)
        return {"case": case, "op": op, "B": B, "X": torch.empty_like(B)}
    y, X = _phenotype(case, seed)
    return {"case": case, "op": op, "y": y, "X": X}


# ---------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "apply":
        X, Y = state["X"], state["Y"]
        n = X.shape[1]
        call = state["op"].apply_device_f32 if case["f32"] else state["op"].apply_device
        call(X.data_ptr(), n, case["k"], Y.data_ptr(), n, case["precision"], stream)
        return Y
    if kind == "half":
        return {"zt": state["op"].multiply_Zt_v(state["X"], case["precision"]),
                "z": state["op"].multiply_Z_v(state["V"], case["precision"])}
    if kind == "pcg":
        B, X = state["B"], state["X"]
        n = B.shape[1]
        cs.pcg_solve_device(state["op"], B.data_ptr(), n, case["k"], X.data_ptr(), n, 0.4, 0.6,
                            tol=case["tol"], relative=True, precision=case["precision"],
                            stream=stream)
        return X
    if kind == "lowrank":
        out, diag = cs.run_lmm_matrix_free(None, case["n"], case["m"], state["y"], state["X"],
                                           rank=case["rank"], precision="mixed",
                                           genotypes=state["g"])
        return {**{k: out[k] for k in ("beta", "se", "p", "log10p", "freq", "tested")},
                "sigma2": np.array([diag["sigma2_g"], diag["sigma2_e"], diag["trace"]])}
    if kind == "aireml":
        vce = cs.StcgVce()
        r = vce.solve(state["op"], state["y"], state["X"], max_iter=case["iters"],
                      mc_samples=case["probes"], precision="mixed")
        beta, a, _ = vce.solution()
        vce.close()
        return {"sigma2": np.array([r["sigma2_g"], r["sigma2_e"]]), "logl": r["logl"],
                "beta": beta, "a": a}
    g = cs.Genotypes.from_bed_bytes(state["bed"], case["n"], case["m"])
    op = cs.KinshipOperator(g, state["keep"], state["variants"])
    out = {**g.stats(), "trace": op.trace(), "diagonal": op.getDiagonal()}
    op.close()
    g.close()
    return out


def work(case):
    n, m = _used(case)
    kind = case["kind"]
    packed = m * ((n + 3) // 4)
    if kind == "apply":
        return {"bytes": packed + (8 if case["f32"] else 16) * n * case["k"],
                "flops": 4 * n * m * case["k"]}
    if kind == "half":
        return {"bytes": packed + 16 * (n + m) * case["k"], "flops": 4 * n * m * case["k"]}
    if kind == "pcg":  # about fifteen steps to these tolerances at this ratio of variances
        return {"bytes": packed + 16 * n * case["k"], "flops": 15 * 4 * n * m * case["k"]}
    if kind == "lowrank":  # four sketch products
        return {"bytes": packed + 8 * n * 4 + 44 * m, "flops": 4 * 4 * n * m * (case["rank"] + 10)}
    if kind == "aireml":  # per iteration about fifteen steps of the probe block
        return {"bytes": packed + 8 * n * 5,
                "flops": case["iters"] * 15 * 4 * n * m * (case["probes"] + 1 + COVARIATES)}
    return {"bytes": case["m"] * (2 * ((case["n"] + 3) // 4) + 28) + 8 * n, "flops": 0}


# ---------------------------------------------------------------- the same in 64 bits

def _standardised(case, seed):
    """Blocks of Z^T (variants x samples) of the operator's selection, (position, block, mean,
    1/sd, count, sum) with the statistics over all samples."""
    n = case["n"]
    keep = None
    pick = None
    if case.get("subset") or case["kind"] == "open":
        keep, variants = (torch.as_tensor(v, device="cuda").long() for v in _selection(case, seed))
        pick = torch.zeros(case["m"], dtype=torch.bool, device="cuda")
        pick[variants] = True
    dosage = torch.tensor([2.0, 0.0, 1.0, 0.0], device="cuda", dtype=torch.float64)
    for r, code in _codes(case, seed):
        for q in range(0, code.shape[0], 2048):
            c = code[q:q + 2048, :n].long()
            seen = c != 1
            x = dosage[c]
            count = seen.sum(1)
            total = x.sum(1)
            mean = torch.where(count > 0, total / count.clamp(min=1), torch.zeros_like(total))
            p = mean / 2
            var = 2 * p * (1 - p)
            scale = torch.where(var < 1e-9, torch.zeros_like(var), 1 / torch.sqrt(var))
            z = (x - mean[:, None]) * seen * scale[:, None]
            used = z
            if keep is not None:
                used = z[pick[r + q:r + q + c.shape[0]]][:, keep]
            yield used, mean, scale, count, total


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lowrank", "aireml"):
        return None  # random sketches and probes: no value without the package's own streams
    n, m = _used(case)
    if kind == "apply":
        X = _normal(case, seed, 3, case["k"], n)
        if case["f32"]:
            X = X.float().double()
        Y = torch.zeros_like(X)
        for z, *_ in _standardised(case, seed):
            Y += (X @ z.T) @ z
        return Y / m
    if kind == "half":
        X = _normal(case, seed, 3, case["k"], n)
        V = _normal(case, seed, 4, case["k"], m)
        zt, z_v, at = [], torch.zeros_like(X), 0
        for z, *_ in _standardised(case, seed):
            zt.append(X @ z.T)
            z_v += V[:, at:at + z.shape[0]] @ z
            at += z.shape[0]
        return {"zt": torch.cat(zt, 1).T.cpu().numpy(), "z": z_v.T.cpu().numpy()}
    if kind == "pcg":
        A = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        for z, *_ in _standardised(case, seed):
            A.addmm_(z.T, z)
        A *= 0.4 / m
        A.diagonal().add_(0.6)
        B = _normal(case, seed, 3, case["k"], n)
        return torch.cholesky_solve(B.T, torch.linalg.cholesky(A)).T
    parts = [[], [], [], []]
    diagonal = torch.zeros(n, device="cuda", dtype=torch.float64)
    for z, *stats in _standardised(case, seed):
        diagonal += (z * z).sum(0)
        for p, s in zip(parts, stats):
            p.append(s)
    mean, scale, count, total = (torch.cat(p).cpu().numpy() for p in parts)
    diagonal /= m
    return {"mean": mean, "inv_std": scale, "count": count.astype(np.int32), "sum": total,
            "trace": float(diagonal.sum()), "diagonal": diagonal.cpu().numpy()}
