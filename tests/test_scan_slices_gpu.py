"""FP64 scans on the int8 digits against the same scans on the FP64 pipe (a process with
CS_B200_FP64_DMMA=1): a cohort in file order, one of selected and permuted samples, a window of
SNPs, and the exact scan.

Both are FP64 products; in the low-rank route the basis moves by the products' last bits times the
inverse gaps of the spectrum (below 1e6 here), 2^-48 1e6 = 4e-9 of a standard error; 1e-7 is asked.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
from test_scan_slices_gpu import scans
np.savez(sys.argv[2], **scans())
"""


def scans():
    n, m = 803, 1201
    d = synth.cohort(n, m, 5, missing=0.03, n_causal=20, maf_lo=0.02)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    rng = np.random.default_rng(2)
    out = {}
    for name, keep in (("all", np.arange(n)), ("some", rng.permutation(n)[:611])):
        keep = keep.astype(np.int32)
        y = d["y"][keep]
        X = np.asfortranarray(np.c_[np.ones(len(keep)), rng.standard_normal(len(keep))])
        op = cs.createKinshipOperator(g, keep, np.arange(m, dtype=np.int32))
        eng = cs.LmmEngine()
        eng.prepareLowRankMatrixFree(y, X, op, rank=40, precision="fp64")
        for part, r in (("scan", eng.scan(g, keep)), ("window", eng.scan_window(g, keep, 100, 777))):
            for key in ("beta", "se", "tested", "freq"):
                out["%s_%s_%s" % (name, part, key)] = r[key]
    r, _ = cs.run_lmm_exact(g, d["y"], np.asfortranarray(np.ones((n, 1))), precision="fp64")
    for key in ("beta", "se", "tested", "freq"):
        out["exact_scan_" + key] = r[key]
    return out


def test_fp64_scans(tmp_path):
    other = tmp_path / "pipe.npz"
    env = dict(os.environ, CS_B200_FP64_DMMA="1")
    res = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, str(other)], env=env,
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    want, got = np.load(other), scans()
    for key in want.files:
        if key.endswith("tested") or key.endswith("freq"):
            assert np.array_equal(got[key], want[key]), key
    for name in ("all_scan", "all_window", "some_scan", "some_window", "exact_scan"):
        t, se = want[name + "_tested"], want[name + "_se"]
        assert t.sum() > 100
        for key in ("_beta", "_se"):
            assert (np.abs(got[name + key] - want[name + key])[t] <= 1e-7 * se[t]).all(), (name, key)
