"""The FP64-pipe kernels behind the operator's products (device memory short, no sample-major copy, or
chosen by environment): the FP64 tests of the products again in processes that choose each family, and
output blocks that overlap the input.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FAMILIES = [("CS_B200_FP64_DMMA", "0"), ("CS_B200_FP64_DMMA", "1"), ("CS_B200_FP64_NARROW", "0")]


@pytest.mark.parametrize("name,value", FAMILIES)
def test_products_on(name, value):
    files = ["tests/test_%s_gpu.py" % f for f in ("edges", "kinship", "genotype_matrix")]
    res = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", *files], cwd=ROOT,
                         env=dict(os.environ, **{name: value}), capture_output=True, text=True)
    assert res.returncode == 0, res.stdout[-3000:] + res.stderr[-1000:]


def overlapping():
    """Z^T X and Z V of 1 and 5 columns whose output starts inside the input, with variants that vary in no
    sample (their rows of Z^T X are cleared): 1e-12 of a column's largest entry, FP64 sums of a thousand
    terms."""
    import torch

    from cosmicscanner_b200 import _abi

    d = synth.cohort(700, 1000, 17, missing=0.02, n_causal=5)
    rows = d["bed"][3:].reshape(1000, -1)
    rows[[0, 5, 899]] = 0xFF
    d["bed"][3:] = rows.ravel()
    g = cs.Genotypes.from_bed_bytes(d["bed"], 700, 1000)
    rng = np.random.default_rng(0)
    keep = np.sort(rng.choice(700, 601, replace=False)).astype(np.int32)
    variants = np.arange(0, 900, dtype=np.int32)
    Z = oracle.Bed(rows, 700).dense_z(keep, variants)
    op = cs.createKinshipOperator(g, keep, variants)
    n, m = 601, 900
    lib = _abi.lib()
    for k in (1, 5):
        X, V = rng.standard_normal((n, k)), rng.standard_normal((m, k))
        for call, src, rows_in, rows_out, want in ((lib.cs_genotype_multiply_zt, X, n, m, Z.T @ X),
                                                   (lib.cs_genotype_multiply_z, V, m, n, Z @ V)):
            for shift in (0, 3, 650):
                buf = torch.zeros(k * m + 1000, dtype=torch.float64, device="cuda")
                buf[: k * rows_in] = torch.tensor(src.T.copy(), device="cuda").ravel()
                torch.cuda.synchronize()
                cs._check(call(op._h, buf.data_ptr(), rows_in, k, buf.data_ptr() + 8 * shift, rows_out, 0, None))
                torch.cuda.synchronize()
                got = buf[shift: shift + k * rows_out].reshape(k, rows_out).cpu().numpy().T
                assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max(), (call.__name__, k, shift)


def test_overlapping_blocks_on_the_digits():
    pytest.importorskip("torch")
    overlapping()


@pytest.mark.parametrize("name,value", FAMILIES)
def test_overlapping_blocks_on(name, value):
    pytest.importorskip("torch")
    script = ("import sys; sys.path.insert(0, %r); sys.path.insert(0, %r); import test_fp64_pipe_gpu as t; "
              "t.overlapping(); print('compared')" % (ROOT, os.path.join(ROOT, "tests")))
    res = subprocess.run([sys.executable, "-c", script], env=dict(os.environ, **{name: value}),
                         capture_output=True, text=True)
    assert res.returncode == 0 and "compared" in res.stdout, res.stdout + res.stderr
