"""A tensor-core pass of the FP64 form that gave up waiting is an error of the call that ran it,
whichever of its column chunks or products that was, and of no later call.

No wait runs out here: CS_B200_GIVE_UP=i has the library report the process's pass number i so, and a
process runs one scenario.  An apply makes two passes per chunk of 288 columns.
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
import sys
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
import test_gave_up_gpu
test_gave_up_gpu.SCENARIOS[sys.argv[2]]()
print("scenario ran")
"""


def cohort(n=400, m=900):
    d = synth.cohort(n, m, 5, missing=0.02, n_causal=20)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    return d, g, cs.createKinshipOperator(g), np.random.default_rng(1)


def gives_up(call):
    with pytest.raises(RuntimeError, match="gave up waiting"):
        call()


def wide_apply():
    _, _, op, rng = cohort()
    X = rng.standard_normal((400, 289))
    gives_up(lambda: op.apply(X))  # pass 0: rows of the first chunk
    assert np.isfinite(op.apply(X)).all()


def wide_half_pass():
    _, _, op, rng = cohort()
    V = rng.standard_normal((900, 289))
    gives_up(lambda: op.multiply_Z_v(V))
    assert np.isfinite(op.multiply_Z_v(V)).all()


def unreported():
    """A device-buffer call does not wait for the stream: its result is NaN.  The calls after it,
    of either form, succeed."""
    torch = pytest.importorskip("torch")
    _, _, op, rng = cohort()
    X = rng.standard_normal((400, 3))
    x = torch.tensor(X.T.copy(), device="cuda")
    y = torch.empty_like(x)
    op.apply_device(x.data_ptr(), 400, 3, y.data_ptr(), 400)
    torch.cuda.synchronize()
    assert bool(torch.isnan(y).all())
    assert np.isfinite(op.apply(X, precision="mixed")).all()
    op.apply_device(x.data_ptr(), 400, 3, y.data_ptr(), 400)
    assert np.isfinite(op.apply(X)).all() and bool(torch.isfinite(y).all())


def solve():
    _, _, op, rng = cohort()
    B = rng.standard_normal((400, 300))
    pcg = cs.MatrixFreePCG(op, 0.5, 0.5, precision="fp64")
    gives_up(lambda: pcg.solve(B))  # pass 4: the second product
    assert np.isfinite(pcg.solve(B)).all()


def exact_scan():
    d, g, _, _ = cohort()
    gives_up(lambda: cs.run_lmm_exact(g, d["y"], np.asfortranarray(np.ones((400, 1))), precision="fp64"))


def sketch():
    d, _, op, _ = cohort()
    eng = cs.LmmEngine()
    gives_up(lambda: eng.prepareLowRankMatrixFree(d["y"], np.asfortranarray(np.ones((400, 1))), op, rank=20,
                                                  precision="fp64"))


def multi_trait():
    d, _, op, rng = cohort()
    Y = np.asfortranarray(np.c_[d["y"], rng.standard_normal(400)])
    gives_up(lambda: cs.mv_stcg_solve(op, Y, np.ones((400, 1)), precision="fp64"))


SCENARIOS = {f.__name__: f for f in (wide_apply, wide_half_pass, unreported, solve, exact_scan, sketch,
                                     multi_trait)}


@pytest.mark.parametrize("name,which", [("wide_apply", 0), ("wide_apply", 1), ("wide_half_pass", 0),
                                        ("unreported", 0), ("unreported", 1), ("solve", 4),
                                        ("exact_scan", 0), ("sketch", 0), ("multi_trait", 2)])
def test_pass_that_gave_up(name, which):
    env = dict(os.environ, CS_B200_GIVE_UP=str(which))
    res = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, name], env=env, capture_output=True, text=True)
    assert res.returncode == 0 and "scenario ran" in res.stdout, res.stdout + res.stderr
