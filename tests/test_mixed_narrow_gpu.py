"""The mixed passes of few columns on the four-K-block kernel: K slices of 2, 5, 9 and 20 K-blocks (a
packed tile holds four), column counts at the edges of its widths.

The rows pass has one arithmetic form, so that its result is compared bit for bit with the kernels
that keep A in shared memory (a process with CS_B200_TMEM_A=0).  The samples pass there has another
form (five operand sets instead of six): it is compared with the FP64 product, within the mixed
form's 1e-6 of a column's largest entry.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(2000, 10000), (5003, 20011), (9000, 20000), (20011, 20000)]
WIDTHS = [1, 3, 8, 9, 16, 17, 24, 25, 32, 33, 40, 48]

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import cosmicscanner_b200 as cs
sys.path.insert(0, sys.argv[1] + "/tests")
from test_mixed_narrow_gpu import problem, SHAPES, WIDTHS
out = {}
for n, m in SHAPES:
    op, X, V = problem(n, m)
    for k in WIDTHS:
        out["%d_%d" % (n, k)] = op.multiply_Zt_v(X[:, :k], "mixed")
np.savez(sys.argv[2], **out)
"""


def problem(n, m):
    rng = np.random.default_rng(n)
    bed = np.empty(3 + m * ((n + 3) // 4), np.uint8)
    bed[:3] = (0x6C, 0x1B, 0x01)
    bed[3:] = rng.integers(0, 256, bed.size - 3, dtype=np.uint8)  # a quarter of the calls missing
    op = cs.createKinshipOperator(cs.Genotypes.from_bed_bytes(bed, n, m))
    return op, rng.standard_normal((n, max(WIDTHS))), rng.standard_normal((m, max(WIDTHS)))


def test_narrow_passes(tmp_path):
    other = tmp_path / "shared.npz"
    env = dict(os.environ, CS_B200_TMEM_A="0", CS_B200_AUTOTUNE="0")
    res = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, str(other)], env=env,
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    want = np.load(other)
    for n, m in SHAPES:
        op, X, V = problem(n, m)
        E = op.multiply_Z_v(V)
        for k in WIDTHS:
            assert np.array_equal(op.multiply_Zt_v(X[:, :k], "mixed"), want["%d_%d" % (n, k)]), (n, k)
            Y = op.multiply_Z_v(V[:, :k], "mixed")
            err = (np.abs(Y - E[:, :k]).max(axis=0) / np.abs(E[:, :k]).max(axis=0)).max()
            assert err < 1e-6, (n, k, err)
