"""The mixed form's operand kernels at the edges of their tiles (16 rows a thread, 64 a tile, 256 of
padding) and on both sides of the row count up to which one block holds a column.

Bound: a quantised element is off by at most max|x - mean| / (2 127 254^2) = 3.1e-8 of the maximum
(three digits), and standardised genotypes have mean square 1, so that a product over n rows is off
by about 3.1e-8 / sqrt(3) sqrt(n) max; sixteen standard deviations of that hold for every entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402


@pytest.mark.parametrize("n", [3, 63, 64, 65, 255, 256, 257, 511, 513, 8191, 8192, 8193, 8449])
@pytest.mark.parametrize("k", [1, 3, 17, 40])
def test_rows_operand(n, k):
    m = 150
    d = synth.cohort(n, m, n, missing=0.02, n_causal=5, maf_lo=0.2)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    op = cs.createKinshipOperator(g)
    Z = oracle.Bed(d["bed"][3:].reshape(m, -1), n).dense_z(None, None)
    X = np.random.default_rng(k).standard_normal((n, k)) + 10.0 * np.arange(k)
    E = Z.T.astype(np.longdouble) @ X
    spread = np.abs(X - X.mean(axis=0)).max(axis=0)
    scale = np.sqrt((Z * Z).sum(axis=0))[:, None]  # sqrt(n) for complete, common variants
    tol = 16 * 3.1e-8 / np.sqrt(3) * spread * scale + 1e-12 * np.abs(E).max()
    U = op.multiply_Zt_v(X, "mixed")
    assert (np.abs(U - E) <= tol).all()
    # single precision: the same digits from the same values
    X32 = torch.from_numpy(X.T.astype(np.float32)).cuda()
    X64, Y32 = X32.double(), torch.empty_like(X32)
    Y64 = torch.empty_like(X64)
    op.apply_device_f32(X32.data_ptr(), n, k, Y32.data_ptr(), n, "mixed")
    op.apply_device(X64.data_ptr(), n, k, Y64.data_ptr(), n, "mixed")
    torch.cuda.synchronize()
    assert torch.equal(Y32, Y64.float())
