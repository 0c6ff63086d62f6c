"""FP64 kinship products on the int8 tensor cores (seven exact int8 digits per column).

Reference: the product in extended precision (numpy longdouble) of the operator's Z, so the
check resolves the FP64 result's own last bits.  Bound: a column's fixed-point error is 2^-55 of
its maximum per element, which over a sum of n terms gives about 2^-55.8 sqrt(n) max, that is
2^-54 of the result for normal columns; with the few FP64 roundings of the joins, the scalings and
the second pass the result stays within 2^-50 of its column's largest entry, and 2^-48 leaves a
factor of four.  Sizes sit at the edges of the 128-row tiles, 256-sample padding and K slices;
widths at the edges of the column tiles (1..4 digit-adjacent, 8-column steps, pairs, several
tiles, the 288-column chunk).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402

TOL = 2.0 ** -48


def problem(n, m, seed, missing=0.02, maf_lo=0.05):
    d = synth.cohort(n, m, seed, missing=missing, n_causal=5, maf_lo=maf_lo)
    ref = oracle.Bed(d["bed"][3:].reshape(m, -1), n)
    return cs.Genotypes.from_bed_bytes(d["bed"], n, m), ref


def exact_apply(ref, X, keep=None, variants=None):
    Z = ref.dense_z(keep, variants).astype(np.longdouble)
    return Z @ (Z.T @ X.astype(np.longdouble)) / Z.shape[1]


def rel(Y, E):
    return float((np.abs(Y - E).max(axis=0) / np.abs(E).max(axis=0)).max())


@pytest.mark.parametrize("n,m", [(127, 383), (128, 128), (129, 257), (256, 640), (511, 129), (300, 1300)])
@pytest.mark.parametrize("k", [1, 2, 4, 5, 8, 9, 17])
def test_tile_edges(n, m, k):
    g, ref = problem(n, m, n + m)
    op = cs.createKinshipOperator(g)
    X = np.random.default_rng(k).standard_normal((n, k))
    Y = op.apply(X)
    assert rel(Y, exact_apply(ref, X)) < TOL
    assert np.array_equal(op.apply(X), Y)


@pytest.mark.parametrize("k", [24, 25, 33, 48, 64, 65, 266, 288, 289])
def test_widths(k):
    g, ref = problem(300, 1000, 7, maf_lo=0.01)
    keep = np.sort(np.random.default_rng(1).choice(300, 271, replace=False)).astype(np.int32)
    variants = np.arange(0, 1000, 2, dtype=np.int32)
    op = cs.createKinshipOperator(g, keep, variants)
    X = np.random.default_rng(k).standard_normal((271, k))
    X[:, 0] = 1e3 + 1e-3 * X[:, 0]   # a mean far above the spread
    X[:, 1] = X[:, 1] > 0            # an indicator
    X[:, 2] *= 1e-200
    E = exact_apply(ref, X, keep, variants)
    Y = op.apply(X)
    assert rel(Y[:, 1:], E[:, 1:]) < TOL
    # K 1 is not zero where calls are missing, so the mean does not cancel out of the result
    assert rel(Y[:, :1], E[:, :1]) < TOL


def test_long_contractions():
    """Several K slices and int32 accumulators near their longest run."""
    for n, m in ((200, 70001), (9001, 300)):
        g, ref = problem(n, m, n)
        op = cs.createKinshipOperator(g)
        X = np.random.default_rng(n).standard_normal((n, 3))
        assert rel(op.apply(X), exact_apply(ref, X)) < TOL


def test_columns_outside_the_fixed_point_range():
    """Columns with a non-finite value, with elements spread over hundreds of binades, or at the
    ends of the exponent range run on the FP64 pipe; their neighbours and zero columns do not
    notice."""
    n, m = 400, 700
    g, ref = problem(n, m, 3)
    op = cs.createKinshipOperator(g)
    rng = np.random.default_rng(0)
    X = rng.standard_normal((n, 12))
    clean = op.apply(X)
    E = exact_apply(ref, X)
    X[5, 1] = np.nan
    X[5, 3] = np.inf
    X[:, 4] = 0.0
    X[:, 6] = rng.standard_normal(n) * 10.0 ** rng.uniform(-150, 150, n)
    X[:, 8] *= 1e-300
    X[0, 9] = 1e20
    Y = op.apply(X)
    same = [0, 2, 5, 7, 10, 11]
    assert np.array_equal(Y[:, same], clean[:, same])
    assert np.all(np.isnan(Y[:, 1])) and not np.any(np.isfinite(Y[:, 3]))
    assert np.all(Y[:, 4] == 0.0)
    for c in (6, 8, 9):
        assert rel(Y[:, c:c + 1], exact_apply(ref, X[:, c:c + 1])) < 1e-13, c
    assert rel(Y[:, same], E[:, same]) < TOL
    # samples whose call at SNP t is missing see only the small elements of column 9
    U = exact_apply(ref, X[:, 9:10])
    assert np.abs(Y[:, 9:10] - U).max() <= 1e-13 * np.abs(U).max()


def test_result_may_overwrite_its_input():
    torch = pytest.importorskip("torch")
    g, ref = problem(600, 900, 5)
    op = cs.createKinshipOperator(g)
    for k in (1, 3, 40):
        X = np.random.default_rng(k).standard_normal((600, k))
        X[3, 0] = 1e25  # this column runs on the FP64 pipe, from X again
        t = torch.tensor(X.T.copy(), device="cuda")
        op.apply_device(t.data_ptr(), 600, k, t.data_ptr(), 600)
        torch.cuda.synchronize()
        assert rel(t.cpu().numpy().T, exact_apply(ref, X)) < 1e-13


@pytest.mark.parametrize("k", [1, 3, 8, 20, 300])
def test_half_passes(k):
    """Z^T X and Z V over a selection with variants that vary in no sample (dropped from the packed
    view, zero rows of Z) and with a column outside the fixed-point range."""
    n, m = 700, 900
    d = synth.cohort(n, m, 17, missing=0.02, n_causal=5)
    rows = d["bed"][3:].reshape(m, -1)
    rows[[0, 5, 899]] = 0xFF  # every call 11
    d["bed"][3:] = rows.ravel()
    ref = oracle.Bed(rows, n)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    keep = np.sort(np.random.default_rng(1).choice(n, 601, replace=False)).astype(np.int32)
    variants = np.r_[np.arange(0, 450), [700, 899]].astype(np.int32)
    op = cs.createKinshipOperator(g, keep, variants)
    Z = ref.dense_z(keep, variants).astype(np.longdouble)
    rng = np.random.default_rng(k)
    X, V = rng.standard_normal((601, k)), rng.standard_normal((len(variants), k))
    U, Y = op.multiply_Zt_v(X), op.multiply_Z_v(V)
    assert np.all(U[[0, 5, 451]] == 0.0)
    assert rel(U, Z.T @ X) < TOL and rel(Y, Z @ V) < TOL
    X[7, 0] = V[7, 0] = 1e22
    assert rel(op.multiply_Zt_v(X), Z.T @ X) < 1e-13
    assert rel(op.multiply_Z_v(V), Z @ V) < 1e-13


def test_overlapping_blocks():
    """Output blocks that overlap the input other than in place give the same result."""
    torch = pytest.importorskip("torch")
    n, k = 800, 6
    g, ref = problem(n, 1200, 9)
    op = cs.createKinshipOperator(g)
    X = np.random.default_rng(0).standard_normal((n, k))
    buf = torch.empty(k * n + 3 * n, dtype=torch.float64, device="cuda")
    buf[: k * n] = torch.tensor(X.T.copy(), device="cuda").ravel()
    op.apply_device(buf.data_ptr(), n, k, buf.data_ptr() + 8 * 2 * n, n)
    torch.cuda.synchronize()
    Y = buf[2 * n: 2 * n + k * n].reshape(k, n).cpu().numpy().T
    assert rel(Y, exact_apply(ref, X)) < TOL
