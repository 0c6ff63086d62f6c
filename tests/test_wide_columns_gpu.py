"""FP64 products of columns outside the fixed-point range, which the reduction kernels sum directly:
groups of four columns, tables of 64, 256 or 1024 SNP rows and of 256 SNPs, tiles of 32 samples.

Reference: the product in extended precision.  Plain FP64 sums of K terms are off by about
2^-53 sqrt(K) of the sum of magnitudes, 2^-45 for the few thousand terms here and the cancellation
between them; 1e-13 of a column's largest entry is asked.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")

TOL = 1e-13


def problem(n, m):
    d = synth.cohort(n, m, n + m, missing=0.03, n_causal=3)
    ref = oracle.Bed(d["bed"][3:].reshape(m, -1), n)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    return cs.createKinshipOperator(g), ref.dense_z(None, None).astype(np.longdouble)


def columns(rng, n, k, wide):
    X = rng.standard_normal((n, k))
    X[:, wide] *= 10.0 ** rng.uniform(-120, 120, (n, len(wide)))
    return X


def rel(Y, E):
    return float((np.abs(Y - E).max(axis=0) / np.abs(E).max(axis=0)).max())


# the last two take tables of 256 and 1024 rows
@pytest.mark.parametrize("n,m,k", [(31, 63, 1), (33, 65, 5), (63, 255, 33), (65, 257, 4), (129, 300, 160),
                                   (97, 1100, 160), (2500, 64, 3), (70, 5000, 2)])
def test_every_column_or_some(n, m, k):
    op, Z = problem(n, m)
    rng = np.random.default_rng(k)
    plain = rng.standard_normal((n, k))
    clean, clean_u = op.apply(plain), op.multiply_Zt_v(plain)
    for wide in (np.arange(k), np.arange(0, k, 3), np.array([k - 1])):
        X = columns(rng, n, k, wide)
        rest = np.setdiff1d(np.arange(k), wide)
        X[:, rest] = plain[:, rest]
        U = Z.T @ X.astype(np.longdouble)
        Y, u = op.apply(X), op.multiply_Zt_v(X)
        assert rel(Y, Z @ U / m) < TOL and rel(u, U) < TOL
        assert np.array_equal(Y[:, rest], clean[:, rest]) and np.array_equal(u[:, rest], clean_u[:, rest])
        V = columns(rng, m, k, wide)
        assert rel(op.multiply_Z_v(V), Z @ V.astype(np.longdouble)) < TOL


def test_inside_a_solver():
    """The solver's blocks are row-major; a right-hand side with one huge entry keeps its neighbours."""
    n, m = 300, 700
    op, Z = problem(n, m)
    rng = np.random.default_rng(0)
    B = rng.standard_normal((n, 6))
    B[3, 2] = 1e9
    x = cs.MatrixFreePCG(op, 0.6, 0.4, precision="fp64").solve(B, tol=1e-11, relative=True)
    V = 0.6 * (Z @ Z.T).astype(np.float64) / m + 0.4 * np.eye(n)
    assert (np.linalg.norm(V @ x - B, axis=0) < 1e-10 * np.linalg.norm(B, axis=0)).all()
