"""Cohorts of selected samples and variants, and the sample-major copy: code movement only, so the
reference is the same code moved by numpy and the products agree to FP64 rounding.

Sizes sit at the edges of what a block of the repacking kernel takes: rows up to 14,080 bytes (eight
rows a block), up to 56,320 bytes (four) and longer ones; SNP counts that leave the last block part
full; keep lists that are sorted, permuted and shorter than a word.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402


def problem(n, m, seed):
    d = synth.cohort(n, m, seed, missing=0.05, n_causal=2, maf_lo=0.05)
    ref = oracle.Bed(d["bed"][3:].reshape(m, -1), n)
    return cs.Genotypes.from_bed_bytes(d["bed"], n, m), ref


@pytest.mark.parametrize("n,m,n_keep", [
    (61, 17, 3), (130, 8, 64), (1025, 9, 700), (56320, 11, 40001), (56577, 11, 56000),
    (225280, 5, 1000), (225537, 5, 100001)])
@pytest.mark.parametrize("order", ["sorted", "permuted"])
def test_selected_samples_and_variants(n, m, n_keep, order):
    g, ref = problem(n, m, n + m)
    rng = np.random.default_rng(n_keep)
    keep = rng.choice(n, n_keep, replace=False).astype(np.int32)
    if order == "sorted":
        keep = np.sort(keep)
    variants = np.arange(m - 1, -1, -2, dtype=np.int32)
    op = cs.createKinshipOperator(g, keep, variants)
    Z = ref.dense_z(keep, variants)
    X = rng.standard_normal((n_keep, 2))
    E = Z @ (Z.T @ X) / Z.shape[1]
    # FP64 sums of n terms in two orders: n^0.5 2^-53 of the column's largest entry, times 64
    tol = 64 * np.sqrt(n_keep) * 2.0 ** -53
    Y = op.apply(X)
    assert (np.abs(Y - E).max(axis=0) <= tol * np.abs(E).max(axis=0)).all()


@pytest.mark.parametrize("n,m", [(3, 2), (255, 257), (256, 256), (257, 1023), (1000, 511)])
def test_sample_major_copy(n, m):
    """The samples pass reads the transposed codes: with Z^T X known, Z V pins each of them."""
    g, ref = problem(n, m, n * m)
    op = cs.createKinshipOperator(g)
    Z = ref.dense_z(None, None)
    V = np.random.default_rng(m).standard_normal((m, 1))
    E = Z @ V
    Y = op.multiply_Z_v(V)
    assert np.abs(Y - E).max() <= 64 * np.sqrt(m) * 2.0 ** -53 * np.abs(E).max()
