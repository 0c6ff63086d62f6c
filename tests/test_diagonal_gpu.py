"""The diagonal of K at the edges of its kernel: odd row counts (two rows a step, 64 a table), samples
that leave words and blocks part full, cohorts and monomorphic variants.

Both sides sum m squares in FP64, in different orders: sqrt(m) 2^-53 of the sum, times 64.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402


@pytest.mark.parametrize("n,m", [(3, 1), (17, 2), (64, 63), (255, 65), (2047, 129), (2049, 1000), (9001, 700)])
@pytest.mark.parametrize("cohort", [False, True])
def test_diagonal(n, m, cohort):
    d = synth.cohort(n, m, n + m, missing=0.05, n_causal=1, maf_lo=0.1)
    rows = d["bed"][3:].reshape(m, -1)
    if m > 5:
        rows[4] = 0xFF  # every call 11: no variance
    d["bed"][3:] = rows.ravel()
    ref = oracle.Bed(rows, n)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    rng = np.random.default_rng(n)
    keep = rng.permutation(n)[: max(2, n - n // 5)].astype(np.int32) if cohort else None
    variants = np.arange(0, m, 2, dtype=np.int32) if cohort else None
    op = cs.createKinshipOperator(g, keep, variants) if cohort else cs.createKinshipOperator(g)
    Z = ref.dense_z(keep, variants).astype(np.longdouble)
    E = (Z * Z).sum(axis=1) / Z.shape[1]
    assert (np.abs(op.getDiagonal() - E) <= 64 * np.sqrt(m) * 2.0 ** -53 * np.maximum(E, 1e-300)).all()
