"""FP64 products where W = s^2 o Z^T x is uneven: cohorts with variants that one sample, or up to
twenty, carry among common ones (s^2 is n for the former).

Reference: the product in extended precision.  Bound, relative in the 2-norm of a column: plain FP64
sums are off by about 1e-15 at these sizes (2^-53 sqrt(K) of partial sums in a random walk); the
fixed-point products must not be further off than that.  A column in 63 bits whose elements lie 2^8
below its maximum holds them to 2^-55, and the two roundings of u, the two of W and the one of the
result are independent, about 2^-53 sqrt(5) / 3 together; 2^-51 leaves a factor of five and is half
of the FP64 sums' error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")

TOL = 2.0 ** -51


def cohort(n, m, rare, counts, missing, seed):
    """.bed bytes and Z (extended precision) of common variants and a share `rare` of rare ones."""
    rng = np.random.default_rng(seed)
    maf = rng.uniform(0.01, 0.5, (m, 1))
    G = (rng.random((m, n)) < maf).astype(np.int8) + (rng.random((m, n)) < maf)
    for t in np.flatnonzero(rng.random(m) < rare):
        G[t] = 0
        G[t, rng.choice(n, rng.integers(counts[0], counts[1] + 1), replace=False)] = 1
    miss = rng.random((m, n)) < missing
    miss[G.sum(axis=1) <= counts[1]] &= G[G.sum(axis=1) <= counts[1]] == 0  # carriers stay
    code = np.where(miss, 1, np.array([3, 2, 0], dtype=np.uint8)[G]).astype(np.uint8)
    pad = np.ones((m, -(-n // 4) * 4), dtype=np.uint8)
    pad[:, :n] = code
    q = pad.reshape(m, -1, 4)
    rows = q[:, :, 0] | (q[:, :, 1] << 2) | (q[:, :, 2] << 4) | (q[:, :, 3] << 6)
    bed = np.concatenate([np.array([0x6C, 0x1B, 0x01], np.uint8), rows.ravel()])
    return bed, G, miss


def exact_z(g, G, miss):
    """The Z of the matrix's own FP64 means and scales, (samples, variants)."""
    st = g.stats()
    mean, inv_std = st["mean"], st["inv_std"]
    Z = (G.astype(np.longdouble) - mean.astype(np.longdouble)[:, None]) * inv_std.astype(np.longdouble)[:, None]
    Z[miss] = 0
    return Z.T


@pytest.mark.parametrize("n,m,rare,counts,missing", [(6000, 3000, 0.05, (1, 1), 0.0),
                                                     (6000, 3000, 0.05, (1, 1), 0.02),
                                                     (12000, 1500, 0.05, (1, 1), 0.01),
                                                     (9001, 1300, 0.02, (1, 20), 0.02)])
def test_error_against_extended_precision(n, m, rare, counts, missing):
    bed, G, miss = cohort(n, m, rare, counts, missing, n + m)
    g = cs.Genotypes.from_bed_bytes(bed, n, m)
    op = cs.createKinshipOperator(g)
    Z = exact_z(g, G, miss)
    rng = np.random.default_rng(1)
    err = lambda y, e: float(np.sqrt((((y - e) ** 2).sum(axis=0) / (e ** 2).sum(axis=0)).max()))
    for k in (1, 5):
        X, V = rng.standard_normal((n, k)), rng.standard_normal((m, k))
        U = Z.T @ X.astype(np.longdouble)
        assert err(op.apply(X), Z @ U / m) < TOL, k
        assert err(op.multiply_Zt_v(X), U) < TOL, k
        assert err(op.multiply_Z_v(V), Z @ V.astype(np.longdouble)) < TOL, k
