"""Matrices large enough for the staged upload: the same codes, statistics and products as numpy's,
at row lengths with every remainder of four samples, spare bits set in the file, a last piece that
is part full, and several threads uploading at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")
import oracle  # noqa: E402


def check(n, m, seed, pinned=False):
    d = synth.cohort(n, m, seed, missing=0.03, n_causal=2, maf_lo=0.05)
    rows = d["bed"][3:].reshape(m, -1)
    ref = oracle.Bed(rows.copy(), n)
    if n % 4:
        rows[:, -1] |= (0xFF << (2 * (n % 4))) & 0xFF  # spare codes of the last byte: not samples
    d["bed"][3:] = rows.ravel()
    bed = d["bed"]
    if pinned:
        torch = pytest.importorskip("torch")
        hold = torch.empty(bed.size, dtype=torch.uint8, pin_memory=True)
        hold.numpy()[:] = bed
        bed = hold.numpy()
    g = cs.Genotypes.from_bed_bytes(bed, n, m)
    s = g.stats()
    assert np.array_equal(s["mean"], ref.mean) and np.array_equal(s["inv_std"], ref.inv_std)
    op = cs.createKinshipOperator(g)
    X = np.random.default_rng(seed).standard_normal((n, 2))
    # Z^T X pins every row's place and every sample's: FP64 sums in two orders
    E = ref.dense_z(None, None).T @ X
    tol = 64 * np.sqrt(n) * 2.0 ** -53
    assert (np.abs(op.multiply_Zt_v(X) - E).max(axis=0) <= tol * np.abs(E).max(axis=0)).all()


# around the 2 MiB at which the staged copy begins, and several pieces a thread
@pytest.mark.parametrize("n,m", [(253, 32767), (256, 32768), (1001, 8193), (1002, 40000), (1003, 9000), (70001, 130)])
def test_staged_upload(n, m):
    check(n, m, n)


@pytest.mark.parametrize("n,m", [(253, 32768), (1002, 9000), (16383, 600), (16385, 600)])
def test_page_locked_source(n, m):
    check(n, m, n, pinned=True)


def test_uploads_from_several_threads():
    errors = []

    def one(seed):
        try:
            check(1001 + seed, 9000, seed)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=one, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
