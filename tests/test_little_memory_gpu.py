"""FP64 products where device memory is short: wide calls run in narrower chunks, and where not even those
fit on the FP64-pipe kernels, until the memory is there.

CS_B200_ALLOC_LIMIT has the library refuse blocks above a size as a full device would.  Both forms are FP64
products; against each other (and against the undivided call, whose slice sums differ) 2^-46 of a
column's largest entry, a few times what either is off by.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")

N, M = 6000, 8000  # the sample-major copy takes 12 MB, 288 columns' digits 38 MB, one column of the pipe kernels 6
TOL = 2.0 ** -46


@pytest.fixture
def limit():
    def set_to(nbytes):
        if nbytes is None:
            os.environ.pop("CS_B200_ALLOC_LIMIT", None)
        else:
            os.environ["CS_B200_ALLOC_LIMIT"] = str(nbytes)
    yield set_to
    set_to(None)


@pytest.fixture(scope="module")
def genotypes():
    d = synth.cohort(N, M, 3, missing=0.02, n_causal=5)
    return cs.Genotypes.from_bed_bytes(d["bed"], N, M)


def routed(call):
    cs.profile_enable()
    out = call()
    names = [k["name"] for k in cs.profile_summary()["kernels"]]
    cs.profile_enable(False)
    return out, any("_slices" in s for s in names)


def close(a, b):
    return bool((np.abs(a - b).max(axis=0) <= TOL * np.abs(b).max(axis=0)).all())


def test_narrower_chunks(genotypes, limit):
    X = np.random.default_rng(0).standard_normal((N, 300))
    want, on_digits = routed(lambda: cs.createKinshipOperator(genotypes).apply(X))
    assert on_digits
    op = cs.createKinshipOperator(genotypes)
    limit(14 << 20)
    got, on_digits = routed(lambda: op.apply(X))
    assert on_digits and close(got, want)
    limit(None)
    got, on_digits = routed(lambda: op.apply(X))
    assert on_digits and np.array_equal(got, want)


def test_pipe_kernels_until_there_is_room(genotypes, limit):
    rng = np.random.default_rng(1)
    X, V = rng.standard_normal((N, 1)), rng.standard_normal((M, 1))
    whole = cs.createKinshipOperator(genotypes)
    calls = (lambda op: op.apply(X), lambda op: op.multiply_Z_v(V), lambda op: op.multiply_Zt_v(X))
    want = [f(whole) for f in calls]
    op = cs.createKinshipOperator(genotypes)
    limit(8 << 20)
    for f, w in list(zip(calls, want))[:2]:  # the third needs no copy
        got, on_digits = routed(lambda: f(op))
        assert not on_digits and close(got, w)
    limit(None)
    for f, w in zip(calls, want):
        got, on_digits = routed(lambda: f(op))
        assert on_digits and np.array_equal(got, w)


def test_wide_call_that_fails_leaves_narrow_ones_alone(genotypes, limit):
    X = np.random.default_rng(2).standard_normal((N, 64))
    op = cs.createKinshipOperator(genotypes)
    want = op.apply(X[:, :1])
    limit(1 << 19)  # room for neither form's 64 columns
    with pytest.raises(cs.CosmicError, match="allocation"):
        op.apply(X)
    limit(None)
    got, on_digits = routed(lambda: op.apply(X[:, :1]))
    assert on_digits and np.array_equal(got, want)


def pool_used():
    """Bytes in use in the device's default memory pool."""
    import ctypes as C

    cuda = C.CDLL("libcuda.so.1")
    dev, pool, used = C.c_int(), C.c_void_p(), C.c_uint64()
    assert cuda.cuDeviceGet(C.byref(dev), 0) == 0
    assert cuda.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    assert cuda.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


def test_failed_solve_keeps_no_workspace(genotypes, limit):
    """64 columns' blocks take 3 MB each; the product's buffers do not fit, so the solve fails with the
    blocks made.  What a failed product leaves with its operator is there before."""
    pytest.importorskip("torch")
    op = cs.createKinshipOperator(genotypes)
    B = np.random.default_rng(3).standard_normal((N, 64))
    pcg = cs.MatrixFreePCG(op, 0.5, 0.5, precision="fp64")
    limit(4 << 20)
    with pytest.raises(cs.CosmicError, match="allocation"):
        op.apply(B)
    before = pool_used()
    with pytest.raises(cs.CosmicError, match="allocation"):
        pcg.solve(B)
    assert pool_used() - before < 1 << 20
    limit(None)
    x = pcg.solve(B)
    assert np.isfinite(x).all()
