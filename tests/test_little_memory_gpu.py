"""FP64 products where device memory is short: wide calls run in narrower chunks, and where not even those
fit on the FP64-pipe kernels, until the memory is there.

CS_B200_ALLOC_LIMIT=bytes:count has the library refuse its first `count` blocks above a size as a full
device would; a process runs one scenario.  Both forms are FP64 products; against each other (and against the
undivided call, whose slice sums differ) 2^-46 of a column's largest entry, a few times what either is off
by.
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
# the packed matrix takes 12.3 MB, its sample-major copy 12.6, the digits of 288, 144 and 72 columns 38, 19, 9
N, M = 6000, 8000
COPY = 12_400_000
TOL = 2.0 ** -46


def operators():
    d = synth.cohort(N, M, 3, missing=0.02, n_causal=5)
    g = cs.Genotypes.from_bed_bytes(d["bed"], N, M)
    return cs.createKinshipOperator(g), cs.createKinshipOperator(g), np.random.default_rng(0)


def routed(call):
    cs.profile_enable()
    out = call()
    names = [k["name"] for k in cs.profile_summary()["kernels"]]
    cs.profile_enable(False)
    return out, any("_slices" in s for s in names)


def close(a, b):
    return bool((np.abs(a - b).max(axis=0) <= TOL * np.abs(b).max(axis=0)).all())


def narrower_chunks():
    op, whole, rng = operators()
    X = rng.standard_normal((N, 300))
    got, on_digits = routed(lambda: op.apply(X))
    again, _ = routed(lambda: op.apply(X))
    want = whole.apply(X)
    assert on_digits and close(got, want) and not np.array_equal(got, want)
    assert np.array_equal(again, want)


def pipe_kernels_until_there_is_room():
    op, whole, rng = operators()
    X, V = rng.standard_normal((N, 1)), rng.standard_normal((M, 1))
    calls = (lambda o: o.apply(X), lambda o: o.multiply_Z_v(V), lambda o: o.multiply_Zt_v(X))
    short = [routed(lambda: f(op)) for f in calls]
    assert [on_digits for _, on_digits in short] == [False, False, True]  # the last needs no copy
    for f, (got, _) in zip(calls, short):
        want = f(whole)
        later, on_digits = routed(lambda: f(op))
        assert close(got, want) and on_digits and np.array_equal(later, want)


def wide_call_that_fails():
    """Neither the copy nor, on the pipe kernels, the 64 columns' sums fit; narrow calls later do not mind."""
    op, whole, rng = operators()
    X = rng.standard_normal((N, 64))
    with pytest.raises(cs.CosmicError, match="allocation"):
        op.apply(X)
    got, on_digits = routed(lambda: op.apply(X[:, :1]))
    assert on_digits and np.array_equal(got, whole.apply(X[:, :1]))


def pool_used():
    """Bytes in use in the device's default memory pool."""
    import ctypes as C

    cuda = C.CDLL("libcuda.so.1")
    dev, pool, used = C.c_int(), C.c_void_p(), C.c_uint64()
    assert cuda.cuDeviceGet(C.byref(dev), 0) == 0
    assert cuda.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    assert cuda.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


def failed_solve_keeps_no_workspace():
    """64 columns' blocks take 3 MB each; the product's buffers do not fit, so the solve fails with the
    blocks made.  What a failed product leaves with its operator is there before."""
    pytest.importorskip("torch")
    op, _, rng = operators()
    B = rng.standard_normal((N, 64))
    pcg = cs.MatrixFreePCG(op, 0.5, 0.5, precision="fp64")
    with pytest.raises(cs.CosmicError, match="allocation"):
        op.apply(B)
    before = pool_used()
    with pytest.raises(cs.CosmicError, match="allocation"):
        pcg.solve(B)
    assert pool_used() - before < 1 << 20
    assert np.isfinite(pcg.solve(B)).all()


SCENARIOS = {f.__name__: f for f in (narrower_chunks, pipe_kernels_until_there_is_room, wide_call_that_fails,
                                     failed_solve_keeps_no_workspace)}
SCRIPT = r"""
import sys
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
import test_little_memory_gpu
test_little_memory_gpu.SCENARIOS[sys.argv[2]]()
print("scenario ran")
"""


@pytest.mark.parametrize("name,limit,count", [("narrower_chunks", 14 << 20, 2),
                                              ("pipe_kernels_until_there_is_room", COPY, 2),
                                              ("wide_call_that_fails", COPY, 2),
                                              ("failed_solve_keeps_no_workspace", COPY, 4)])
def test_with_little_memory(name, limit, count):
    env = dict(os.environ, CS_B200_ALLOC_LIMIT="%d:%d" % (limit, count))
    res = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, name], env=env, capture_output=True, text=True)
    assert res.returncode == 0 and "scenario ran" in res.stdout, res.stdout + res.stderr
