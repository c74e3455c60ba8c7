"""The plain FP64 path where device memory is short.  QS_ALLOC_LIMIT_MB refuses
larger single allocations as if the device had no room for them."""
import numpy as np
import pytest

from qspace_gb300.grouped import DeviceBatch, Packed

U = 2.0 ** -53


def _batch(sizes, seed=0):
    rng = np.random.default_rng(seed)
    m = lambda r, c: rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))  # noqa: E731
    A, B = [m(M, K) for M, N, K in sizes], [m(K, N) for M, N, K in sizes]
    return DeviceBatch(Packed(A, B, rng.uniform(0.5, 1.0, len(sizes)))), A, B


def _runs(db):
    """Results of the one-shot call and of a plan's first and replayed run."""
    db.run("fp64")
    out = [[c.copy() for c in db.result()]]
    plan = db.plan("fp64")
    for _ in range(2):
        db.dC.fill_(float("nan"))
        db.torch.cuda.synchronize()
        db.run_plan(plan)
        out.append([c.copy() for c in db.result()])
    plan.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("limit", ["64", "16", "7"])
def test_several_launches_give_the_same_bits(limit, monkeypatch):
    """Digits of eight blocks, 6.3 MB each: in one launch where there is room,
    else in several that share the memory."""
    db, _, _ = _batch([(256, 256, 256)] * 8 + [(40, 50, 60), (5, 6, 7), (8, 8, 400)])
    want = _runs(db)[0]
    monkeypatch.setenv("QS_ALLOC_LIMIT_MB", limit)
    from qspace_gb300 import Context
    ctx = Context(0)  # no scratch of earlier calls
    db.ctx = ctx
    for got in _runs(db):
        assert all(np.array_equal(c, w) for c, w in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("limit", ["3", "0.2"])
def test_no_room_for_a_block(limit, monkeypatch):
    """Where one block's digits do not fit, the FP64 tiles compute the list, in
    the one-shot call and from a plan."""
    db, A, B = _batch([(256, 256, 256), (300, 40, 64), (70, 80, 90), (3, 4, 5)])
    monkeypatch.setenv("QS_ALLOC_LIMIT_MB", limit)
    from qspace_gb300 import Context
    db.ctx = Context(0)
    runs = _runs(db)
    for a, b, f, *cs in zip(A, B, db.pk.afac, *runs):
        r = (a * f).astype(np.clongdouble) @ b.astype(np.clongdouble)
        s = (np.abs(a.real) + np.abs(a.imag)) @ (np.abs(b.real) + np.abs(b.imag))
        for c in cs:
            assert np.all(np.abs(c - r).astype(float) <= (2 * a.shape[1] + 2) * U * s)
            assert np.array_equal(c, cs[0])


def _pool_used(high=False):
    """Bytes of the device's default pool in use (now, or at most since the
    last call with high=True)."""
    import ctypes
    import glob
    import os
    import torch
    torch.cuda.synchronize()
    names = ["libcudart.so.13", "libcudart.so.12", "libcudart.so"]
    names += glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "*", "lib", "libcudart.so*"))
    names += glob.glob("/usr/local/cuda/lib64/libcudart.so*")
    for n in names:
        try:
            rt = ctypes.CDLL(n)
            break
        except OSError:
            pass
    else:
        pytest.skip("no CUDA runtime library")
    pool, v = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    # cudaMemPoolAttrUsedMemCurrent = 7, cudaMemPoolAttrUsedMemHigh = 8
    assert rt.cudaMemPoolGetAttribute(pool, 8 if high else 7, ctypes.byref(v)) == 0
    used = v.value
    if high:
        zero = ctypes.c_uint64(0)
        assert rt.cudaMemPoolSetAttribute(pool, 8, ctypes.byref(zero)) == 0
    return used


@pytest.mark.gpu
def test_digits_go_back_to_the_pool():
    """A plain FP64 call leaves at most 16 MB of its digits with the context."""
    from qspace_gb300 import Context
    db, _, _ = _batch([(700, 600, 500), (900, 800, 300)])
    db.ctx = Context(0)
    db.ctx.sync()
    before = _pool_used()
    for _ in range(2):
        db.run("fp64")
        db.ctx.sync()
        assert _pool_used() - before <= 17 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("budget", [9, 14, 20, 40])
@pytest.mark.parametrize("nblk,n", [(1, 700), (4, 350)])
def test_serving_budget_covers_fp64_digits(nblk, n, budget):
    """Plain FP64 requests whose result and copies fit the budget are served
    within it: with all of their digits (17 MB here), with fewer at a time, or
    by the FP64 tiles."""
    from qspace_gb300 import Context, QSpace, contract_dev, upload
    from qspace_gb300.serve import Server
    rng = np.random.default_rng(5)
    q = np.arange(nblk, dtype=np.int32).reshape(-1, 1)
    a, b = ([rng.standard_normal((n, n)) for _ in range(nblk)] for _ in range(2))
    ctx = Context(0)
    A, B = upload(QSpace([q, q.copy()], a), ctx), upload(QSpace([q, q.copy()], b), ctx)
    want = contract_dev(A, "2", B, "1", prec="fp64").download().data
    ctx.sync()
    with Server(nslots=2, hbm_budget=budget << 20, ctx=ctx) as srv:
        before = _pool_used()
        _pool_used(high=True)
        tickets = [srv.submit(A, "2", B, "1") for _ in range(4)]
        for t in tickets:
            c, _ = srv.wait(t)
            got = c.download().data
            for x, y, r in zip(a, b, got):
                assert np.all(np.abs(r - x @ y) <= 2 * n * U * (np.abs(x) @ np.abs(y)))
            if budget == 40 or nblk == 4 and budget >= 14:
                assert all(np.array_equal(r, w) for r, w in zip(got, want))
            c.free()
        results = 4 * 8 * nblk * n * n  # of requests that are done, not yet collected
        assert _pool_used(high=True) - before <= (budget + 1 << 20) + results
