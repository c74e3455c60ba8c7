"""The plain FP64 path's tensor-core launch: outputs stay at the level of an
FP64 sum entry by entry, whatever the operands hold.

The bound is the one of an FP64 dot product of real depth n in any order,
n u sum_k |a_ik b_kj| (u = 2^-53), times 4.3 for the digits' truncation (the
certificate of the launch) plus one rounding of the result; operands that miss
the certificate are recomputed by the FP64 kernel and meet the same bound."""
import numpy as np
import pytest

from qspace_gb300._capi import QSError
from qspace_gb300.grouped import DeviceBatch, Packed

U = 2.0 ** -53


def _ops(rng, M, N, K, cplx):
    a, b = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    if cplx:
        a = a + 1j * rng.standard_normal((M, K))
        b = b + 1j * rng.standard_normal((K, N))
    return a, b


def _stored(x, trans, conj):
    """The array to store so that op(stored) = x."""
    x = x.conj() if conj else x
    return x.T if trans else x


def _batch(ops, afac, blk, trans):
    """DeviceBatch whose pair p computes afac ops[p][0] @ ops[p][1]."""
    cplx = np.iscomplexobj(ops[0][0])
    pk = Packed([a for a, _ in ops], [b for _, b in ops], afac, blk=blk, cplx=cplx)
    pk.trans = np.asarray(trans, np.int32)
    flat = lambda xs: np.concatenate([np.asarray(x, pk.abuf.dtype).reshape(-1, order="F") for x in xs])  # noqa: E731
    pk.abuf = flat([_stored(a, t & 1, t & 4) for (a, _), t in zip(ops, trans)])
    pk.bbuf = flat([_stored(b, t & 2, t & 8) for (_, b), t in zip(ops, trans)])
    pk.lda = np.maximum(np.where(pk.trans & 1, pk.K, pk.M), 1).astype(np.int32)
    pk.ldb = np.maximum(np.where(pk.trans & 2, pk.N, pk.K), 1).astype(np.int32)
    return DeviceBatch(pk)


def _reference(ops, afac, blk):
    """Per block: the product in extended precision, sum |a||b| and depth."""
    out = {}
    for (a, b), f, g in zip(ops, afac, blk):
        wide = np.clongdouble if np.iscomplexobj(a) else np.longdouble
        fa = (a * f).astype(wide)       # the factor enters as the FP64 kernel applies it
        c = fa @ b.astype(wide)
        s = np.abs(a.real * f) @ np.abs(b.real) + np.abs(a.imag * f) @ np.abs(b.imag) + \
            np.abs(a.real * f) @ np.abs(b.imag) + np.abs(a.imag * f) @ np.abs(b.real)
        n = a.shape[1] * (2 if np.iscomplexobj(a) else 1)
        if g in out:
            c0, s0, n0 = out[g]
            out[g] = (c0 + c, s0 + s, n0 + n)
        else:
            out[g] = (c, s, n)
    return [out[g] for g in sorted(out)]


def _check(got, ref):
    for c, (r, s, n) in zip(got, ref):
        d = c - r
        err = np.maximum(np.abs(d.real), np.abs(d.imag)).astype(float)
        # n + 1: the factor's rounding in FP64 (exact in the digits)
        bound = 4.3 * (n + 1) * U * s + 2 * U * np.abs(r).astype(float)
        assert np.all(err <= bound), float(np.max(err / np.maximum(bound, 1e-300)))


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shape", [(64, 64, 48), (40, 70, 24), (65, 33, 96), (129, 31, 97), (1, 700, 130), (700, 1, 130),
                                   (128, 32, 193), (63, 127, 512), (31, 33, 9), (17, 48, 20), (64, 16, 16),
                                   (1, 33, 17), (300, 200, 5), (260, 515, 9)])
def test_f64_tensor_sizes(shape, cplx):
    rng = np.random.default_rng(5)
    M, N, K = shape
    ks = [K, max(K // 3, 1), 1]
    ops = [_ops(rng, M, N, k, cplx) for k in ks]
    afac, blk = [0.75, -0.3137, 1.0], [0, 0, 0]
    ref = _reference(ops, afac, blk)
    norm = float(np.linalg.norm(ref[0][0].astype(complex)))
    for trans in ([0, 0, 0], [1, 2, 3], [15, 7, 8]):
        trans = [t if cplx else t & 3 for t in trans]
        db = _batch(ops, afac, blk, trans)
        db.run("fp64")
        got = db.result()
        _check(got, ref)
        d = (got[0] - ref[0][0]).astype(complex)
        assert np.linalg.norm(d) <= 4e-16 * np.sqrt(ref[0][2]) * norm
        # the plan runs the same launches: same bits
        plan = db.plan("fp64")
        for _ in range(3):
            db.dC.zero_()
            db.torch.cuda.synchronize()
            db.run_plan(plan)
            assert np.array_equal(db.result()[0], got[0])
        plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["graded", "sparse", "tiny_overlap", "zero_line", "huge", "subnormal", "factors"])
def test_f64_tensor_hard_operands(kind):
    """Entries of very different sizes, disjoint supports, extreme
    exponents: every output keeps the FP64 bound."""
    rng = np.random.default_rng(11)
    M, N, K = 90, 75, 200
    a, b = _ops(rng, M, N, K, False)
    afac = [1.0, 0.5]
    if kind == "graded":
        a *= 10.0 ** -np.linspace(0, 30, K)[None, :]
        b *= 10.0 ** -np.linspace(30, 0, K)[:, None]
    elif kind == "sparse":
        a *= rng.random((M, K)) < 0.02
        b *= rng.random((K, N)) < 0.02
    elif kind == "tiny_overlap":
        a[:, K // 2:] *= 1e-14
        b[:K // 2, :] = 0.0
    elif kind == "zero_line":
        a[7, :] = 0.0
        b[:, 11] = 0.0
        a[:, 5] = 0.0
    elif kind == "huge":
        a *= 1e200
        b *= 1e-190
        a[3, 3] = 1e307
    elif kind == "subnormal":
        a *= 1e-160
        b *= 1e-150
    else:
        afac = [1e-290, 3.0]
    ops = [(a, b), _ops(rng, M, N, 64, False)]
    if kind in ("huge", "subnormal"):
        ops = ops[:1]
    afac, blk = afac[:len(ops)], [0] * len(ops)
    db = _batch(ops, afac, blk, [0] * len(ops))
    db.run("fp64")
    if kind == "subnormal":  # results below the normal range: absolute spacing 2^-1074
        r, s, n = _reference(ops, afac, blk)[0]
        err = np.abs(db.result()[0] - r).astype(float)
        assert np.all(err <= 4.3 * (n + 1) * U * s + 2 * U * np.abs(r).astype(float) + n * 2.0 ** -1074)
    else:
        _check(db.result(), _reference(ops, afac, blk))


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
def test_f64_tensor_nonfinite(cplx):
    """Infinities and NaN in the operands reach the outputs that FP64
    arithmetic gives them, and no others."""
    rng = np.random.default_rng(3)
    M, N, K = 150, 140, 80
    a, b = _ops(rng, M, N, K, cplx)
    a[17, 5] = np.nan
    a[70, 9] = np.inf
    b[3, 100] = -np.inf
    ok = np.ones((M, N), bool)
    ok[17, :] = ok[70, :] = False
    ok[:, 100] = False
    db = _batch([(a, b)], [1.0], [0], [0])
    db.run("fp64")
    c = db.result()[0]
    assert np.all(np.isfinite(c[ok])) and not np.any(np.isfinite(c[~ok]))
    a2, b2 = np.where(np.isfinite(a), a, 0), np.where(np.isfinite(b), b, 0)
    r, s, n = _reference([(a2, b2)], [1.0], [0])[0]
    err = np.abs(c[ok] - r[ok]).astype(float)
    assert np.all(err <= 4.3 * 2 * (n + 1) * U * s[ok])
    if not cplx:
        with np.errstate(invalid="ignore"):
            w = a @ b
        assert np.array_equal(np.isnan(c), np.isnan(w)) and np.array_equal(c[np.isinf(w)], w[np.isinf(w)])


@pytest.mark.gpu
def test_f64_tensor_alone_and_in_a_list():
    """A block gives the same bits alone and in a list of others."""
    rng = np.random.default_rng(8)
    sizes = [(100, 90, 60), (8, 8, 8), (300, 20, 333), (64, 64, 47), (33, 257, 129)]
    ops = [_ops(rng, *s, True) for s in sizes]
    afac = list(rng.uniform(-1, 1, len(ops)))
    db = _batch(ops, afac, list(range(len(ops))), [0] * len(ops))
    db.run("fp64")
    for p, c in enumerate(db.result()):
        one = _batch([ops[p]], [afac[p]], [0], [0])
        one.run("fp64")
        assert np.array_equal(one.result()[0], c)


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_shallow_blocks(prec, cplx):
    """Blocks with at most eight summed terms: either side long, remainders of
    the register and line blocking, several pairs, factors, every flag."""
    rng = np.random.default_rng(21)
    ops, afac, blk, trans = [], [], [], []
    for g, (M, N) in enumerate([(1, 1), (1, 700), (700, 1), (31, 40), (32, 31), (513, 9), (5, 1025), (2, 513), (70, 17)]):
        for K, f in ((3, 1.0), (1, -0.31), (0, 1.0), (4, 0.77)):
            ops.append(_ops(rng, M, N, K, cplx))
            afac.append(f)
            blk.append(g)
            trans.append(int(rng.integers(0, 16 if cplx else 4)))
    db = _batch(ops, afac, blk, trans)
    db.run(prec)
    got = db.result()
    ref = _reference(ops, afac, blk)
    if prec == "fp64":
        _check(got, ref)
    else:  # blocks that the digits take instead: the path's own tolerance
        for c, (r, s, n) in zip(got, ref):
            assert np.linalg.norm((c - r).astype(complex)) <= 1e-12 * np.linalg.norm(s)
    plan = db.plan(prec)
    db.run_plan(plan)
    for c, d in zip(db.result(), got):
        assert np.array_equal(c, d)
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1])
def test_shallow_complex_alignment(shift):
    """Complex buffers at an odd multiple of eight bytes, direct blocks."""
    rng = np.random.default_rng(2)
    ops = [_ops(rng, 50, 3, 2, True), _ops(rng, 4, 90, 5, True)]
    db = _batch(ops, [1.0, 0.5], [0, 1], [0, 0])
    t = db.torch
    pad = lambda x: t.cat([t.zeros(shift, dtype=t.float64, device=x.device), x])[shift:]  # noqa: E731
    want = _reference(ops, [1.0, 0.5], [0, 1])
    db.dA, db.dB, db.dC = pad(db.dA), pad(db.dB), pad(db.dC)
    t.cuda.synchronize()
    db.run("fp64")
    _check(db.result(), want)


def _shifted(db, shift):
    t = db.torch
    pad = lambda x: t.cat([t.zeros(shift, dtype=t.float64, device=x.device), x])[shift:]  # noqa: E731
    db.dA, db.dB, db.dC = pad(db.dA), pad(db.dB), pad(db.dC)
    t.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 32, 8), (64, 64, 8), (256, 256, 8), (90, 130, 5), (33, 200, 6)])
def test_large_shallow_blocks_take_any_alignment(shape):
    """A block summed over at most 8 terms is computed directly on the FP64
    path whatever its size: with the bits of the aligned call, from buffers at
    an odd multiple of eight bytes too, alone, with others and from a plan."""
    M, N, K = shape
    rng = np.random.default_rng(7)
    ops, afac, blk, trans = [_ops(rng, M, N, K, True), _ops(rng, 3, 5, 2, True)], [-0.7, 1.0], [0, 1], [5, 10]
    db = _batch(ops, afac, blk, trans)
    db.run("fp64")
    want = [c.copy() for c in db.result()]
    _check(want, _reference(ops, afac, blk))
    _shifted(db, 1)
    db.run("fp64")
    for c, w in zip(db.result(), want):
        assert np.array_equal(c, w)
    plan = db.plan("fp64")
    db.dC.fill_(float("nan"))
    db.torch.cuda.synchronize()
    db.run_plan(plan)
    for c, w in zip(db.result(), want):
        assert np.array_equal(c, w)
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_deeper_misaligned_blocks_are_refused_on_the_host(prec):
    """Tiles move whole complex values: buffers that are not aligned to them
    are an error, raised before anything is launched."""
    rng = np.random.default_rng(8)
    ops = [_ops(rng, 40, 40, 48, True), _ops(rng, 4, 6, 2, True)]
    db = _batch(ops, [1.0, 1.0], [0, 1], [0, 0])
    _shifted(db, 1)
    db.dC.fill_(7.0)
    db.torch.cuda.synchronize()
    plan = db.plan(prec)
    n0 = db.ctx.launches
    with pytest.raises(QSError, match="aligned to 16"):
        db.run(prec)
    with pytest.raises(QSError, match="aligned to 16"):
        db.run_plan(plan)
    assert db.ctx.launches == n0
    plan.close()
    db.ctx.sync()
    assert bool((db.dC == 7.0).all())


def _digits(d0, low):
    """An entry below 1 whose 8-bit digits are d0 and then `low` six times."""
    return d0 * 2.0 ** -8 + sum(low * 2.0 ** (-8 * t) for t in range(2, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("K,d0,low", [(4103, 1, -128), (4103, 1, 127), (2050, 2, -128), (1030, 5, -128), (66, 20, -128),
                                      (66, 19, -128), (66, 20, 127), (34, 28, -128), (34, 40, -128), (200, 12, -128)])
@pytest.mark.parametrize("trans", [0, 3])
def test_f64_tensor_bound_of_an_fp64_sum(K, d0, low, trans):
    """Every digit product that is left out has the same sign, and the leading
    digits overstate (or understate) the entries; one full-scale entry per line
    faces a zero.  The bound is an FP64 dot product's own, n u sum |a_k b_k|, with
    one rounding each for the factor and the result."""
    M, N = 64, 40
    a, b = np.full((M, K), _digits(d0, low)), np.full((K, N), _digits(d0, low))
    a[:, 0], b[0, :] = 0.75, 0.0
    a[:, 1], b[1, :] = 0.0, -0.875
    ops, afac = [(a, b)], [1.0]
    db = _batch(ops, afac, [0], [trans])
    db.run("fp64")
    (r, s, n), = _reference(ops, afac, [0])
    err = np.abs(db.result()[0] - r).astype(float)
    assert np.all(err <= n * U * s + 2 * U * np.abs(r).astype(float)), float(np.max(err / (n * U * s)))


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("K", [31, 32, 33, 64, 700])
def test_f64_tensor_skewed_entries(K, cplx):
    """Log-normal entries: many outputs are far below their lines' maxima."""
    rng = np.random.default_rng(K)
    a, b = _ops(rng, 70, 99, K, cplx)
    a, b = a * np.exp(2 * rng.standard_normal(a.shape)), b * np.exp(2 * rng.standard_normal(b.shape))
    db = _batch([(a, b)], [0.6], [0], [0])
    db.run("fp64")
    (r, s, n), = _reference([(a, b)], [0.6], [0])
    d = db.result()[0] - r
    err = np.maximum(np.abs(d.real), np.abs(d.imag)).astype(float)
    assert np.all(err <= (n + 1) * U * s + 2 * U * np.abs(r).astype(float))


@pytest.mark.gpu
@pytest.mark.parametrize("f", [2.0 ** -1022, 1e-312, -1e-315, 3e-320, 2e-322, 2.0 ** -1074])
def test_subnormal_factors(f):
    """Large entries times a subnormal factor are ordinary numbers, exact to
    one rounding of x f."""
    rng = np.random.default_rng(13)
    a, b = _ops(rng, 70, 60, 96, False)
    a *= 1e290 if abs(f) > 1e-318 else 1e300
    ops, afac = [(a, b)], [f]
    db = _batch(ops, afac, [0], [0])
    db.run("fp64")
    ref = _reference(ops, afac, [0])
    (r, s, n), = ref
    err = np.abs(db.result()[0] - r).astype(float)
    assert np.all(err <= (n + 1) * U * s + 2 * U * np.abs(r).astype(float))
    for nslices in (0, 7):
        db.run("split", nslices=nslices)
        d = ((db.result()[0] - r) * 2.0 ** 60).astype(float)
        assert np.linalg.norm(d) <= 1e-12 * np.linalg.norm((s * 2.0 ** 60).astype(float))


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
def test_f64_cells_of_a_list(cplx):
    """Blocks of which all, some or no outputs are computed again, depths far
    apart, edges of the 16 x 16 cells; from a plan the cells are listed anew on
    every run."""
    rng = np.random.default_rng(17)
    ops, trans = [], []
    for M, N, K in [(16, 16, 2100), (17, 31, 640), (1, 513, 99), (513, 1, 99), (15, 90, 70), (160, 48, 33), (49, 64, 257),
                    (300, 260, 40)]:
        for kind in ("skew", "identity", "some", "none"):
            a, b = _ops(rng, M, N, K, cplx)
            if kind == "skew":
                a = a * np.exp(3 * rng.standard_normal(a.shape))
                b = b * np.exp(3 * rng.standard_normal(b.shape))
            elif kind == "identity":
                a = np.eye(M, K, dtype=a.dtype)
            elif kind == "some":
                a[M // 2, 1:] *= 1e-9
            ops.append((a, b))
            trans.append(int(rng.integers(0, 16 if cplx else 4)))
    n = len(ops)
    afac, blk = list(rng.uniform(0.5, 1.0, n)), list(range(n))
    db = _batch(ops, afac, blk, trans)
    db.run("fp64")
    got = [c.copy() for c in db.result()]
    for c, (r, s, k) in zip(got, _reference(ops, afac, blk)):
        d = c - r
        err = np.maximum(np.abs(d.real), np.abs(d.imag)).astype(float)
        assert np.all(err <= (k + 1) * U * s + 2 * U * np.abs(r).astype(float))
    plan = db.plan("fp64")
    for _ in range(3):
        db.dC.fill_(float("nan"))
        db.torch.cuda.synchronize()
        db.run_plan(plan)
        for c, w in zip(db.result(), got):
            assert np.array_equal(c, w)
    plan.close()


@pytest.mark.gpu
def test_long_columns_of_c():
    """Complex columns 2^30 elements apart: in doubles the stride leaves 32
    bits.  The FP64 path takes them, the split path refuses them on the host."""
    rng = np.random.default_rng(4)
    M, N, K, ldc = 64, 2, 256, 1 << 30
    ops = [_ops(rng, M, N, K, True)]
    db = _batch(ops, [1.0], [0], [0])
    db.pk.ldc[:] = ldc
    t = db.torch
    db.dC = t.empty((2 * (ldc * (N - 1) + M),), dtype=t.float64, device="cuda")
    t.cuda.synchronize()
    with pytest.raises(QSError, match="leading dimension"):
        db.run("split")
    db.run("fp64")
    db.ctx.sync()
    got = t.stack([db.dC[:2 * M], db.dC[2 * ldc:]]).cpu().numpy().view(np.complex128).T
    _check([got], _reference(ops, [1.0], [0]))


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("scale", [(1e200, 1e200, 1e-300), (1e-300, 1e200, 1e200), (1e-200, 1e-200, 1e250),
                                   (1e250, 1e-200, 1e-200), (1.0, 1e-315, 1e300), (1e300, 1e-315, 1.0)])
def test_shallow_factors_scale_the_sum(scale, cplx):
    """x f leaves the normal numbers, on some lines or all, where f (x y) does
    not: either side long, lines past the first of a thread, plans."""
    rng = np.random.default_rng(23)
    sa, f, sb = scale
    ops, afac, blk, trans = [], [], [], []
    for g, (M, N, K) in enumerate([(1, 1, 1), (700, 3, 4), (3, 700, 4), (5, 600, 1), (300, 33, 5), (129, 2, 3)]):
        a, b = _ops(rng, M, N, K, cplx)
        a[::3] *= sa
        b[:, ::2] *= sb
        ops += [(a, b), tuple(x * 1e-140 for x in _ops(rng, M, N, 2, cplx))]
        afac += [f, -0.31]
        blk += [g, g]
        trans += [int(t) for t in rng.integers(0, 16 if cplx else 4, 2)]
    db = _batch(ops, afac, blk, trans)
    db.run("fp64")
    got = [c.copy() for c in db.result()]
    wide = np.clongdouble if cplx else np.longdouble
    for g, c in enumerate(got):
        r, s, n = 0, 0, 1
        for (a, b), w in zip(ops[2 * g:2 * g + 2], afac[2 * g:2 * g + 2]):
            w = np.longdouble(w)
            r = r + w * (a.astype(wide) @ b.astype(wide))
            m = [np.abs(x).astype(np.longdouble) for x in (a.real, a.imag, b.real, b.imag)]
            s = s + abs(w) * ((m[0] + m[1]) @ (m[2] + m[3]))
            n += a.shape[1] * (2 if cplx else 1) + 1
        d = c - r
        err = np.maximum(np.abs(d.real), np.abs(d.imag))
        fits = s < 1e307  # others overflow
        assert np.all((err <= n * U * s + 1e-320)[fits]), float(np.max((err / s)[fits]))
    plan = db.plan("fp64")
    db.dC.fill_(float("nan"))
    db.torch.cuda.synchronize()
    db.run_plan(plan)
    for c, w in zip(db.result(), got):
        assert np.array_equal(c, w)
    plan.close()


@pytest.mark.gpu
def test_misaligned_blocks_are_refused_before_tuning():
    """A plan that times its digit widths on the first run looks at the buffers
    before that, and runs once they are aligned."""
    rng = np.random.default_rng(31)
    ops = [_ops(rng, 43, 41, 59, True), _ops(rng, 4, 6, 2, True)]
    db = _batch(ops, [1.0, 0.5], [0, 1], [0, 0])
    aligned = db.dA, db.dB, db.dC
    plan = db.plan("split", autotune=True)
    _shifted(db, 1)
    n0 = db.ctx.launches
    with pytest.raises(QSError, match="aligned to 16"):
        db.run_plan(plan)
    assert db.ctx.launches == n0
    db.dA, db.dB, db.dC = aligned
    db.run_plan(plan)
    for c, (r, s, n) in zip(db.result(), _reference(ops, [1.0, 0.5], [0, 1])):
        assert np.linalg.norm((c - r).astype(complex)) <= 1e-12 * np.linalg.norm(s)
    plan.close()
