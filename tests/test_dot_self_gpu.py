"""Deep sums of few outputs: an operand against its own conjugate takes a form of
its own (two multiply-adds per term, imaginary part zero), any other pair of
operands and sums that are not finite the general one.

Bound: an FP64 dot product of n terms in any order, n u sum_k |a_k|^2."""
import numpy as np
import pytest

from qspace_gb300 import QSpace, contract_dev, upload

U = 2.0 ** -53


def _tensor(seed, L, s, R):
    rng = np.random.default_rng(seed)
    q = [np.zeros((1, 1), np.int32) for _ in range(3)]
    return QSpace(q, [rng.standard_normal((L, s, R)) + 1j * rng.standard_normal((L, s, R))])


def _rho(T, ia, ib):
    t = upload(T)
    out = np.asarray(contract_dev(t, ia, t, ib, prec="fp64").download().data[0])
    t.free()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("L,s,R", [(91, 1, 97), (128, 2, 64), (8193, 3, 1), (331, 2, 257)])
@pytest.mark.parametrize("first", [True, False])
def test_self_products(L, s, R, first):
    T = _tensor(3, L, s, R)
    out = _rho(T, *(("13*", "13") if first else ("13", "13*"))).reshape(s, s)
    x = T.data[0].transpose(1, 0, 2).reshape(s, -1).astype(np.clongdouble)
    ref = (x.conj() @ x.T) if first else (x @ x.conj().T)
    mag = np.sqrt(np.outer((np.abs(x) ** 2).sum(1), (np.abs(x) ** 2).sum(1))).astype(float)
    d = out - ref
    n = 2 * L * R
    assert np.all(np.abs(d.real) <= n * U * mag) and np.all(np.abs(d.imag) <= n * U * mag)
    assert np.all(np.abs(np.diag(out).imag) <= n * U * np.diag(mag))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [complex(np.inf, 1.0), complex(1.0, -np.inf), complex(np.nan, 0.0), 1e200 + 1j])
def test_self_products_not_finite(value):
    """As an ordinary sum: Re and Im of each product added up."""
    T = _tensor(4, 96, 2, 91)
    T.data[0][7, 1, 5] = value
    out = _rho(T, "13*", "13").reshape(2, 2)
    v = np.float64(value.real), np.float64(value.imag)
    with np.errstate(invalid="ignore", over="ignore"):
        re, im = v[0] * v[0] + v[1] * v[1], v[0] * v[1] - v[1] * v[0]
    for got, want in ((out[1, 1].real, re), (out[1, 1].imag, im)):
        assert np.isnan(got) if np.isnan(want) else got == want if np.isinf(want) else np.isfinite(got)
    assert np.isfinite(out[0, 0])
