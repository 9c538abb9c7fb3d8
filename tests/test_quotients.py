"""Quotients through a reciprocal (div_by) against division, bit for bit, over
the range of exponents that its check admits and at the ends of it; and the
plane normals and lengths built on them against the reference's operations in
numpy (IEEE double division and square root, no contraction)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe():
    from libsupermesh_b200 import build

    return ctypes.CDLL(str(build.build_probe()))


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _quotients(probe, a, b):
    a, b = np.broadcast_arrays(a, b)
    da, db = _dev(a.ravel()), _dev(b.ravel())
    q, by = torch.empty_like(da), torch.empty_like(da)
    ok = torch.empty(len(da), dtype=torch.int32, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (da, db, q, by, ok)]
    torch.cuda.synchronize()
    assert probe.lsm_probe_quotients(ctypes.c_int64(len(da)), *p) == 0
    return a.ravel(), b.ravel(), q.cpu().numpy(), by.cpu().numpy(), ok.cpu().numpy().astype(bool)


def _check(probe, a, b, ok=True):
    a, b, q, by, admitted = _quotients(probe, a, b)
    with np.errstate(all="ignore"):
        assert np.array_equal(q.view(np.int64), (a / b).view(np.int64))
    assert np.array_equal(admitted, np.broadcast_to(ok, admitted.shape))
    assert np.array_equal(by[admitted].view(np.int64), q[admitted].view(np.int64))


def _mantissas(kind, n, rng):
    m = rng.integers(0, 1 << 52, n)
    if kind == "low":  # next to 1
        m = rng.integers(0, 64, n)
    elif kind == "high":  # next to 2
        m = (1 << 52) - 1 - rng.integers(0, 64, n)
    elif kind == "few":  # few bits set
        m = (1 << rng.integers(0, 52, n)) | (1 << rng.integers(0, 52, n))
    return (m | (1023 << 52)).view(np.float64) * rng.choice([-1.0, 1.0], n)


@pytest.mark.parametrize("ka", ["any", "low", "high", "few"])
@pytest.mark.parametrize("kb", ["any", "low", "high", "few"])
@pytest.mark.parametrize("ea,eb", [(0, 0), (399, -400), (-400, 399), (None, None)])
def test_quotients(probe, ka, kb, ea, eb):
    rng = np.random.default_rng([ord(ka[0]), ord(kb[0]), ea is None])
    n = 1 << 20
    a, b = _mantissas(ka, n, rng), _mantissas(kb, n, rng)
    e = [rng.integers(-400, 400, n) if x is None else x for x in (ea, eb)]
    _check(probe, np.ldexp(a, e[0]), np.ldexp(b, e[1]))


def test_quotients_next_to_a_rounding_boundary(probe):
    """a as near as doubles come to (q + half a unit) b: the quotients whose
    rounding is closest."""
    rng = np.random.default_rng(1)
    n = 1 << 20
    b, q = np.abs(_mantissas("any", n, rng)), np.abs(_mantissas("any", n, rng))
    a = b * q + b * 2.0 ** -53
    for step in range(-2, 3):
        _check(probe, (a.view(np.int64) + step).view(np.float64), b)


def test_range_ends(probe):
    """Admitted: magnitudes from 2^-400 to 2^400 (by the high word, so a
    millionth beyond); not zero, subnormals, infinities or NaN."""
    ends = np.array([2.0 ** -400, 2.0 ** 400, 1.0, -2.0 ** -400, -2.0 ** 400, 2.0 ** 400 * (1 - 2.0 ** -53),
                     2.0 ** -400 * (1 + 2.0 ** -52)])
    _check(probe, ends[:, None], ends[None])
    out = np.array([0.0, -0.0, 5e-324, 2.0 ** -1022, 2.0 ** -400 * (1 - 2.0 ** -53), 2.0 ** -401, 2.0 ** 400 * (1 + 2.0 ** -20),
                    2.0 ** 401, 1.7e308, np.inf, -np.inf, np.nan, -2.0 ** -402, -2.0 ** 900])
    for x, y in ((out[:, None], ends[None]), (ends[:, None], out[None]), (out[:, None], out[None])):
        a, b, _, _, admitted = _quotients(probe, x, y)
        assert not admitted.any(), (a[admitted], b[admitted])


def _norm2(v):
    """gfortran's NORM2 of a 3-vector, component by component."""
    scale, res = np.zeros(len(v)), np.ones(len(v))
    for x in np.abs(v).T:
        up = scale < x
        val = np.where(up, scale, x) / np.where(up, x, scale)
        r = np.where(up, 1.0 + res * (val * val), res + val * val)
        res, scale = np.where(x != 0.0, r, res), np.where((x != 0.0) & up, x, scale)
    return np.sqrt(res) * scale


@pytest.mark.parametrize("kind", ["any", "equal", "zeros", "scales", "large", "small", "not finite"])
def test_normals(probe, kind):
    rng = np.random.default_rng(len(kind))
    uv = rng.standard_normal((1 << 19, 6))
    if kind == "equal":  # equal components, equal and opposite vectors
        uv = np.round(uv)
    elif kind == "zeros":
        uv[rng.random(uv.shape) < 0.5] = 0.0
        uv[rng.random(uv.shape) < 0.1] = -0.0
    elif kind == "scales":
        uv *= 10.0 ** rng.uniform(-60, 60, uv.shape)
    elif kind == "large":
        uv *= 10.0 ** rng.uniform(50, 160, (len(uv), 1))
    elif kind == "small":
        uv *= 10.0 ** rng.uniform(-170, -50, (len(uv), 1))
    elif kind == "not finite":
        uv[rng.random(uv.shape) < 0.1] = np.inf
        uv[rng.random(uv.shape) < 0.1] = np.nan
    out = torch.empty((len(uv), 4), dtype=torch.float64, device="cuda")
    d = _dev(uv)
    torch.cuda.synchronize()
    assert probe.lsm_probe_normals(ctypes.c_int64(len(uv)), ctypes.c_void_p(d.data_ptr()),
                                   ctypes.c_void_p(out.data_ptr())) == 0
    (a, b, c), (x, y, z) = uv[:, :3].T, uv[:, 3:].T
    with np.errstate(all="ignore"):
        o = np.stack([b * z - c * y, c * x - a * z, a * y - b * x], 1)
        ref = np.concatenate([o / _norm2(o)[:, None], _norm2(uv[:, :3])[:, None]], 1)
    got = out.cpu().numpy()
    assert np.array_equal(got, ref, equal_nan=True)
    assert np.array_equal(np.signbit(got[~np.isnan(ref)]), np.signbit(ref[~np.isnan(ref)]))
