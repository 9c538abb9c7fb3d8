"""The converged triangle clip of the mesh paths (clip_tri_c) against the
walking one that explicit pairs take (clip_tri): the same operations on the
same values, so measures, counts and triangles are compared exactly; and
u^T M v by triangles against the assembled blocks."""
import time

import numpy as np
import pytest

from libsupermesh_b200 import meshes as M

pytestmark = pytest.mark.gpu


def _soup(kind, n, seed):
    """Two meshes of n triangles of their own nodes, in the unit square."""
    rng = np.random.default_rng(seed)
    a, b = (rng.random((n, 1, 2)) + 0.2 * rng.random((n, 3, 2)) for _ in range(2))
    if kind == "lattice":  # vertices on lines, shared and parallel edges
        a, b = np.round(a * 16) / 16, np.round(b * 16) / 16
    elif kind == "equal":
        b[::2] = a[::2][:, ::-1]
        b[1::4, :2] = a[1::4, :2]
    elif kind == "degenerate":
        a[::3, 2], b[::5, 1] = a[::3, 1], b[::5, 0]
    elif kind == "slivers":  # along common lines, as wide as rounding: 0.3 % are not convex after a cut
        base = rng.integers(0, 3, (n, 1, 2)) / 3.0 + 1.0
        ang = 2 * np.pi * rng.integers(0, 7, (n, 1)) / 7 + 0.1
        d = np.stack([np.cos(ang), np.sin(ang)], 2)
        eps = np.array([1e-16, 1e-15, 4e-16, 2e-16])[np.arange(n) % 4][:, None, None]
        a, b = (base + (2 * rng.random((n, 3, 1)) - 1) * d + eps * rng.standard_normal((n, 3, 2)) for _ in range(2))
    elif kind == "large":
        a, b = a * 1e160, b * 1e160  # products beyond the range of float64
    elif kind == "infinite":
        a[::4, 1, 0] = np.inf
        b[::7, 2, 1] = -np.inf
    en = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    return (a.reshape(-1, 2), en), (b.reshape(-1, 2), en)


@pytest.mark.parametrize("kind", ["plain", "lattice", "equal", "degenerate", "slivers", "large", "infinite"])
@pytest.mark.parametrize("n", [33, 2500])
def test_mesh_clip_matches_explicit_pairs(gpu_ctx, kind, n):
    A, B = _soup(kind, n, n)
    gpu_ctx.supermesh(A, B)
    cand = gpu_ctx.find_candidates(A, B)
    gpu_ctx.clip_candidates()
    ip, ind = gpu_ctx.get_candidates(n, cand)
    m, k = gpu_ctx.pair_results(cand)
    ra, rb = np.repeat(np.arange(n), np.diff(ip)), ind
    rm, rk, re = gpu_ctx.intersect_pairs(2, A[0][A[1]][ra], B[0][B[1]][rb], want_elems=True)
    assert np.array_equal(k, rk)
    assert np.array_equal(m, rm, equal_nan=True)
    el = gpu_ctx.supermesh_elements(A, B)
    ref = re[np.arange(22)[None] < rk[:, None]]
    got = next(x for x in (el if isinstance(el, tuple) else el.values())
               if isinstance(x, np.ndarray) and x.dtype == np.float64 and x.size == ref.size)
    assert np.array_equal(got.reshape(ref.shape), ref, equal_nan=True)


@pytest.mark.parametrize("na,nb,ja,jb", [(1, 1, 0.0, 0.0), (5, 5, 0.0, 0.0), (40, 33, 0.3, 0.0), (90, 120, 0.3, 0.3)])
@pytest.mark.parametrize("idx", [np.int32, np.int64])
def test_p1_integral_matches_blocks(gpu_ctx, na, nb, ja, jb, idx):
    A, B = M.grid2d(na, 3, ja), M.grid2d(nb, 2, jb)
    A, B = (A[0], A[1].astype(idx)), (B[0], B[1].astype(idx))
    u, v = np.cos(np.arange(len(A[0]))), np.sin(np.arange(len(B[0])))
    val, _ = gpu_ctx.p1_mass(A, B, u, v)
    ref, blocks = gpu_ctx.p1_mass(A, B, u, v, want_blocks=True)
    ip, ind = gpu_ctx.get_candidates(len(A[1]), len(blocks))
    ra = np.repeat(np.arange(len(A[1])), np.diff(ip))
    blocks = blocks.reshape(-1, 3, 3)
    # both sides round each of at most 12 terms of an entry a few tens of
    # times; the terms of an entry have one sign up to rounding
    size = np.einsum("pr,prc,pc->", np.abs(u[A[1]])[ra], np.abs(blocks), np.abs(v[B[1]])[ind])
    assert abs(val - ref) <= 64 * np.finfo(float).eps * size


def _hex(t):
    return np.array([[float.fromhex(x) for x in v] for v in t])


# Slivers as wide as rounding, one of whose lines crosses four edges of the
# polygon: the converged clip leaves them to the walking one.
_WIDE = [
    (_hex([("0x1.25ec3edd666e7p+1", "0x1.700d0fac74731p+0"), ("0x1.95566c555b37bp-1", "0x1.fc20a58afc4e9p+0"),
           ("0x1.4506cae77802fp+1", "0x1.596d9d3050b26p+0")]),
     _hex([("0x1.f413f2c3882f4p+0", "0x1.8ff826c2656e9p+0"), ("0x1.39f03c9cd95e6p+1", "0x1.617e32a93ccf8p+0"),
           ("0x1.430a68c3d917cp+0", "0x1.d05a25290acbfp+0")])),
    (_hex([("0x1.c188dd133aeafp+0", "0x1.b585e3d3c94dap+0"), ("0x1.be7ee163f36cap+0", "0x1.b537d4cde65b5p+0"),
           ("0x1.1bd3908418d4dp+1", "0x1.c15fd61e44f5fp+0")]),
     _hex([("0x1.1bb94011a4bfcp+1", "0x1.c15a8e51dfd0fp+0"), ("0x1.28b1c9f671cc0p+1", "0x1.c3f4e2e13f0c2p+0"),
           ("0x1.0242da45cea97p+0", "0x1.a254e6bb822dcp+0")])),
]


def _most_cuts(a, b):
    """The most edges of a's clipped polygon that one of b's lines crosses."""
    n = [(-(b[(i + 1) % 3][1] - b[i][1]), b[(i + 1) % 3][0] - b[i][0]) for i in range(3)]
    if (b[1] - b[0]) @ n[2] > 0:
        n = [(-x, -y) for x, y in n]
    p, most = [tuple(v) for v in a], 0
    for (nx, ny), (px, py) in zip(n, b):
        d = [nx * (x - px) + ny * (y - py) for x, y in p]
        q, cuts = [], 0
        for i, j in zip(range(len(p)), [*range(1, len(p)), 0]):
            if d[i] <= 0:
                q.append(p[i])
            if d[i] * d[j] < 0:
                f = abs(d[i]) / (abs(d[i]) + abs(d[j]))
                q.append(tuple(s + f * (t - s) for s, t in zip(p[i], p[j])))
                cuts += 1
        most, p = max(most, cuts), q
    return most


def _copies(t, other, n):
    """n triangles with their own nodes: t, every fifth one another."""
    v = np.repeat(t[None], n, 0)
    v[4::5] = other
    return v.reshape(-1, 2), np.arange(3 * n, dtype=np.int32).reshape(n, 3)


@pytest.mark.parametrize("a,b", _WIDE)
@pytest.mark.parametrize("n", [1, 4, 37, 300])
def test_pairs_left_to_the_walking_clip(gpu_ctx, oracle_mod, a, b, n):
    """Meshes most of whose candidates are such pairs (all, below n = 5), next
    to ordinary ones: measures against explicit pairs, and u^T M v with and
    without blocks, where a pair left out or taken twice is in plain sight."""
    assert _most_cuts(a, b) > 2
    plain = np.array([[0.9, 0.5], [2.4, 0.6], [1.6, 2.1]])
    A, B = _copies(a, plain, n), _copies(b, plain[::-1], n)
    st, _ = gpu_ctx.supermesh(A, B)
    cand = st.n_candidates
    assert cand == n * n
    m, k = gpu_ctx.pair_results(cand)
    ip, ind = gpu_ctx.get_candidates(n, cand)
    ra = np.repeat(np.arange(n), np.diff(ip))
    va, vb = A[0][A[1]][ra], B[0][B[1]][ind]
    rm, rk, re = gpu_ctx.intersect_pairs(2, va, vb, want_elems=True)
    assert np.array_equal(k, rk) and np.array_equal(m, rm)
    assert (k[(ra % 5 != 4) & (ind % 5 != 4)] > 2).all()
    # the largest basis value of any candidate at its points' surroundings
    used = np.arange(22)[None] < k[:, None]
    pts = (re[:, :, None] * (np.ones((3, 3)) / 6 + np.eye(3) / 2)[None, None, :, :, None]).sum(3)
    size = 1.0
    for v in (va, vb):
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        det = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
        r = pts - v[:, None, None, 0]
        l1 = (r[..., 0] * e2[:, None, None, 1] - r[..., 1] * e2[:, None, None, 0]) / det[:, None, None]
        l2 = (r[..., 1] * e1[:, None, None, 0] - r[..., 0] * e1[:, None, None, 1]) / det[:, None, None]
        size = max(size, *(np.abs(x[used]).max() for x in (l1, l2, 1 - l1 - l2)))
    # a value by numpy is off by rounding, which on these elements is as large
    # as the value: twice the size; a term is at most |u| |v| (3 size)^2 w, and
    # each side rounds it a few tens of times
    tol = 64 * np.finfo(float).eps * (6 * size) ** 2 * m.sum()
    one = np.ones(3 * n)
    val, _ = gpu_ctx.p1_mass(A, B, one, one)
    assert abs(val - m.sum()) <= tol
    u, v = np.cos(np.arange(3 * n)), np.sin(np.arange(3 * n) + 1.0)
    val, _ = gpu_ctx.p1_mass(A, B, u, v)
    ref, blocks = gpu_ctx.p1_mass(A, B, u, v, want_blocks=True)
    assert abs(val - ref) <= tol
    _, _, ob = oracle_mod.p1_mass(2, A, B, ip, ind, u, v, want_blocks=True)
    assert np.array_equal(blocks, ob.reshape(blocks.shape))


def test_many_pairs_left_to_the_walking_clip(gpu_ctx):
    """250,000 such pairs must not take one warp's time (19 ms; 0.11 ms spread
    over the chip, where 250,000 ordinary pairs take 0.04): at most forty
    times as long as the ordinary ones."""
    a, b = _WIDE[0]
    plain = np.array([[0.9, 0.5], [2.4, 0.6], [1.6, 2.1]])
    took = []
    for x, y in ((plain, plain[::-1] + 0.1), (a, b)):
        gpu_ctx.supermesh(_copies(x, x, 500), _copies(y, y, 500))
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            st = gpu_ctx.clip_candidates()
            best = min(best, time.perf_counter() - t)
        assert st.n_candidates == 250000 and st.n_intersecting == 250000
        took.append(best)
    print("narrow phase of ordinary and such pairs, us:", [round(x * 1e6, 1) for x in took])
    assert took[1] <= 40 * took[0]
