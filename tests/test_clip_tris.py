"""The converged triangle clip of the mesh paths (clip_tri_c) against the
walking one that explicit pairs take (clip_tri): the same operations on the
same values, so measures, counts and triangles are compared exactly; and
u^T M v by triangles against the assembled blocks."""
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
