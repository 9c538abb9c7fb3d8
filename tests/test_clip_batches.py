"""The tet clippers (k_clip_tets_bf and k_clip_tets_ix) at the edges of their batches
and on inputs outside the ordinary: against the one-launch clipper that
batches below 2048 pairs take, and the P1 mass blocks against the oracle.
Both sides run the same operations in the same order, so every comparison is
exact."""
import numpy as np
import pytest
import torch

import libsupermesh_b200 as lsm
from libsupermesh_b200 import meshes as M

pytestmark = pytest.mark.gpu


def _pairs(n, seed):
    """n pairs of overlapping tets: runs of 1 to 40 pairs with the same A,
    among them A inside B, A equal to B, shared faces and vertices, and
    elements with a repeated vertex."""
    rng = np.random.default_rng(seed)
    a = np.empty((n, 4, 3))
    b = rng.random((n, 4, 3))
    i = 0
    while i < n:
        k = int(rng.integers(1, 41))
        a[i:i + k] = rng.random((4, 3))
        i += k
    kind = rng.integers(0, 12, n)
    a[kind == 0] = 0.4 + 0.01 * rng.random((int((kind == 0).sum()), 4, 3))
    b[kind == 0] = np.array([[-2, -2, -2], [5, 0, 0], [0, 5, 0], [0, 0, 5]])
    b[kind == 1] = a[kind == 1]
    b[kind == 2, :3] = a[kind == 2, :3]
    b[kind == 3, 2] = a[kind == 3, 1]
    b[kind == 4, 3] = b[kind == 4, 0]
    a[kind == 5, 3] = a[kind == 5, 1]
    return a, b


def _small(ctx, a, b):
    """The same pairs through the one-launch clipper, 2000 at a time."""
    r = [ctx.intersect_pairs(3, a[i:i + 2000], b[i:i + 2000], want_elems=True) for i in range(0, len(a), 2000)]
    return [np.concatenate(x) for x in zip(*r)]


def _same(got, ref):
    assert np.array_equal(got[1], ref[1])
    assert np.array_equal(got[0], ref[0])
    if got[2] is not None:
        used = np.arange(81)[None] < got[1][:, None]
        assert np.array_equal(got[2][used], ref[2][used])


@pytest.mark.parametrize("n", [2048, 2049, 2079, 2081, 2111, 2113, 5003])
@pytest.mark.parametrize("elems", [False, True])
def test_batches_match_one_launch_clipper(gpu_ctx, n, elems):
    a, b = _pairs(n, n)
    _same(gpu_ctx.intersect_pairs(3, a, b, want_elems=elems), _small(gpu_ctx, a, b))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e200])
def test_coordinates_that_are_not_finite(gpu_ctx, value):
    """Some vertices of A with a coordinate that is not finite, or whose
    products overflow."""
    a, b = _pairs(2300, 5)
    rng = np.random.default_rng(6)
    rows = rng.choice(len(a), 700, replace=False)
    a[rows, rng.integers(0, 4, 700), rng.integers(0, 3, 700)] = value
    _same(gpu_ctx.intersect_pairs(3, a, b, want_elems=True), _small(gpu_ctx, a, b))


@pytest.mark.parametrize("na,nb,ja,jb,scale", [
    (4, 4, 0.0, 0.0, 1.0),       # identical regular meshes: vertices and edges coincide
    (4, 6, 0.0, 0.25, 1.0),
    (7, 5, 0.25, 0.25, 2.0 ** -250),  # far from 1 in both directions
    (5, 6, 0.2, 0.0, 2.0 ** 100),
])
def test_p1_blocks_match_oracle(gpu_ctx, oracle_mod, na, nb, ja, jb, scale):
    A, B = M.grid3d(na, 3, ja), M.grid3d(nb, 2, jb)
    A, B = (A[0] * scale, A[1]), (B[0] * scale, B[1])
    u, v = np.cos(np.arange(len(A[0]))), np.sin(np.arange(len(B[0])))
    val, blocks = gpu_ctx.p1_mass(A, B, u, v, want_blocks=True)
    ip, ind = gpu_ctx.get_candidates(len(A[1]), len(blocks))
    _, _, ref = oracle_mod.p1_mass(3, A, B, ip, ind, u, v, want_blocks=True)
    assert np.array_equal(blocks, ref.reshape(blocks.shape))


@pytest.mark.parametrize("exponent", [-40, 300, 339, 340, 341, 342, 343, 344, 346, 352])
def test_pairs_whose_projections_overflow(gpu_ctx, exponent):
    """Explicit pairs at the scales where products of three coordinates leave
    the range: the second early-out's projections then prove nothing."""
    a, b = _pairs(4001, 12)
    a, b = a * 2.0 ** exponent, b * 2.0 ** exponent
    (m, k, _), (rm, rk, _) = gpu_ctx.intersect_pairs(3, a, b), _small(gpu_ctx, a, b)
    assert (rk > 0).sum() > 100
    assert np.array_equal(k, rk)
    assert np.array_equal(m, rm, equal_nan=True)


@pytest.mark.parametrize("exponent", [343, 344, 345, 348, 400, 500])
def test_volumes_that_overflow(gpu_ctx, exponent):
    """Coordinates whose volumes' products overflow: a kept tet of NaN volume
    counts (in either clipper; the binned order takes the depth-first one) and
    makes its pair's measure and every entry of its mass block NaN; the
    elements' two passes agree on the count."""
    A, B = M.grid3d(4, 3, 0.2), M.grid3d(5, 2, 0.2)
    A, B = (A[0] * 2.0 ** exponent, A[1]), (B[0] * 2.0 ** exponent, B[1])
    cand = gpu_ctx.find_candidates(A, B)
    gpu_ctx.clip_candidates()
    m, k = gpu_ctx.pair_results(cand)
    lsm.set_option("tet_schedule", 2)
    try:
        gpu_ctx.clip_candidates()
        rm, rk = gpu_ctx.pair_results(cand)
    finally:
        lsm.set_option("tet_schedule", 0)
    assert np.array_equal(k, rk)
    assert np.array_equal(m, rm, equal_nan=True)
    _, blocks = gpu_ctx.p1_mass(A, B, want_blocks=True)
    assert np.isnan(m).any() == (exponent > 343)
    assert np.isnan(blocks[np.isnan(m)]).all()
    # the emitting pass, into arrays of one element more than the count
    _, off, _, pa, _ = gpu_ctx.supermesh_elements(A, B)
    assert np.array_equal(np.diff(off), k)
    n, dev = int(off[-1]), {"device": "cuda"}
    out = {"cand_capacity": cand, "elem_capacity": n + 1, "elem_offset": torch.zeros(cand + 1, dtype=torch.int64, **dev),
           "elems": torch.full((n + 1, 4, 3), 7.0, dtype=torch.float64, **dev),
           "parent_a": torch.full((n + 1,), -7, dtype=torch.int64, **dev),
           "parent_b": torch.full((n + 1,), -7, dtype=torch.int64, **dev)}
    gpu_ctx.supermesh_elements_device(*(tuple(torch.from_numpy(x).cuda() for x in m_) for m_ in (A, B)), out)
    torch.cuda.synchronize()
    assert np.array_equal(out["parent_a"][:n].cpu().numpy(), pa)
    assert (out["elems"][n] == 7.0).all() and out["parent_a"][n] == -7 and out["parent_b"][n] == -7


@pytest.mark.parametrize("exponent", [342, 343, 344, 345, 348, 352, 400, 500])
def test_volumes_that_overflow_against_one_launch(gpu_ctx, exponent):
    """The keep test's shortcut (vertex-1 volume) where it and its bound are
    infinite: the vertex-4 volume decides, as in the one-launch clipper."""
    A, B = M.grid3d(4, 3, 0.2), M.grid3d(5, 2, 0.2)
    A, B = (A[0] * 2.0 ** exponent, A[1]), (B[0] * 2.0 ** exponent, B[1])
    cand = gpu_ctx.find_candidates(A, B)
    gpu_ctx.clip_candidates()
    ip, ind = gpu_ctx.get_candidates(len(A[1]), cand)
    m, k = gpu_ctx.pair_results(cand)
    ra = np.repeat(np.arange(len(A[1])), np.diff(ip))
    rm, rk, _ = _small(gpu_ctx, A[0][A[1]][ra], B[0][B[1]][ind])
    assert np.array_equal(k, rk)
    assert np.array_equal(m, rm, equal_nan=True)


@pytest.mark.parametrize("value", [None, np.nan, np.inf, 1e200])
def test_tet_hexahedron_batches(gpu_ctx, value):
    """The depth-first clipper's split table, six planes: batches of 2048 and
    more against the one-launch clipper, special tets and (value) coordinates
    that are not finite among them."""
    a, b = _pairs(2307, 9)
    corner = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]], float)
    lo, hi = b.min(1), b.max(1)
    h = lo[:, None] + corner[None] * (hi - lo)[:, None]
    h[::5] = np.round(a[::5, :1] * 4) / 4 + corner[None] * 0.5  # faces through vertices' neighbourhoods
    a[::5] = np.round(a[::5] * 8) / 8
    if value is not None:
        rng = np.random.default_rng(6)
        rows = rng.choice(len(a), 700, replace=False)
        a[rows, rng.integers(0, 4, 700), rng.integers(0, 3, 700)] = value
    got = gpu_ctx.intersect_pairs_mixed(lsm.PAIR_TET_HEX, a, h)
    ref = [gpu_ctx.intersect_pairs_mixed(lsm.PAIR_TET_HEX, a[i:i + 1000], h[i:i + 1000])[:2] for i in (0, 1000, 2000)]
    assert np.array_equal(got[1], np.concatenate([r[1] for r in ref]))
    assert np.array_equal(got[0], np.concatenate([r[0] for r in ref]))


@pytest.mark.parametrize("shift", [0.0, 1.0e4])
def test_pairs_near_touching_across_a_face_of_a(gpu_ctx, shift):
    """B on the far side of a face of A at gaps through zero and the rounding
    margins: the second early-out of the explicit pairs must never drop a
    pair with output."""
    rng = np.random.default_rng(11)
    n = 4000
    a = rng.random((n, 4, 3))
    nrm = np.cross(a[:, 1] - a[:, 0], a[:, 2] - a[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    nrm *= -np.sign(((a[:, 3] - a[:, 0]) * nrm).sum(1))[:, None]  # outwards
    gap = np.concatenate([[0.0], 10.0 ** -np.arange(3, 17), -10.0 ** -np.arange(3, 17)])[rng.integers(0, 29, n)]
    base = a[:, 0] + 0.3 * (a[:, 1] - a[:, 0]) + 0.3 * (a[:, 2] - a[:, 0]) + gap[:, None] * nrm
    u = a[:, 1] - a[:, 0]
    v = np.cross(nrm, u)
    b = np.stack([base, base + 0.4 * u, base + 0.4 * v, base + 0.5 * nrm + 0.1 * u], axis=1)
    _same(gpu_ctx.intersect_pairs(3, a + shift, b + shift, want_elems=True), _small(gpu_ctx, a + shift, b + shift))


def _soup(kind, n):
    """Two meshes of n tets of their own nodes."""
    rng = np.random.default_rng(n)
    a, b = (rng.random((n, 1, 3)) + 0.35 * rng.random((n, 4, 3)) for _ in range(2))
    if kind == "lattice":  # vertices on planes, shared and parallel faces
        a, b = np.round(a * 16) / 16, np.round(b * 16) / 16
    elif kind == "inside":
        a[::2] = b[::2].mean(1, keepdims=True) + 1e-3 * (a[::2] - a[::2, :1])
    elif kind == "degenerate":
        a[::3, 2], b[::5, 1] = a[::3, 1], b[::5, 0]
    elif kind == "large":  # bounds that overflow
        a[::3] *= 1e200
        b[::4] *= 1e200
    elif kind == "infinite":
        a[::4, 1, 0] = np.inf
        a[1::4, 1:, 2] = -np.inf
        b[1::3, :, 0] = [np.inf, 0, 1, -np.inf]
    en = np.arange(4 * n, dtype=np.int32).reshape(n, 4)
    return (a.reshape(-1, 3), en), (b.reshape(-1, 3), en)


@pytest.mark.parametrize("kind", ["plain", "lattice", "inside", "degenerate", "large", "infinite"])
@pytest.mark.parametrize("n", [33, 400])
def test_mesh_early_outs_match_one_launch_clipper(gpu_ctx, kind, n):
    """What the early-out pass rejects or settles, against clipping every
    candidate."""
    A, B = _soup(kind, n)
    cand = gpu_ctx.find_candidates(A, B)
    gpu_ctx.clip_candidates()
    ip, ind = gpu_ctx.get_candidates(n, cand)
    m, k = gpu_ctx.pair_results(cand)
    rm, rk, _ = _small(gpu_ctx, A[0][A[1]][np.repeat(np.arange(n), np.diff(ip))], B[0][B[1]][ind])
    assert np.array_equal(k, rk)
    assert np.array_equal(m, rm, equal_nan=True)
