"""The four-wide box hierarchy of the candidate search at the edges of its
groups and levels, on boxes that FP32 cannot decide, and with both traversals
(a warp per row below 24,576 rows in 2D and 65,536 in 3D, a thread per row
from there on): candidate sets against brute force over the FP64 boxes with
the reference's strict test, rows in the same order from both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _elements(dim, n, rng, size):
    """n small simplices as a mesh of its own nodes."""
    c = rng.random((n, 1, dim))
    pos = (c + size * (rng.random((n, dim + 1, dim)) - 0.5)).reshape(-1, dim)
    return pos, np.arange(n * (dim + 1), dtype=np.int32).reshape(n, dim + 1)


def _rows(ctx, A, B):
    n = ctx.find_candidates(A, B)
    ip, ind = ctx.get_candidates(len(A[1]), n)
    return ip, ind


def _brute(A, B):
    va, vb = A[0][A[1]], B[0][B[1]]
    la, ha, lb, hb = va.min(1), va.max(1), vb.min(1), vb.max(1)
    for a in range(len(la)):
        yield np.flatnonzero(((ha[a] > lb) & (la[a] < hb)).all(1))


def _check(ctx, A, B):
    ip, ind = _rows(ctx, A, B)
    for a, ref in enumerate(_brute(A, B)):
        got = ind[ip[a]:ip[a + 1]]
        assert np.array_equal(np.sort(got), ref), a
    return ip, ind


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("nb", [1, 2, 4, 5, 16, 17, 63, 65, 256, 257, 1023, 1025, 4097])
def test_group_and_level_edges(gpu_ctx, dim, nb):
    rng = np.random.default_rng(nb)
    _check(gpu_ctx, _elements(dim, 300, rng, 0.3), _elements(dim, nb, rng, 0.1))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shift,scale,step", [
    (0.0, 1.0, 8), (-0.5, 1.0, 8),       # many equal coordinates: boxes that touch
    (1.0e6, 1.0, 8), (0.0, 1.0e6, 1000),  # boxes closer than FP32's spacing
    (0.0, 2.0 ** -140, 1 << 20),          # FP32 subnormals
    (3.0e38, 1.0e36, 64),                 # beyond FP32's range
])
def test_boxes_fp32_cannot_decide(gpu_ctx, dim, shift, scale, step):
    rng = np.random.default_rng(dim)
    A, B = _elements(dim, 400, rng, 0.2), _elements(dim, 700, rng, 0.2)
    A, B = ((np.round(m[0] * step) / step * scale + shift, m[1]) for m in (A, B))
    _check(gpu_ctx, A, B)


@pytest.mark.parametrize("dim,na", [(2, 24575), (2, 24576), (3, 65535), (3, 65536)])
def test_both_traversals_give_the_same_rows(gpu_ctx, dim, na):
    """Rows of a large A (around the line between the traversals) and of its
    first 3000 elements alone; long rows among them (more than 256)."""
    rng = np.random.default_rng(na)
    pos, en = _elements(dim, na, rng, 0.02)
    pos[:(dim + 1) * 5] = rng.random(((dim + 1) * 5, dim)) * 1.2
    B = _elements(dim, 5000, rng, 0.05)
    ip, ind = _rows(gpu_ctx, (pos, en), B)
    ips, inds = _check(gpu_ctx, (pos, en[:3000]), B)
    assert np.array_equal(ip[:3001], ips)
    assert np.array_equal(ind[:ips[-1]], inds)


@pytest.mark.parametrize("na", [1, 63, 65, 255, 257, 8191, 8193, 16385, 32768, 32769])
def test_row_offsets_at_the_scan_edges(gpu_ctx, na):
    """Row counts around a warp's rows, a tile and the one-block scan's limit;
    the offsets are whole numbers, compared exactly."""
    rng = np.random.default_rng(na)
    A, B = _elements(2, na, rng, 0.05), _elements(2, 40, rng, 0.2)
    ip, ind = _rows(gpu_ctx, A, B)
    va, vb = A[0][A[1]], B[0][B[1]]
    hit = ((va.max(1)[:, None] > vb.min(1)[None]) & (va.min(1)[:, None] < vb.max(1)[None])).all(2)
    assert np.array_equal(ip, np.concatenate([[0], np.cumsum(hit.sum(1))]))
    assert np.array_equal(np.sort(ind + 40 * np.repeat(np.arange(na), hit.sum(1))), np.flatnonzero(hit))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("nb", [2047, 2049, 2048 * 8 + 1, 2048 * 9, 2048 * 17 + 5])
def test_sort_look_back_edges(gpu_ctx, dim, nb):
    """Trees over one to 18 blocks of the sort, whose look-back takes eight
    blocks at a time; a third of the keys equal."""
    rng = np.random.default_rng(nb)
    pos, en = _elements(dim, nb, rng, 0.05)
    pos[: (dim + 1) * (nb // 3)] = np.tile(pos[: dim + 1], (nb // 3, 1))
    _check(gpu_ctx, _elements(dim, 60, rng, 0.1), (pos, en))


@pytest.mark.parametrize("dim", [2, 3])
def test_fill_row_lengths(gpu_ctx, dim):
    """Rows of 0 to 300 candidates side by side, in the order of the target's
    elements along a line: edges of the lanes that copy a row and of the row
    cache."""
    nb = 300
    lens = np.array([0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 255, 256, 257, 300, 3, 0, 12] * 4 + [5])
    e = np.vstack([np.zeros((1, dim)), np.eye(dim)])
    b = e[None] * 0.5
    b = np.repeat(b, nb, 0)
    b[:, :, 0] += np.arange(nb)[:, None]
    a = np.repeat(e[None], len(lens), 0)
    a[:, :, 0] = a[:, :, 0] * np.maximum(lens - 0.25, 0.25)[:, None] - np.where(lens > 0, 0.0, 1.0)[:, None]
    A = (a.reshape(-1, dim), np.arange(len(lens) * (dim + 1), dtype=np.int32).reshape(-1, dim + 1))
    B = (b.reshape(-1, dim), np.arange(nb * (dim + 1), dtype=np.int32).reshape(-1, dim + 1))
    ip, _ = _check(gpu_ctx, A, B)
    assert np.array_equal(np.diff(ip), lens)
