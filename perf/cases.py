"""Performance cases: the work a program hands to this library, with sizes.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call
(meshes, fields and output arrays on the GPU, a Context), ``run(state)`` is one
pass through the public entry points, ``work(case)`` the bytes and operations
one pass cannot do without, and ``exact(case, seed)`` the results in 64 bits by
plain torch, where they have such values.

Operations (``case["op"]``):

* ``supermesh``  candidate search, clipping, per-element measures and totals of
                 one mesh pair (``Context.supermesh``);
* ``csr``        the same with the candidate CSR and each candidate's measure
                 and count (``Context.supermesh_out``);
* ``elements``   the supermesh's simplices with their parents
                 (``Context.supermesh_elements_device``);
* ``p1``         the P1-P1 mixed mass product u^T M v (``Context.p1_mass``);
* ``pairs``      explicit element pairs (``Context.intersect_pairs_device``);
* ``batched``    many uneven mesh pairs with every per-candidate result and
                 P1 block (``Context.supermesh_batched_pairs``);
* ``dropin``     the reference's own C API on host arrays: one search, then one
                 call per candidate.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libsupermesh_b200 as lsm
from libsupermesh_b200 import meshes


def listed():
    return [
        # The plain 2D supermesh at its usual size (10,658 x 20,000 triangles):
        # a time step's projection between two small meshes, where launches
        # and waits count.
        {"name": "tri_small", "op": "supermesh", "dim": 2, "na": 73, "nb": 100, "jitter": 0.3, "map": "none",
         "index_bytes": 4},
        # A small 3D pair (6,000 x 10,368 tets), same use.
        {"name": "tet_small", "op": "supermesh", "dim": 3, "na": 10, "nb": 12, "jitter": 0.25, "map": "none",
         "index_bytes": 4},
        # The large 2D workload: 1.2 M triangles, rotated and clamped, over 2.1 M.
        {"name": "tri_large_rot", "op": "supermesh", "dim": 2, "na": 777, "nb": 1024, "jitter": 0.3, "map": "rot7",
         "index_bytes": 4},
        # The plain 3D supermesh (118,098 x 196,608 tets) with all that a caller
        # of set_input / get_output / intersect reads back, kept on the GPU;
        # 64-bit element lists, the C API's own type.
        {"name": "tet_csr", "op": "csr", "dim": 3, "na": 27, "nb": 32, "jitter": 0.25, "map": "none",
         "index_bytes": 8},
        # The headline workload: about 1.0 M x 0.8 M graded tets.
        {"name": "tet_graded", "op": "supermesh", "dim": 3, "na": 55, "nb": 51, "jitter": 0.2, "map": "square",
         "index_bytes": 4},
        # The supermesh itself, for callers that integrate over it.
        {"name": "tet_elements", "op": "elements", "dim": 3, "na": 27, "nb": 32, "jitter": 0.25, "map": "none",
         "index_bytes": 4},
        # P1-P1 projection's product in 2D (720,000 x 1,280,000 triangles) ...
        {"name": "p1_tri", "op": "p1", "dim": 2, "na": 600, "nb": 800, "jitter": 0.3, "map": "none",
         "index_bytes": 4},
        # ... and in 3D.
        {"name": "p1_tet", "op": "p1", "dim": 3, "na": 27, "nb": 32, "jitter": 0.25, "map": "none",
         "index_bytes": 4},
        # Callers with their own search hand over element pairs: simplices ...
        {"name": "pairs_tet", "op": "pairs", "kind": "tet", "na": 27, "nb": 32, "n": 1 << 20},
        # ... and tetrahedra against hexahedra.
        {"name": "pairs_tet_hex", "op": "pairs", "kind": "tet_hex", "na": 27, "nb": 32, "n": 1 << 19},
        # Many uneven mesh pairs at once (half 2D, half 3D, 1e3 to 1e5 elements
        # each) with every result and the mass blocks.
        {"name": "batched", "op": "batched", "count": 16, "emin": 1e3, "emax": 1e5},
        # A C or Fortran caller's loop over the reference's API: the smallest
        # calls (a search over host arrays, 64 candidate pairs one by one).
        {"name": "dropin", "op": "dropin", "dim": 3, "na": 5, "nb": 6, "calls": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["supermesh", "supermesh", "supermesh", "csr", "elements", "p1", "pairs", "batched", "dropin"])
    if op in ("supermesh", "csr", "elements", "p1"):
        dim = rng.choice([2, 3])
        # grid sizes up to the listed ones; the two meshes within a factor of
        # two of one another, as meshes of one domain are
        hi = {"supermesh": (1024, 52), "csr": (600, 30), "elements": (400, 28), "p1": (700, 27)}[op][dim - 2]
        na = _log_int(rng, 24 if dim == 2 else 5, hi)
        nb = max(3, min(int(hi * 1.2), int(round(na * math.exp(rng.uniform(math.log(0.6), math.log(1.6)))))))
        mp = "none" if op == "p1" else rng.choice(["none", "square", "rot7"] if dim == 2 else ["none", "square"])
        return {"op": op, "dim": dim, "na": na, "nb": nb, "jitter": rng.choice([0.1, 0.2, 0.3 if dim == 2 else 0.25]),
                "map": mp, "index_bytes": rng.choice([4, 8])}
    if op == "pairs":
        kind = rng.choice(["tri", "tet", "tri_quad", "quad_quad", "tet_hex", "hex_hex"])
        na = rng.randint(7, 60)
        return {"op": op, "kind": kind, "na": na, "nb": max(5, int(na * rng.uniform(0.6, 1.6))),
                "n": _log_int(rng, 1000, 1 << (17 if kind == "hex_hex" else 20))}
    if op == "batched":
        return {"op": op, "count": 2 * rng.randint(2, 10), "emin": 1e3, "emax": _log_int(rng, 3000, 80000)}
    na = rng.randint(4, 9)
    return {"op": "dropin", "dim": rng.choice([2, 3]), "na": na, "nb": na + rng.randint(-1, 3), "calls": rng.randint(16, 128)}


# --- inputs -------------------------------------------------------------------

_MAPS = {"none": None, "square": meshes.grade_square, "rot7": None}


def _mesh(dim, n, seed, jitter, mp):
    grid = meshes.grid2d if dim == 2 else meshes.grid3d
    return grid(n, seed, jitter, _MAPS[mp])


def _mesh_pair(case, seed):
    """Target A and source B of one case (numpy, int32 lists)."""
    A = _mesh(case["dim"], case["na"], 2 * seed + 1, case.get("jitter", 0.25), case.get("map", "none"))
    B = _mesh(case["dim"], case["nb"], 2 * seed, case.get("jitter", 0.25), case.get("map", "none"))
    if case.get("map") == "rot7":
        A = (meshes.rotate_clamp(A[0], 7.0), A[1])
    return A, B


def _capacity(case):
    """Room for a mesh pair's candidates: the usual count and a third, as a
    caller that keeps its arrays from step to step allocates them."""
    return 64 + int(1.33 * _candidates(case["dim"], case["na"], case["nb"]))


def _batch_grids(case):
    """(dim, na, nb) of each mesh pair: element counts log-uniform, half 2D."""
    rs = np.random.RandomState(case["count"] + int(case["emax"]))
    lo, hi = math.log(case["emin"]), math.log(case["emax"])
    grids = []
    for i in range(case["count"]):
        dim = 2 if i < case["count"] // 2 else 3
        ea, eb = np.exp(rs.uniform(lo, hi, 2))
        k = 2 if dim == 2 else 6
        grids.append((dim, max(1, round((ea / k) ** (1 / dim))), max(1, round((eb / k) ** (1 / dim)))))
    return grids


def _fields(case, seed):
    """Coefficients (constant, then one per axis) of the two affine fields."""
    rs = np.random.RandomState(seed & 0x7FFFFFFF)
    return rs.uniform(-1.0, 1.0, (2, 1 + case["dim"]))


_QUAD = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], dtype=np.float64)
_HEX = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]],
                dtype=np.float64)  # Gmsh node order


def _cells(n, dim):
    """The cells of a regular n^dim grid as quadrilaterals or hexahedra, cell
    (i, j[, k]) at i + n (j + n k)."""
    ax = np.meshgrid(*([np.arange(n)] * dim), indexing="ij")
    base = np.stack([x.ravel() for x in reversed(ax)], axis=1).astype(np.float64)
    return (base[:, None, :] + (_QUAD if dim == 2 else _HEX)[None]) / n


def _element_pairs(case, seed):
    """n element pairs as a caller's own search gives them: A's elements in
    order, B's near them (in a cell that A's box reaches)."""
    kind, na, nb, n = case["kind"], case["na"], case["nb"], case["n"]
    dim = 2 if kind in ("tri", "tri_quad", "quad_quad") else 3
    rs = np.random.RandomState(seed & 0x7FFFFFFF)
    if kind in ("quad_quad", "hex_hex"):
        th = math.radians(20.0)  # cells turned against B's
        ea = _cells(na, dim) - 0.5
        x, y = ea[..., 0].copy(), ea[..., 1].copy()
        ea[..., 0], ea[..., 1] = (math.cos(th) * x - math.sin(th) * y) * 0.7, (math.sin(th) * x + math.cos(th) * y) * 0.7
        ea = ea + 0.5 + rs.uniform(-0.02, 0.02, dim)
    else:
        pos, en = _mesh(dim, na, 2 * seed + 1, 0.3 if dim == 2 else 0.25, "none")
        ea = pos[en]
    if kind in ("tri", "tet"):
        pos, en = _mesh(dim, nb, 2 * seed, 0.3 if dim == 2 else 0.25, "none")
        eb = pos[en]
    else:
        eb = _cells(nb, dim)
    per_cell = len(eb) // nb ** dim
    ia = (np.arange(n) * len(ea)) // n if n >= len(ea) else np.sort(rs.choice(len(ea), n, replace=False))
    a = ea[ia]
    lo, hi = a.min(axis=1), a.max(axis=1)
    cell = np.clip(((lo + rs.uniform(0, 1, lo.shape) * (hi - lo)) * nb).astype(np.int64), 0, nb - 1)
    ic = cell[:, dim - 1]
    for c in range(dim - 2, -1, -1):
        ic = ic * nb + cell[:, c]
    b = eb[ic * per_cell + (rs.randint(0, per_cell, n) if per_cell > 1 else 0)]
    return dim, np.ascontiguousarray(a.reshape(n, -1)), np.ascontiguousarray(b.reshape(n, -1))


def _device_mesh(m, index_bytes):
    en = torch.from_numpy(m[1]).cuda()
    return torch.from_numpy(m[0]).cuda(), (en.long() if index_bytes == 8 else en)


_KINDS = {"tri": None, "tet": None, "tri_quad": lsm.PAIR_TRI_QUAD, "quad_quad": lsm.PAIR_QUAD_QUAD,
          "tet_hex": lsm.PAIR_TET_HEX, "hex_hex": lsm.PAIR_HEX_HEX}


def prepare(case, seed):
    op = case["op"]
    s = {"op": op}
    if op == "dropin":
        A, B = _mesh_pair(case, seed)
        s["A"] = (A[0], A[1].astype(np.int64))
        s["B"] = (B[0], B[1].astype(np.int64))
        s["clip"] = lsm.intersect_tris_real if case["dim"] == 2 else lsm.intersect_tets_real
        shape = (lsm.TRI_BUF_SIZE, 3, 2) if case["dim"] == 2 else (lsm.TET_BUF_SIZE, 4, 3)
        s["elems"] = np.zeros((case["calls"],) + shape)
        s["indices"] = np.zeros(_capacity(case), np.int64)
        return s
    s["ctx"] = ctx = lsm.Context(torch.cuda.current_device())
    if op == "pairs":
        dim, a, b = _element_pairs(case, seed)
        n = case["n"]
        s.update(a=torch.from_numpy(a).cuda(), b=torch.from_numpy(b).cuda(), dim=dim, kind=_KINDS[case["kind"]],
                 measure=torch.zeros(n, dtype=torch.float64, device="cuda"),
                 n_out=torch.zeros(n, dtype=torch.int32, device="cuda"))
    elif op == "batched":
        host, cap = [], 0
        for i, (dim, na, nb) in enumerate(_batch_grids(case)):
            c = {"dim": dim, "na": na, "nb": nb, "jitter": 0.3 if dim == 2 else 0.25}
            host.append(_mesh_pair(c, 1000 * seed + i))
            cap += _capacity(c)
        s["pairs"] = [tuple(_device_mesh(m, 4) for m in AB) for AB in host]
        n = case["count"]
        rows = sum(len(A[1]) + 1 for A, _ in host)
        i64 = {"dtype": torch.int64, "device": "cuda"}
        s["out"] = {"totals": np.zeros(n), "n_candidates": np.zeros(n, np.int64), "n_intersecting": np.zeros(n, np.int64),
                    "cand_offset": np.zeros(n, np.int64), "total_candidates": np.zeros(1, np.int64),
                    "p1_offset": np.zeros(n, np.int64), "capacity": cap,
                    "ind_ptr": torch.zeros(rows, **i64), "indices": torch.zeros(cap, **i64),
                    "pair_measure": torch.zeros(cap, dtype=torch.float64, device="cuda"),
                    "pair_n_out": torch.zeros(cap, dtype=torch.int32, device="cuda"),
                    "p1_blocks": torch.zeros(16 * cap, dtype=torch.float64, device="cuda")}
    else:
        A, B = _mesh_pair(case, seed)
        s["A"], s["B"] = (_device_mesh(m, case["index_bytes"]) for m in (A, B))
        f64 = {"dtype": torch.float64, "device": "cuda"}
        i64 = {"dtype": torch.int64, "device": "cuda"}
        torch.cuda.synchronize()
        if op == "supermesh":
            s["measure"] = torch.zeros(len(A[1]), **f64)
        elif op == "csr":
            n = _capacity(case)
            s["out"] = {"elem_measure": torch.zeros(len(A[1]), **f64), "ind_ptr": torch.zeros(len(A[1]) + 1, **i64),
                        "indices": torch.zeros(n, **i64), "pair_measure": torch.zeros(n, **f64),
                        "pair_n_out": torch.zeros(n, dtype=torch.int32, device="cuda"), "capacity": n}
        elif op == "elements":
            nc = _capacity(case)
            ne = int((0.95 if case["dim"] == 2 else 3.0) * nc)
            loc = case["dim"] + 1
            s["out"] = {"cand_capacity": nc, "elem_capacity": ne, "elem_offset": torch.zeros(nc + 1, **i64),
                        "elems": torch.zeros((ne, loc, case["dim"]), **f64),
                        "parent_a": torch.zeros(ne, **i64), "parent_b": torch.zeros(ne, **i64)}
        else:
            fu, fv = _fields(case, seed)
            s["u"] = torch.from_numpy(fu[0] + A[0] @ fu[1:]).cuda()
            s["v"] = torch.from_numpy(fv[0] + B[0] @ fv[1:]).cuda()
    torch.cuda.synchronize()
    return s


def _counts(st):
    return {"n_candidates": st.n_candidates, "n_intersecting": st.n_intersecting, "n_out": st.n_out_simplices,
            "total": st.total_measure}


def run(s):
    op = s["op"]
    if op == "supermesh":
        st, em = s["ctx"].supermesh(s["A"], s["B"], elem_measure=True, on_device=True, out=s["measure"])
        return dict(_counts(st), elem_measure=em)
    if op == "csr":
        st, n = s["ctx"].supermesh_out(s["A"], s["B"], s["out"], on_device=True)
        o = s["out"]
        return dict(_counts(st), n=n, elem_measure=o["elem_measure"], ind_ptr=o["ind_ptr"], indices=o["indices"],
                    pair_measure=o["pair_measure"], pair_n_out=o["pair_n_out"])
    if op == "elements":
        st, nc, ne = s["ctx"].supermesh_elements_device(s["A"], s["B"], s["out"])
        o = s["out"]
        return dict(_counts(st), nc=nc, ne=ne, elem_offset=o["elem_offset"], elems=o["elems"],
                    parent_a=o["parent_a"], parent_b=o["parent_b"])
    if op == "p1":
        return {"integral": s["ctx"].p1_mass(s["A"], s["B"], s["u"], s["v"], on_device=True)[0]}
    if op == "pairs":
        s["ctx"].intersect_pairs_device(s["a"], s["b"], s["measure"], s["n_out"], dim=s["dim"], kind=s["kind"])
        return {"measure": s["measure"], "n_out": s["n_out"]}
    if op == "batched":
        o = s["out"]
        s["ctx"].supermesh_batched_pairs(s["pairs"], capacity=o["capacity"], on_device=True, out=o, p1_blocks=True)
        return {k: o[k] for k in ("totals", "n_candidates", "n_intersecting", "cand_offset", "ind_ptr", "indices",
                                  "pair_measure", "pair_n_out", "p1_offset", "p1_blocks")}
    A, B = s["A"], s["B"]
    ind_ptr, indices = lsm.tree_intersection_finder(*A, *B)
    s["indices"][:len(indices)] = indices
    n_out, a = [], 0
    for p in range(len(s["elems"])):
        while ind_ptr[a + 1] <= p:
            a += 1
        got = s["clip"](A[0][A[1][a]], B[0][B[1][indices[p]]])
        s["elems"][p, :len(got)] = got
        n_out.append(len(got))
    return {"ind_ptr": ind_ptr, "indices": s["indices"], "elems": s["elems"], "n_out": np.array(n_out)}


# --- what a pass cannot do without --------------------------------------------

def _mesh_bytes(dim, n, index_bytes):
    nel = (2 if dim == 2 else 6) * n ** dim
    return 8 * dim * (n + 1) ** dim + index_bytes * (dim + 1) * nel


def _candidates(dim, na, nb):
    """Box-overlapping pairs of two jittered grids (boxes a little wider than a cell)."""
    f, k = (1.092, 2) if dim == 2 else (1.107, 6)
    return (k * na ** dim) * (k * nb ** dim) * min(1.0, f * (1 / na + 1 / nb)) ** dim


# operations of the reference algorithm: per candidate pair (2D, 3D), and of
# the quadrature per output simplex, of which a candidate has 0.92 or 2.54
_CLIP_FLOPS = {2: 84, 3: 413}
_P1_FLOPS = {2: 0.92 * 180, 3: 2.54 * 460}


def work(case):
    op = case["op"]
    if op == "pairs":
        per_a, per_b = {"tri": (6, 6), "tet": (12, 12), "tri_quad": (6, 8), "quad_quad": (8, 8), "tet_hex": (12, 24),
                        "hex_hex": (24, 24)}[case["kind"]]
        flops = {"tri": 130, "tet": 800, "tri_quad": 160, "quad_quad": 200, "tet_hex": 1500, "hex_hex": 6000}
        return {"bytes": case["n"] * (8 * (per_a + per_b) + 12), "flops": case["n"] * flops[case["kind"]]}
    if op == "batched":
        b = f = 0.0
        for dim, na, nb in _batch_grids(case):
            c = _candidates(dim, na, nb)
            b += _mesh_bytes(dim, na, 4) + _mesh_bytes(dim, nb, 4) + 8 * (2 if dim == 2 else 6) * na ** dim
            b += c * (20 + 8 * (dim + 1) ** 2)
            f += c * (_CLIP_FLOPS[dim] + _P1_FLOPS[dim])
        return {"bytes": b, "flops": f}
    dim, na, nb = case["dim"], case["na"], case["nb"]
    nel_a = (2 if dim == 2 else 6) * na ** dim
    cand = _candidates(dim, na, nb)
    ib = case.get("index_bytes", 8)
    b = _mesh_bytes(dim, na, ib) + _mesh_bytes(dim, nb, ib)
    f = cand * _CLIP_FLOPS[dim]
    if op == "supermesh":
        b += 8 * nel_a
    elif op == "csr":
        b += 16 * nel_a + 20 * cand
    elif op == "elements":
        b += 8 * cand + (0.92 if dim == 2 else 2.54) * cand * (8 * dim * (dim + 1) + 16)
    elif op == "p1":
        b += 8 * ((na + 1) ** dim + (nb + 1) ** dim)
        f += cand * _P1_FLOPS[dim]
    else:
        per = 8 * dim * (dim + 1)
        b += 8 * nel_a + 8 * cand + case["calls"] * 4 * per
        f = case["calls"] * _CLIP_FLOPS[dim]
    return {"bytes": b, "flops": f}


# --- results in 64 bits ---------------------------------------------------------

def _measures(t):
    """Measures of simplices t [n][dim + 1][dim]."""
    e = t[:, 1:] - t[:, :1]
    return torch.linalg.det(e).abs() / (2 if t.shape[2] == 2 else 6)


def _simplices(v, dim):
    """Decomposition of elements [n][nodes][dim] into simplices [k][n][dim + 1][dim]."""
    nodes = v.shape[1]
    if nodes == dim + 1:
        return v[None]
    if dim == 2:
        split = [(0, 1, 2), (0, 2, 3)]
    else:  # the six tets around the diagonal 0-6
        split = [(0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6)]
    return torch.stack([v[:, list(s)] for s in split])


def _half_spaces(v, dim):
    """Faces of convex elements [n][nodes][dim] as (normals, points), negative inside."""
    nodes = v.shape[1]
    if dim == 2:
        faces = [(i, (i + 1) % nodes) for i in range(nodes)]
    elif nodes == 4:
        faces = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]
    else:
        faces = [(0, 1, 2), (4, 5, 6), (0, 1, 5), (1, 2, 6), (2, 3, 7), (3, 0, 4)]
    mid = v.mean(dim=1)
    for f in faces:
        p = v[:, f[0]]
        if dim == 2:
            d = v[:, f[1]] - p
            nrm = torch.stack([d[:, 1], -d[:, 0]], dim=1)
        else:
            nrm = torch.linalg.cross(v[:, f[1]] - p, v[:, f[2]] - p)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        nrm = torch.where(((mid - p) * nrm).sum(1, keepdim=True) > 0, -nrm, nrm)
        yield nrm, p


def _clip(t, d):
    """Simplices t [n][dim + 1][dim] cut to the side d <= 0 of a plane (d
    [n][dim + 1]): the pieces and their rows in t."""
    dim = t.shape[2]
    d, at = d.sort(dim=1)
    t = t.gather(1, at[..., None].expand_as(t))
    neg = (d <= 0).sum(1)
    row = torch.arange(len(t), device=t.device)

    def cut(k, i, j):  # the point between vertices i (inside) and j of the simplices k
        w = d[k, i] / (d[k, i] - d[k, j])
        return t[k, i] + w[:, None] * (t[k, j] - t[k, i])

    out = [t[neg == dim + 1]]
    rows = [row[neg == dim + 1]]
    for m in range(1, dim + 1):
        k = row[neg == m]
        v = [t[k, i] for i in range(dim + 1)]
        if m == 1:
            pieces = [[v[0]] + [cut(k, 0, j) for j in range(1, dim + 1)]]
        elif m == dim:  # a prism on the inner face
            top = [cut(k, i, dim) for i in range(dim)]
            pieces = [v[i:dim] + top[: i + 1] for i in range(dim)]
        else:  # 3D, two inside
            a, b, c, e = cut(k, 0, 2), cut(k, 0, 3), cut(k, 1, 2), cut(k, 1, 3)
            pieces = [[v[0], a, b, e], [v[0], a, c, e], [v[0], v[1], c, e]]
        for p in pieces:
            out.append(torch.stack(p, dim=1))
            rows.append(k)
    return torch.cat(out), torch.cat(rows)


def _pair_measures(a, b, dim):
    """Measure of the intersection of each pair of convex elements."""
    n = len(a)
    total = torch.zeros(n, dtype=torch.float64, device=a.device)
    planes = list(_half_spaces(b, dim))
    for t in _simplices(a, dim):
        of = torch.arange(n, device=a.device)
        for nrm, p in planes:
            d = ((t - p[of][:, None]) * nrm[of][:, None]).sum(2)
            t, rows = _clip(t, d)
            of = of[rows]
        total.index_add_(0, of, _measures(t))
    return total


def exact(case, seed):
    op = case["op"]
    if op in ("elements", "dropin"):
        return None  # a subdivision has no values but its own
    if op == "batched":
        none = dict.fromkeys(("n_candidates", "n_intersecting", "cand_offset", "ind_ptr", "indices", "pair_measure",
                              "pair_n_out", "p1_offset", "p1_blocks"))
        return dict(none, totals=np.ones(case["count"]))  # each mesh fills the unit square or cube
    if op == "pairs":
        dim, a, b = _element_pairs(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        a, b = (torch.from_numpy(x).to(dev).reshape(case["n"], -1, dim) for x in (a, b))
        return {"measure": torch.cat([_pair_measures(x, y, dim) for x, y in zip(a.split(1 << 18), b.split(1 << 18))]),
                "n_out": None}
    if op == "p1":
        u, v = _fields(case, seed)
        dim = case["dim"]
        r = u[0] * v[0] + 0.5 * (u[0] * v[1:].sum() + v[0] * u[1:].sum())
        for i in range(dim):
            for j in range(dim):
                r += u[1 + i] * v[1 + j] * (1 / 3 if i == j else 0.25)
        return {"integral": float(r)}
    # B covers all of A, so what lies in an element of A is its own measure
    A, _ = _mesh_pair(case, seed)
    em = _measures(torch.from_numpy(A[0])[torch.from_numpy(A[1]).long()])
    r = {"n_candidates": None, "n_intersecting": None, "n_out": None, "total": math.fsum(em.tolist()),
         "elem_measure": em}
    if op == "csr":
        r.update(n=None, ind_ptr=None, indices=None, pair_measure=None, pair_n_out=None)
    return r
