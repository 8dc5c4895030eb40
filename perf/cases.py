"""The work that users of axgb have it do, as cases that can be timed and compared.

A case names a source and a destination grid, a method and a number of
fields; the calls go through the Python API (``axgb``). Grids are written

    C<n>         cubed sphere, 6 n^2 cells
    L<ni>x<nj>   global regular lat-lon
    T<ni>x<nj>   curvilinear tripole-style ocean grid
    V<n>         spherical Voronoi mesh of n cells

A program generates the weights of a grid pair once and applies them to every
field that follows, so the matrices (with the layouts that the calls use) are
kept here from one state to the next; the fields are new in every state.
"""

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "helm-project_gb300"))

import axgb  # noqa: E402
from axgb import fields, grids  # noqa: E402

NA_THRES = 0.5  # nan cases: a destination cell is kept when half of its weight is valid
N_BASE = 6      # spherical-harmonic patterns that a state's fields are mixed from


def _pairs17():
    """Every cubed sphere against every lat-lon grid, the direction alternating,
    and an ocean grid onto 0.5 degree, with uneven field counts in 1..64."""
    rng = np.random.default_rng(4)
    pairs = []
    for i, c in enumerate(("C48", "C96", "C192", "C384")):
        for j, q in enumerate(("L180x90", "L360x180", "L720x360", "L1440x720")):
            s, d = (c, q) if (i + j) % 2 == 0 else (q, c)
            pairs.append("%s>%s:%d" % (s, d, rng.integers(1, 65)))
    pairs.append("T1440x1080>L720x360:%d" % rng.integers(1, 65))
    return " ".join(pairs)


def listed():
    return [
        # one FP64 field on small grids through the reference's own call: launch and host latency
        {"name": "f64_one_1deg_c48", "kind": "apply", "src": "L360x180", "dst": "C48", "fields": 1},
        # one 2-D field (a surface variable) at 0.25 degree
        {"name": "split_one_0p25_c384", "kind": "split", "src": "L1440x720", "dst": "C384", "fields": 1, "hilo": False},
        # a handful of coupling fluxes whose integrals have to be kept: hi+lo outputs
        {"name": "split_fluxes_c192_0p5", "kind": "split", "src": "C192", "dst": "L720x360", "fields": 7, "hilo": True},
        # the levels of one ocean variable; odd sizes on the source side (rows of the field array are not 16-byte aligned)
        {"name": "split_ragged_ocean_1deg", "kind": "split", "src": "T361x271", "dst": "L360x180", "fields": 45,
         "hilo": False},
        # coarsening: a fine analysis onto a climate grid, rows of about a hundred to some thousand entries
        {"name": "split_coarsen_0p25_c48", "kind": "split", "src": "L1440x720", "dst": "C48", "fields": 45,
         "hilo": False},
        # all tracers and levels of a high-resolution model at once
        {"name": "split_tracers_c768_0p25", "kind": "split", "src": "C768", "dst": "L1440x720", "fields": 1016,
         "hilo": False},
        # the levels of one variable of an unstructured mesh, cells in an order without locality, an odd number of them
        {"name": "split_voronoi_0p5", "kind": "split", "src": "V163843", "dst": "L720x360", "fields": 64, "hilo": False},
        # the levels of one variable in FP64
        {"name": "f64_levels_c192_0p5", "kind": "f64", "src": "C192", "dst": "L720x360", "fields": 64},
        # ocean fields with land missing (skipna)
        {"name": "nan_0p25_c384", "kind": "nan", "src": "L1440x720", "dst": "C384", "fields": 16},
        # a coupler's exchange: 17 grid pairs of uneven sizes and field counts in one call
        {"name": "batch_17_pairs", "kind": "batch", "pairs": _pairs17()},
        # making the weights of a pair and taking them out (to a file or another program)
        {"name": "generate_cons_0p25_c384", "kind": "generate", "src": "L1440x720", "dst": "C384",
         "method": "conservative"},
        {"name": "generate_bilinear_0p25_c384", "kind": "generate", "src": "L1440x720", "dst": "C384",
         "method": "bilinear"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng, most=1_000_000):
    cells = _log_uniform(rng, 3_000, most)
    kind = rng.choice("CCLLLTV")
    if kind == "C":
        return "C%d" % max(8, round(math.sqrt(cells / 6)))
    if kind == "V":
        return "V%d" % min(cells, 40_000)
    ni = max(16, round(math.sqrt(cells * (2.0 if kind == "L" else 4 / 3))))
    return "%s%dx%d" % (kind, ni, max(12, round(cells / ni)))


def _draw_pair(rng, most=1_000_000):
    """Either side may be the finer one; ocean and Voronoi grids are sources."""
    while True:
        s, d = _draw_grid(rng, most), _draw_grid(rng, most)
        if d[0] in "CL":
            return s, d


def draw(rng):
    kind = rng.choice(["apply", "split", "split", "split", "f64", "nan", "batch", "generate"])
    if kind == "batch":
        pairs = []
        for _ in range(rng.randint(2, 8)):
            s, d = _draw_pair(rng, 200_000)
            pairs.append("%s>%s:%d" % (s, d, rng.randint(1, 64)))
        return {"kind": kind, "pairs": " ".join(pairs)}
    s, d = _draw_pair(rng)
    if kind == "generate":
        return {"kind": kind, "src": s, "dst": d, "method": rng.choice(["conservative", "conservative", "bilinear"])}
    case = {"kind": kind, "src": s, "dst": d, "fields": 1}
    if kind != "apply":
        most = max(1, min(1016, int(1.5e9 / (8 * (_cells(s) + _cells(d))))))  # at most 1.5 GB of FP64 fields
        case["fields"] = _log_uniform(rng, 1, most)
    if kind == "split":
        case["hilo"] = rng.random() < 0.2
    return case


# ─── grids, weights and fields ────────────────────────────────────────────


def _dims(spec):
    return tuple(int(v) for v in spec[1:].split("x"))


def _cells(spec):
    d = _dims(spec)
    return 6 * d[0] ** 2 if spec[0] == "C" else d[0] if spec[0] == "V" else d[0] * d[1]


@functools.lru_cache(maxsize=16)
def _grid(spec):
    d = _dims(spec)
    if spec[0] == "C":
        return grids.cubed_sphere(d[0])
    if spec[0] == "L":
        return grids.regular_latlon(*d)
    if spec[0] == "T":
        return grids.tripole(*d)
    return grids.voronoi(d[0], lloyd=1)


@functools.lru_cache(maxsize=16)
def _centroids(spec):
    return torch.tensor(grids.cell_centroids_xyz(_grid(spec)), device="cuda")


@functools.lru_cache(maxsize=40)
def _matrix(src, dst, layout):
    m = axgb.generate_weights(axgb.Mesh.from_grid(_grid(src)), axgb.Mesh.from_grid(_grid(dst)),
                              {"method": "conservative"})
    m.prepare(layout)
    return m


def _fields(spec, n, seed, dtype):
    """[n, cells] fields: seeded spherical harmonics (l <= 16), mixed anew for
    every field and times a lognormal(0, 1) scale, as a model's levels differ."""
    base = fields.sh_fields(_centroids(spec), 16, [seed * N_BASE + k for k in range(N_BASE)]).to(dtype)
    rng = np.random.default_rng(seed)
    mix = rng.standard_normal((n, N_BASE)) * rng.lognormal(0.0, 1.0, (n, 1))
    mix = torch.tensor(mix, dtype=dtype, device=base.device)
    x = torch.empty((n, base.shape[1]), dtype=dtype, device=base.device)
    for f in range(n):
        torch.mv(base.T, mix[f], out=x[f])
    return x


def _pairs(case):
    for p in case["pairs"].split():
        grid_pair, n = p.split(":")
        s, d = grid_pair.split(">")
        yield s, d, int(n)


def _inputs(case, seed):
    """The fields of a state (those of a nan case with land missing)."""
    kind = case["kind"]
    if kind == "batch":
        return [_fields(s, n, seed + 101 * k, torch.float32) for k, (s, _, n) in enumerate(_pairs(case))]
    x = _fields(case["src"], case["fields"], seed, torch.float32 if kind == "split" else torch.float64)
    if kind == "apply":
        return x[0] + 280.0
    if kind == "nan":
        land = fields.sh_fields(_centroids(case["src"]), 16, [seed + 7])[0]
        x[:, land > torch.quantile(land[:: max(1, land.numel() // 100_000)], 0.7)] = float("nan")
    return x


def prepare(case, seed):
    axgb.init(0)
    kind = case["kind"]
    if kind == "generate":
        # other coordinates for other seeds: the source turned by some degrees is another mesh
        turn = float(np.random.default_rng(seed).uniform(0.0, 0.2))
        s, d = _grid(case["src"]), _grid(case["dst"])
        node = s.node_lonlat + np.array([turn, 0.0])
        return {"kind": kind, "method": case["method"],
                "src": axgb.make_ugrid_mesh(node, s.conn_offsets, s.conn_indices), "dst": axgb.Mesh.from_grid(d)}
    x = _inputs(case, seed)
    if kind == "batch":
        ms = [_matrix(s, d, 2) for s, d, _ in _pairs(case)]
        ns = [n for _, _, n in _pairs(case)]
        y = [torch.empty((n, m.n_dst), dtype=torch.float32, device="cuda") for m, n in zip(ms, ns)]
        return {"kind": kind, "b": axgb.Batch(ms, ns), "x": x, "y": y}
    m = _matrix(case["src"], case["dst"], 2 if kind == "split" else 0)
    state = {"kind": kind, "m": m, "x": x}
    if kind != "apply":
        state["y"] = torch.empty((case["fields"], m.n_dst), dtype=x.dtype, device="cuda")
    if kind == "split":
        state["lo"] = torch.empty_like(state["y"]) if case["hilo"] else None
    return state


def run(state):
    kind = state["kind"]
    if kind == "generate":
        return axgb.generate_weights(state["src"], state["dst"], {"method": state["method"]}).to_csr()
    if kind == "batch":
        state["b"].apply(state["x"], state["y"])
        return state["y"]
    if kind == "apply":
        return axgb.apply_weights(state["m"], state["x"])
    if kind == "f64":
        return axgb.apply_f64(state["m"], state["x"], state["y"])
    if kind == "nan":
        return axgb.nan_apply_f64(state["m"], state["x"], NA_THRES, state["y"])
    if state["lo"] is not None:
        return axgb.apply_f32split_hilo(state["m"], state["x"], state["y"], state["lo"])
    return axgb.apply_f32split(state["m"], state["x"], state["y"])


# ─── what a pass cannot do without ────────────────────────────────────────


def _nnz(src, dst, method="conservative"):
    """Overlapping pairs of two tilings of the sphere, their cells taken as
    randomly turned squares (the kinematic formula; within a few per cent)."""
    ns, nd = _cells(src), _cells(dst)
    return 4 * nd if method == "bilinear" else ns + nd + 8.0 / math.pi * math.sqrt(ns * nd)


def _apply_work(src, dst, n, size, out=1):
    ns, nd, nnz = _cells(src), _cells(dst), _nnz(src, dst)
    return {"bytes": size * n * (ns + out * nd) + 12 * nnz + 4 * (nd + 1), "flops": 2 * nnz * n}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_apply_work(s, d, n, 4) for s, d, n in _pairs(case)]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    if kind == "generate":
        ns, nd, nnz = _cells(case["src"]), _cells(case["dst"]), _nnz(case["src"], case["dst"], case["method"])
        # nodes (16 B) and four vertices a cell in; index, weight, fractions and areas out;
        # a clip of two quadrilaterals and the area of the result, or four products
        return {"bytes": 32 * (ns + nd) + 12 * nnz + 16 * (ns + nd),
                "flops": nnz * (400 if case["method"] == "conservative" else 4)}
    if kind == "split":
        return _apply_work(case["src"], case["dst"], case["fields"], 4, 2 if case["hilo"] else 1)
    w = _apply_work(case["src"], case["dst"], case["fields"], 8)
    return {"bytes": w["bytes"], "flops": 2 * w["flops"] if kind == "nan" else w["flops"]}


# ─── the same in 64 bits ──────────────────────────────────────────────────


def _csr(m):
    """The matrix that the state holds (its weights are the apply's input), for torch."""
    c = m.to_csr()
    return torch.sparse_csr_tensor(torch.tensor(c["row_ptr"]), torch.tensor(c["col"]), torch.tensor(c["val"]),
                                   size=(m.n_dst, m.n_src), dtype=torch.float64).cuda()


def _spmm(a, x):
    """a @ x[f] for every field f, in 64 bits."""
    y = torch.empty((x.shape[0], a.shape[0]), dtype=torch.float64, device="cuda")
    for f in range(0, x.shape[0], 32):
        y[f:f + 32] = (a @ x[f:f + 32].double().T.contiguous()).T
    return y


def _sphere_area(spec):
    """Areas of the cells between great circles, by the angle excess of the fan
    of triangles from the first vertex (cubed spheres and lat-lon grids)."""
    if spec[0] not in "CL":
        return None
    g = _grid(spec)
    lon, lat = np.radians(g.node_lonlat).T
    p = np.stack([np.cos(lat) * np.cos(lon), np.cos(lat) * np.sin(lon), np.sin(lat)], axis=1)
    v = p[g.conn_indices.reshape(-1, 4)]
    area = 0.0
    for b, c in ((1, 2), (2, 3)):
        x, y, z = v[:, 0], v[:, b], v[:, c]
        det = np.einsum("ij,ij->i", x, np.cross(y, z))
        area = area + 2.0 * np.arctan2(det, 1.0 + (x * y).sum(1) + (x * z).sum(1) + (y * z).sum(1))
    return np.abs(area)


def _exact_generate(case, seed):
    d, ns, nd = _grid(case["dst"]), _cells(case["src"]), _cells(case["dst"])
    out = dict.fromkeys(("row_ptr", "col", "val", "frac_a", "frac_b", "area_a", "area_b"))
    if case["method"] == "conservative":
        if case["src"][0] != "L" or case["dst"][0] != "L":  # two lat-lon grids have bands between parallels
            out["area_a"], out["area_b"] = _sphere_area(case["src"]), _sphere_area(case["dst"])
        return out
    if case["src"][0] != "L" or case["dst"][0] == "L":
        return out
    # bilinear between the centres of a lat-lon source at the mean corner of each destination cell
    ni, nj = _dims(case["src"])
    turn = float(np.random.default_rng(seed).uniform(0.0, 0.2))
    nv = np.diff(d.conn_offsets)
    cell = np.repeat(np.arange(nd), nv)
    lon, lat = (np.bincount(cell, d.node_lonlat[d.conn_indices, k], nd) / nv for k in (0, 1))
    fx, fy = (lon - turn) * (ni / 360.0) - 0.5, (lat + 90.0) * (nj / 180.0) - 0.5
    tx = np.clip(fx - np.clip(np.floor(fx), 0, ni - 2), 0.0, 1.0)
    ty = np.clip(fy - np.clip(np.floor(fy), 0, nj - 2), 0.0, 1.0)
    out["val"] = np.stack([(1 - tx) * (1 - ty), tx * (1 - ty), (1 - tx) * ty, tx * ty], axis=1).reshape(-1)
    out["frac_a"], out["frac_b"] = np.ones(ns), np.ones(nd)
    return out


def exact(case, seed):
    axgb.init(0)
    kind = case["kind"]
    if kind == "generate":
        return _exact_generate(case, seed)
    x = _inputs(case, seed)
    if kind == "batch":
        return [_spmm(_csr(_matrix(s, d, 2)), x[k]) for k, (s, d, _) in enumerate(_pairs(case))]
    a = _csr(_matrix(case["src"], case["dst"], 2 if kind == "split" else 0))
    if kind == "nan":
        ok = ~torch.isnan(x)
        total, valid = _spmm(a, torch.ones_like(x[:1])), _spmm(a, ok)
        y = _spmm(a, torch.where(ok, x, 0.0)) / valid
        return torch.where((valid > 0) & (total > 0) & (valid / total >= 1.0 - NA_THRES - 1e-6), y, float("nan"))
    y = _spmm(a, x.reshape(case["fields"], -1))
    if kind == "apply":
        return y[0]
    if kind == "split" and case["hilo"]:
        return y, y - y.float().double()
    return y
