"""Weight generation on cells of many shapes: vertex counts at and past what
the convex clipper keeps, cells that are not convex, regular and
unstructured meshes on either side. The bars are those of the parity tests:
index set exact, values within 1e-12."""
import numpy as np
import pytest

from axgb import grids

from test_gpu_parity import _check_weights

pytestmark = pytest.mark.gpu


def _subdivided(m, k, bulge=0.0):
    """m with k points on every edge (from its first vertex on) of each cell,
    the inner ones moved towards the cell's mean by bulge: 4 k vertices a
    quadrilateral, concave for bulge > 0."""
    ll, idx = m.node_lonlat, m.conn_indices.reshape(-1, 4)
    v = ll[idx]  # [cells, 4, 2]
    mean = v.mean(axis=1, keepdims=True)
    pts = []
    for e in range(4):
        a, b = v[:, e], v[:, (e + 1) % 4]
        for q in range(k):
            p = a + (b - a) * (q / k)
            if q:
                p = p + bulge * (mean[:, 0] - p)
            pts.append(p)
    node = np.stack(pts, axis=1).reshape(-1, 2)
    n = m.n_cells
    return grids.MeshArrays(node, np.arange(0, 4 * k * n + 1, 4 * k, dtype=np.int64), np.arange(4 * k * n), name="sub")


@pytest.mark.parametrize("side", ["src", "dst"])
@pytest.mark.parametrize("k,bulge", [(2, 0.0), (3, 0.0), (4, 0.0), (9, 0.0), (2, 0.15), (3, 0.3)])
def test_many_vertices_and_concave_cells(gpu, oracle, k, bulge, side):
    """8 to 36 vertices a cell (12 are kept by the convex clipper, 32 by any)."""
    a = _subdivided(grids.rectilinear(np.linspace(20.0, 70.0, 21), np.linspace(-30.0, 25.0, 19)), k, bulge)
    b = grids.cubed_sphere(12)
    src, dst = (a, b) if side == "src" else (b, a)
    M = gpu.generate_weights(gpu.Mesh.from_grid(src), gpu.Mesh.from_grid(dst), {"method": "conservative"})
    _check_weights(M, oracle.conservative(src, dst))
    if side == "src" and (bulge > 0.0 or 4 * k > 12):  # the source cell is the polygon that is cut
        assert M.stats()["fallback_clips"] > 0


def _band(n_lon, lat_edges):
    return grids.rectilinear(np.linspace(0.0, 360.0, n_lon + 1), lat_edges)


@pytest.mark.parametrize("name,src,dst", [
    # a few destination cells over thousands of source cells: every row is walked by a warp, the CSR order
    # comes from the radix sort
    ("coarse", lambda: grids.cubed_sphere(48), lambda: grids.latlon_deg(60.0)),
    # rows of 1 to 720 candidates in one matrix (polar cells of a lat-lon source), direct placement
    ("polar", lambda: _band(720, np.linspace(-90.0, 90.0, 181)), lambda: grids.cubed_sphere(90)),
    # rows within one candidate of what a thread keeps, few cells
    ("tiny", lambda: grids.cubed_sphere(5), lambda: grids.cubed_sphere(3)),
    ("one", lambda: grids.cubed_sphere(4), lambda: grids.regular_latlon(1, 1, 10.0, -20.0, 30.0, 25.0)),
])
@pytest.mark.parametrize("norm", [0, 1])
def test_search_and_placement_paths(gpu, oracle, name, src, dst, norm):
    """Candidate search by threads and by warps, CSR placement by ranks and by
    the radix sort, both normalisations."""
    src, dst = src(), dst()
    M = gpu.generate_weights(gpu.Mesh.from_grid(src), gpu.Mesh.from_grid(dst),
                             {"method": "conservative", "norm_type": norm})
    wo = oracle.conservative(src, dst, norm_type=norm)
    _check_weights(M, wo)
    st = M.stats()
    assert st["gated_pairs"] == wo.stats["cap_pass"]


@pytest.mark.parametrize("name,src,dst", [
    # edges along the same great circles: vertices on the edges they are tested against
    ("aligned", lambda: grids.cubed_sphere(16), lambda: grids.cubed_sphere(8)),
    # edges of 1e-8 radian, where no FP32 side test decides
    ("tiny_cells", lambda: _subdivided(grids.rectilinear(10.0 + 6e-7 * np.arange(9), 20.0 + 6e-7 * np.arange(8)), 2),
     lambda: _subdivided(grids.rectilinear(10.0 + 7.1e-7 * np.arange(6), 20.0 + 5.3e-7 * np.arange(7)), 2)),
    # cells with caps of more than a radian on either side
    ("huge_src", lambda: grids.rectilinear(np.linspace(0.0, 360.0, 4), np.array([-90.0, -10.0, 90.0])),
     lambda: grids.cubed_sphere(6)),
    ("huge_dst", lambda: grids.cubed_sphere(6),
     lambda: grids.rectilinear(np.linspace(0.0, 360.0, 4), np.array([-90.0, -10.0, 90.0]))),
])
def test_side_tests_at_their_limits(gpu, oracle, name, src, dst):
    src, dst = src(), dst()
    M = gpu.generate_weights(gpu.Mesh.from_grid(src), gpu.Mesh.from_grid(dst), {"method": "conservative"})
    _check_weights(M, oracle.conservative(src, dst))


@pytest.mark.parametrize("nnz", [0, 10, 65536, 65537, 131072, 131073, 1048577])
def test_export_round_trip(gpu, nnz):
    """CSR export below and above the size from which threads move it, at the
    ends of their pieces (131,072 indices, 65,536 values), twice into arrays
    that hold something else."""
    rng = np.random.default_rng(nnz)
    n_dst, n_src = max(1, nnz // 7), 1000 + nnz // 3
    lens = np.bincount(rng.integers(0, n_dst, nnz), minlength=n_dst)
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = rng.integers(0, n_src, nnz)
    row = np.repeat(np.arange(n_dst), lens)
    col = col[np.lexsort((col, row))]
    val, fa, fb, aa, ab = (rng.standard_normal(n) for n in (nnz, n_src, n_dst, n_src, n_dst))
    M = gpu.Matrix.from_csr(n_src, n_dst, rp, col, val, fa, fb, aa, ab)
    for _ in range(2):
        c = M.to_csr()
        for k, v in dict(row_ptr=rp, col=col, val=val, frac_a=fa, frac_b=fb, area_a=aa, area_b=ab).items():
            assert np.array_equal(c[k], v), k
