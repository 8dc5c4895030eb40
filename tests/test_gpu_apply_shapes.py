"""Applies on row lengths, field counts and alignments at the edges of the
kernels' tiles, on matrices built from given rows. Every split kernel has to
give the same bits, and each result is checked against the oracle's
compensated FP64 sums.

Tolerances: a split output is the compensated sum rounded once to FP32, so it
is within half an ulp (2^-24 of its value) plus the sum's own error, at most
n 2^-46 <= 1e-10 of the row's condition sum |w x| for the rows used here; an
FP64 output carries n rounding errors of 2^-53 of the condition (n <= 4300:
5e-13, 1e-12 allowed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows_matrix(gpu, lens, n_src, seed):
    """Rows of the given lengths: ascending columns in runs with gaps, as the
    rows of a finer source have, weights uniform in (0, 1] over the length."""
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = np.empty(rp[-1], np.int64)
    for r, n in enumerate(lens):
        span = min(n_src, n + n // 3 + 2)
        start = rng.integers(0, n_src - span + 1)
        col[rp[r]:rp[r + 1]] = start + np.sort(rng.choice(span, n, replace=False))
    val = rng.uniform(1e-3, 1.0, rp[-1]) / np.maximum(1, np.repeat(lens, lens))
    return gpu.Matrix.from_csr(n_src, len(lens), rp, col, val)


def _reference(M, oracle, X):
    """Compensated FP64 sums and the condition of every output."""
    from oracle import Weights
    c = M.to_csr()
    row = np.repeat(np.arange(M.n_dst), np.diff(c["row_ptr"])).astype(np.int64)
    w = Weights(M.n_src, M.n_dst, row, c["col"].astype(np.int64), c["val"], c["frac_a"], c["frac_b"], c["area_a"],
                c["area_b"])
    x = X.astype(np.float64)
    return oracle.apply_csr(w, x, compensated=True), oracle.apply_csr(w, np.abs(x), compensated=True)


def _check_split(y, ref, cond):
    assert np.all(np.abs(y.astype(np.float64) - ref) <= 1.0001 * 2.0**-24 * np.abs(ref) + 1e-10 * cond)


def _check_f64(y, ref, cond):
    assert np.all(np.abs(y - ref) <= 1e-12 * cond)


LONG = [33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 159, 160, 161, 192, 255, 256, 257, 1000]
SHORT = [0, 1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17, 31, 32]


def _mixed_lens(seed):
    rng = np.random.default_rng(seed)
    mixed = np.array((LONG + SHORT) * 12)
    rng.shuffle(mixed)
    # whole slices of long rows, an empty slice, short slices, and a ragged end
    return np.concatenate([mixed, [40] * 160, [0] * 64, rng.choice(SHORT, 300), [70] * 3, [3] * 2]).astype(np.int64)


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 7, 8, 9, 17, 33])
def test_mixed_row_lengths(gpu, oracle, nf):
    """Rows longer than 32 entries among short ones: the long rows' tree for
    every count of fields a warp carries, blocks staged without their long
    rows, and blocks of nothing else."""
    import torch
    M = _rows_matrix(gpu, _mixed_lens(1), 4000, 2)
    X = np.random.default_rng(3).standard_normal((nf, M.n_src)).astype(np.float32)
    ref, cond = _reference(M, oracle, X)
    xs = torch.tensor(X, device="cuda")
    y = gpu.apply_f32split(M, xs).cpu().numpy()
    _check_split(y, ref, cond)
    forms = [(0, 0, 1), (0, 0, 4), (1, 0, 4), (1, 8, 8), (2, 0, 4), (3, 0, 4), (3, 8, 4), (4, 0, 1), (5, 0, 32)]
    for v, fpp, u in forms:
        assert np.array_equal(gpu.apply_f32split(M, xs, fields_per_pass=fpp, unroll=u, variant=v).cpu().numpy(), y), v
    assert M.device_status() == 0
    for f in {0, nf - 1}:
        assert np.array_equal(gpu.apply_f32split(M, xs[f:f + 1]).cpu().numpy()[0], y[f])
    B = gpu.Batch([M, M], [nf, 1])
    ys = [torch.empty((n, M.n_dst), dtype=torch.float32, device="cuda") for n in (nf, 1)]
    B.apply([xs, xs[nf - 1:]], ys)
    assert np.array_equal(ys[0].cpu().numpy(), y) and np.array_equal(ys[1].cpu().numpy()[0], y[nf - 1])
    d = gpu.apply_f64(M, xs.double()).cpu().numpy()
    _check_f64(d, ref, cond)
    assert np.array_equal(gpu.apply_f64(M, xs[:1].double()).cpu().numpy()[0], d[0])


@pytest.mark.parametrize("nf,rows", [(8, 31), (40, 129), (129, 1000), (500, 260), (200, 5000)])
def test_fields_per_work_item(gpu, oracle, nf, rows):
    """The default split of the fields over work items, which depends on the
    matrix's size, against one work item for all fields."""
    import torch
    M = _rows_matrix(gpu, np.random.default_rng(4).choice(SHORT, rows), 900, 5)
    X = np.random.default_rng(6).standard_normal((nf, M.n_src)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    y = gpu.apply_f32split(M, xs).cpu().numpy()
    assert np.array_equal(gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=4, variant=3).cpu().numpy(), y)
    _check_split(y, *_reference(M, oracle, X))


@pytest.mark.parametrize("nf,rows", [(65, 300), (130, 64000)])
def test_f64_field_tiles(gpu, oracle, nf, rows):
    """FP64 applies whose warps take 8 and 16 fields, the last tile in part."""
    import torch
    M = _rows_matrix(gpu, np.random.default_rng(14).choice(SHORT + [40], rows), 900, 15)
    X = np.random.default_rng(16).standard_normal((nf, M.n_src))
    xs = torch.tensor(X, device="cuda")
    d = gpu.apply_f64(M, xs).cpu().numpy()
    _check_f64(d, *_reference(M, oracle, X))
    for f in (0, 8, nf - 1):
        assert np.array_equal(gpu.apply_f64(M, xs[f:f + 1]).cpu().numpy()[0], d[f])


@pytest.mark.parametrize("lens", [[3], [1, 8], [4] * 31 + [5], list(range(33)), [2] * 128 + [1, 30], [40] + [0] * 40 + [2]],
                         ids=["equal", "alternating", "one longer", "ascending", "by group", "empty"])
@pytest.mark.parametrize("nf,rows", [(3, 127), (4, 129), (9, 1001)])
def test_f64_row_orders(gpu, oracle, nf, rows, lens):
    """FP64 applies whose groups of rows run in their own order and by length,
    the last group in part: from three fields up, against one field."""
    import torch
    M = _rows_matrix(gpu, np.resize(lens, rows).astype(np.int64), 900, 41)
    X = np.random.default_rng(42).standard_normal((nf, M.n_src))
    xs = torch.tensor(X, device="cuda")
    d = gpu.apply_f64(M, xs).cpu().numpy()
    _check_f64(d, *_reference(M, oracle, X))
    for f in range(nf):
        assert np.array_equal(gpu.apply_f64(M, xs[f:f + 1]).cpu().numpy()[0], d[f])


@pytest.mark.parametrize("nf", [1, 3, 16, 17, 37])
@pytest.mark.parametrize("weights,na_thres", [("positive", 0.5), ("positive", 0.0), ("positive", 1.0), ("signed", 0.5),
                                              ("positive", -1.0), ("tiny", 0.3)])
def test_nan_apply_row_shapes(gpu, oracle, nf, weights, na_thres):
    """NaN-aware apply, bit for bit, on rows without NaN, with some and with
    nothing else; weights whose sums cancel or lie outside the range of the
    shortened division, infinite and zero fields, and a threshold above 1."""
    import torch
    M = _rows_matrix(gpu, _mixed_lens(21), 4000, 22)
    c = M.to_csr()
    rng = np.random.default_rng(23)
    if weights == "signed":
        c["val"] = c["val"] * rng.choice([-1.0, 1.0], M.nnz)
    if weights == "tiny":
        c["val"] = c["val"] * 2.0**-700
    if weights != "positive":
        M = gpu.Matrix.from_csr(M.n_src, M.n_dst, c["row_ptr"], c["col"], c["val"])
    X = rng.standard_normal((nf, M.n_src)) * np.array([1.0, 2.0**400, 2.0**-600])[np.arange(nf) % 3][:, None]
    X[:, 500:900] = np.nan  # land
    X[rng.random((nf, M.n_src)) < 0.02] = np.nan
    X[nf - 1, ::7] = np.inf
    X[0, 2000:2400] = 0.0
    if nf > 2:
        X[1] = np.nan
        X[2] = np.where(np.isnan(X[2]), 1.0, X[2])
    from oracle import Weights
    row = np.repeat(np.arange(M.n_dst), np.diff(c["row_ptr"])).astype(np.int64)
    w = Weights(M.n_src, M.n_dst, row, c["col"].astype(np.int64), c["val"], c["frac_a"], c["frac_b"], c["area_a"],
                c["area_b"])
    ref = oracle.nan_batch_apply(w, X, na_thres)
    y = gpu.nan_apply_f64(M, torch.tensor(X, device="cuda"), na_thres).cpu().numpy()
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.array_equal(y[~np.isnan(y)], ref[~np.isnan(ref)])


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15])
@pytest.mark.parametrize("lens", [LONG, [40, 33] * 33, [33, 1000, 5, 64, 0, 128, 32] * 3], ids=["long", "even", "mixed"])
def test_nan_long_rows_side_by_side(gpu, oracle, nf, lens):
    """Few fields: a warp takes several long rows, of different lengths, the
    last warp fewer; bit for bit."""
    import torch
    from oracle import Weights
    M = _rows_matrix(gpu, np.array(lens, np.int64), 4000, 51)
    X = np.random.default_rng(52).standard_normal((nf, M.n_src))
    X[:, ::5] = np.nan
    X[nf - 1, 1000:3000] = np.nan
    c = M.to_csr()
    row = np.repeat(np.arange(M.n_dst), np.diff(c["row_ptr"])).astype(np.int64)
    w = Weights(M.n_src, M.n_dst, row, c["col"].astype(np.int64), c["val"], c["frac_a"], c["frac_b"], c["area_a"],
                c["area_b"])
    ref = oracle.nan_batch_apply(w, X, 0.5)
    y = gpu.nan_apply_f64(M, torch.tensor(X, device="cuda"), 0.5).cpu().numpy()
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.array_equal(y[~np.isnan(y)], ref[~np.isnan(ref)])


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 8, 9, 45])
def test_unaligned_fields(gpu, oracle, nf):
    """Fields whose rows do not start on 16 bytes (an odd number of cells, and
    a view one element into a buffer): the same bits as from aligned rows,
    the hi+lo form included."""
    import torch
    M = _rows_matrix(gpu, _mixed_lens(31), 4001, 32)
    X = np.random.default_rng(33).standard_normal((nf, M.n_src)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    pad = torch.zeros((nf, 4004), dtype=torch.float32, device="cuda")
    pad[:, :4001] = xs
    off = torch.zeros(nf * 4004 + 1, dtype=torch.float32, device="cuda")[1:].view(nf, 4004)
    off[:, :4001] = xs
    y, lo = gpu.apply_f32split_hilo(M, pad[:, :4001])
    _check_split(y.cpu().numpy(), *_reference(M, oracle, X))
    for x in (xs, off[:, :4001]):
        y2, lo2 = gpu.apply_f32split_hilo(M, x)
        assert torch.equal(y2, y) and torch.equal(lo2, lo)
        assert torch.equal(gpu.apply_f32split(M, x), y)
    for v, u in ((0, 1), (0, 2), (0, 4), (1, 4), (3, 4)):
        assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=3, unroll=u, variant=v), y)


@pytest.mark.parametrize("nf", [1, 2, 3, 8, 40])
def test_rows_too_scattered_to_stage(gpu, oracle, nf):
    """Blocks of 128 rows that touch more source chunks than a staging slot
    holds go to the direct kernel, slice by slice."""
    import torch
    rng = np.random.default_rng(41)
    lens = rng.integers(20, 33, 400)
    lens[128:256] = rng.integers(0, 4, 128)  # one block that is staged
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = np.concatenate([np.sort(rng.choice(60000, n, replace=False)) for n in lens])
    M = gpu.Matrix.from_csr(60000, 400, rp, col, rng.uniform(0.0, 1.0, rp[-1]))
    X = rng.standard_normal((nf, M.n_src)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    y = gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=4, variant=3)
    _check_split(y.cpu().numpy(), *_reference(M, oracle, X))
    for v, fpp, u in ((0, 0, 1), (0, 4, 4), (1, 0, 4), (2, 0, 4), (4, 0, 1)):
        assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=fpp, unroll=u, variant=v), y)
    assert torch.equal(gpu.apply_f32split(M, xs), y)


@pytest.mark.parametrize("nf", [1, 3, 70])
@pytest.mark.parametrize("window", [3000, 9000, 20003])
def test_renumbered_sources(gpu, oracle, window, nf):
    """Source cells numbered without locality inside windows of a latitude
    band's size (gathered through shared memory) or of the whole mesh (gathered
    from memory); an odd number of cells, the last tile and window in part."""
    import torch
    n_src, n_dst = 20003, 9000
    rng = np.random.default_rng(51)
    perm = np.concatenate([w + rng.permutation(min(window, n_src - w)) for w in range(0, n_src, window)])
    lens = rng.integers(1, 8, n_dst)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.minimum(np.arange(n_dst) * n_src // n_dst, n_src - 8)
    col = np.concatenate([np.sort(perm[s:s + n]) for s, n in zip(start, lens)])
    M = gpu.Matrix.from_csr(n_src, n_dst, rp, col, rng.uniform(0.1, 1.0, rp[-1]))
    X = rng.standard_normal((nf, n_src)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    y = gpu.apply_f32split(M, xs)
    assert M.stats()["source_renumbered"]
    _check_split(y.cpu().numpy(), *_reference(M, oracle, X))
    for v, fpp, u in ((0, 0, 2), (3, 8, 4), (4, 0, 1), (5, 0, 32)):
        assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=fpp, unroll=u, variant=v), y)
    B = gpu.Batch([M], [nf])
    yb = torch.empty_like(y)
    B.apply([xs], [yb])
    assert torch.equal(yb, y)


@pytest.mark.parametrize("most", [4, 8])
@pytest.mark.parametrize("nf", [8, 15, 16, 17, 31, 33, 100])
def test_short_rows_little_staging(gpu, oracle, nf, most):
    """A destination much finer than the source: short rows, few source chunks a
    block, 16 fields a stage (8 in a batch), the last stage in part."""
    import torch
    rng = np.random.default_rng(61)
    n_src, n_dst = 500, 3001
    lens = rng.integers(0, most + 1, n_dst)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.minimum(np.arange(n_dst) * n_src // n_dst, n_src - 9)
    col = np.concatenate([s + np.sort(rng.choice(9, n, replace=False)) for s, n in zip(start, lens)])
    M = gpu.Matrix.from_csr(n_src, n_dst, rp, col, rng.uniform(0.1, 1.0, rp[-1]))
    X = rng.standard_normal((nf, n_src)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    y = gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=4, variant=3)
    _check_split(y.cpu().numpy(), *_reference(M, oracle, X))
    for v, fpp, u in ((0, 0, 4), (1, 0, 8), (2, 0, 4), (3, 20, 4), (4, 0, 1)):
        assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=fpp, unroll=u, variant=v), y)
    B = gpu.Batch([M, M], [nf, 5])
    yb = [torch.empty((n, n_dst), dtype=torch.float32, device="cuda") for n in (nf, 5)]
    B.apply([xs, xs[:5]], yb)
    assert torch.equal(yb[0], y) and torch.equal(yb[1], y[:5])
    assert M.device_status() == 0
