"""Forms of the FP64 and NaN-aware applies that depend on the rows' lengths:
against the oracle's sums (bit for bit for the NaN-aware apply)."""
import numpy as np
import pytest

from test_gpu_apply_shapes import _check_f64, _check_split, _reference, _rows_matrix

pytestmark = pytest.mark.gpu


def _nan_check(gpu, oracle, lens, nf, seed):
    import torch
    from oracle import Weights
    M = _rows_matrix(gpu, np.asarray(lens, np.int64), 4000, seed)
    rng = np.random.default_rng(seed + 1)
    X = rng.standard_normal((nf, M.n_src))
    X[rng.random((nf, M.n_src)) < 0.05] = np.nan
    X[nf - 1, 1000:3000] = np.nan
    c = M.to_csr()
    row = np.repeat(np.arange(M.n_dst), np.diff(c["row_ptr"])).astype(np.int64)
    w = Weights(M.n_src, M.n_dst, row, c["col"].astype(np.int64), c["val"], c["frac_a"], c["frac_b"], c["area_a"],
                c["area_b"])
    ref = oracle.nan_batch_apply(w, X, 0.5)
    y = gpu.nan_apply_f64(M, torch.tensor(X, device="cuda"), 0.5).cpu().numpy()
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.array_equal(y[~np.isnan(y)], ref[~np.isnan(ref)])


@pytest.mark.parametrize("nf", [8, 9, 10, 11, 12, 13, 15, 16, 17, 27])
@pytest.mark.parametrize("lens", [[33, 40, 37] * 40, [33, 5, 20, 40] * 40, [60] * 90, [100, 3] * 50],
                         ids=["all long", "a quarter", "sixty", "hundred"])
def test_nan_fields_beside_long_rows(gpu, oracle, nf, lens):
    """Field counts that leave part of a long row's lanes without a field; 9 to
    11 in one launch and in two."""
    _nan_check(gpu, oracle, lens, nf, 61)


@pytest.mark.parametrize("heavy", [1, 7, 30, 120])
def test_heavy_rows_between_others(gpu, oracle, heavy):
    """Rows of more than 256 entries come first in the long rows' list, others
    between them: few, as many as the others, and more than those."""
    import torch
    rng = np.random.default_rng(71)
    lens = np.concatenate([rng.integers(257, 1200, heavy), rng.integers(33, 257, 60), rng.integers(0, 33, 200)])
    rng.shuffle(lens)
    M = _rows_matrix(gpu, lens, 4000, 72)
    for nf in (1, 5, 20):
        X = np.random.default_rng(73).standard_normal((nf, M.n_src)).astype(np.float32)
        xs = torch.tensor(X, device="cuda")
        ref, cond = _reference(M, oracle, X)
        y = gpu.apply_f32split(M, xs)
        _check_split(y.cpu().numpy(), ref, cond)
        assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=4, variant=3), y)
        _check_f64(gpu.apply_f64(M, xs.double()).cpu().numpy(), ref, cond)
    _nan_check(gpu, oracle, lens, 3, 74)


@pytest.mark.parametrize("nf", [2, 3, 4, 7, 8, 9, 16, 65, 70])
@pytest.mark.parametrize("lens", ["ones", "ones and none", "a warp of ones"])
def test_rows_of_one_entry(gpu, oracle, nf, lens):
    """Warps whose rows have one entry or none take eight fields at a time; the
    others of the matrix do not."""
    import torch
    rng = np.random.default_rng(81)
    n = 3001
    l = {"ones": np.ones(n), "ones and none": rng.integers(0, 2, n),
         "a warp of ones": np.where(np.arange(n) // 128 % 2, 1, rng.integers(0, 7, n))}[lens].astype(np.int64)
    M = _rows_matrix(gpu, l, 900, 82)
    X = rng.standard_normal((nf, M.n_src))
    X[0, :5] = [np.inf, -np.inf, np.nan, -0.0, 0.0]
    xs = torch.tensor(X, device="cuda")
    d = gpu.apply_f64(M, xs).cpu().numpy()
    X0 = X.copy()
    X0[0, :3] = 1.0
    _check_f64(d[1:], *(v[1:] for v in _reference(M, oracle, X0)))
    for f in range(0, nf, max(1, nf // 6)):
        one = gpu.apply_f64(M, xs[f:f + 1]).cpu().numpy()[0]
        assert np.array_equal(one, d[f], equal_nan=True)
        assert np.array_equal(np.signbit(one), np.signbit(d[f]))


@pytest.mark.parametrize("nf,rows", [(21, 64000), (29, 50001), (65, 64000)])
def test_field_tiles_of_eight_and_more(gpu, oracle, nf, rows):
    """Work for which a warp takes tiles of 8 fields, several of them and the last in part
    (at least 38,912 slices times fields), and of 16."""
    import torch
    M = _rows_matrix(gpu, np.random.default_rng(91).integers(0, 9, rows), 900, 92)
    X = np.random.default_rng(93).standard_normal((nf, M.n_src))
    xs = torch.tensor(X, device="cuda")
    d = gpu.apply_f64(M, xs).cpu().numpy()
    _check_f64(d, *_reference(M, oracle, X))
    for f in (0, 7, 8, 16, nf - 1):
        assert np.array_equal(gpu.apply_f64(M, xs[f:f + 1]).cpu().numpy()[0], d[f])
