"""Forms of the FP64 and NaN-aware applies that depend on the rows' lengths:
against the oracle's sums (bit for bit for the NaN-aware apply)."""
import numpy as np
import pytest

from test_gpu_apply_shapes import _check_f64, _reference, _rows_matrix

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
