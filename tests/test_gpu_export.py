"""CSR exports whose size takes every count of host threads, into arrays that
are new and that hold something else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mib", [1.2, 4, 10.1, 12.6, 15.1, 17.6, 25])
def test_exports_by_size(gpu, mib):
    n = int(mib * 2**20 / 16)  # about 16 bytes an entry on the device: index, weight, row start
    rng = np.random.default_rng(n)
    col = rng.integers(0, 1000, n)
    val, aa, ab = rng.standard_normal(n), rng.standard_normal(1000), rng.standard_normal(n)
    M = gpu.Matrix.from_csr(1000, n, np.arange(n + 1), col, val, None, None, aa, ab)
    kept = []
    for _ in range(2):
        c = M.to_csr()
        for k, v in dict(row_ptr=np.arange(n + 1), col=col, val=val, area_a=aa, area_b=ab, frac_a=np.ones(1000),
                         frac_b=np.ones(n)).items():
            assert np.array_equal(c[k], v), k
        kept.append(c)
