"""The staged kernels' forms for blocks of short rows that stage little, chosen
by field count, row order and outputs: bit for bit against the direct kernel,
the low parts of hi+lo outputs included."""
import numpy as np
import pytest

from test_gpu_apply_shapes import _check_split, _reference

pytestmark = pytest.mark.gpu


def _fine(gpu, lens, n_src, seed):
    """A destination much finer than the source: rows of the given lengths over neighbouring cells."""
    rng = np.random.default_rng(seed)
    n = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.minimum(np.arange(n) * n_src // n, n_src - 9)
    col = np.concatenate([s + np.sort(rng.choice(9, k, replace=False)) for s, k in zip(start, lens)])
    return gpu.Matrix.from_csr(n_src, n, rp, col, rng.uniform(0.1, 1.0, rp[-1]))


def _staged_and_direct(gpu, M, xs, fpp):
    """(y, lo) of the hi+lo apply by the producer-warp kernel and by the direct one."""
    nf, out = xs.shape[0], []
    for v, u, st in ((3, 4, 0), (4, 1, 2)):
        gpu.set_kernel_choice(M, nf, variant=v, fields_per_pass=fpp, unroll=u, stages=st)
        out.append(gpu.apply_f32split_hilo(M, xs))
    return out


@pytest.mark.parametrize("rows", ["uniform", "mixed", "eight"])
@pytest.mark.parametrize("nf,fpp", [(1, 0), (15, 0), (16, 0), (17, 0), (33, 16), (40, 20), (100, 0), (100, 52)])
def test_hilo_of_blocks_that_stage_little(gpu, oracle, rows, nf, fpp):
    """Rows of one length keep their order (16 fields a stage), rows of mixed
    lengths do not (4 fields a stage with two outputs)."""
    import torch
    rng = np.random.default_rng(71)
    lens = {"uniform": np.full(3001, 2), "mixed": rng.integers(1, 5, 3001), "eight": rng.integers(0, 9, 3001)}[rows]
    M = _fine(gpu, lens, 500, 72)
    X = rng.standard_normal((nf, 500)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    (y, lo), (y2, lo2) = _staged_and_direct(gpu, M, xs, fpp)
    assert torch.equal(y, y2) and torch.equal(lo, lo2)
    ref, cond = _reference(M, oracle, X)
    _check_split(y.cpu().numpy(), ref, cond)
    # y + lo carries the sum to 2^-46 a term (as the module's note on tolerances has it)
    assert np.all(np.abs(y.cpu().numpy().astype(np.float64) + lo.cpu().numpy() - ref) <= 1e-10 * cond)
    assert torch.equal(gpu.apply_f32split(M, xs), y2)
    assert M.device_status() == 0


def _blocks(gpu, lens, seed):
    """Neighbouring rows share their sources: every block is staged."""
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.arange(len(lens)) // 4
    col = np.arange(rp[-1]) - np.repeat(rp[:-1] - start, lens)
    return gpu.Matrix.from_csr(int(col.max()) + 1, len(lens), rp, col, rng.uniform(0.1, 1.0, rp[-1]))


@pytest.mark.parametrize("nf", [3, 5, 10, 24, 40, 100, 129, 150])
@pytest.mark.parametrize("kind", ["one class", "little and much", "many classes"])
def test_default_split_of_the_fields(gpu, oracle, kind, nf):
    """The default choice's work items, staged (little and much staging joined
    and apart) and direct, against one item for all fields."""
    import torch
    rng = np.random.default_rng(81)
    lens = {"one class": np.full(120000, 4), "little and much": np.full(120000, 3),
            "many classes": np.repeat(np.arange(1, 33), 1900)}[kind]
    M = _blocks(gpu, lens, 82)
    if kind == "little and much":  # some blocks' sources lie apart
        c = M.to_csr()
        col = c["col"].reshape(-1, 3)
        far = (np.arange(120000) // 128) % 3 == 0
        col[far, 2] = M.n_src + np.arange(far.sum())
        M = gpu.Matrix.from_csr(M.n_src + int(far.sum()), M.n_dst, c["row_ptr"], col.reshape(-1), c["val"])
    X = rng.standard_normal((nf, (M.n_src + 3) // 4 * 4)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")[:, :M.n_src]
    y = gpu.apply_f32split(M, xs)
    assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=4, variant=3), y)
    assert torch.equal(gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=1, variant=4), y)
    _check_split(y.cpu().numpy()[:3], *_reference(M, oracle, X[:3, :M.n_src]))
    assert gpu.get_kernel_choice(M, nf)["variant"] in ((3, 4) if nf >= 8 else (1, 4))
    assert M.device_status() == 0


@pytest.mark.parametrize("nfs", [(1, 5, 30, 2), (33, 40, 64, 17), (3, 3, 4, 4)])
def test_batches_of_small_and_large_groups(gpu, nfs):
    """Batches whose classes of few blocks are joined across lengths and
    strides, beside large ones that are not; bit for bit the single applies."""
    import torch
    rng = np.random.default_rng(91)
    few = np.repeat(np.arange(1, 33), 300)  # three blocks a length
    wide = rng.integers(1, 33, 5000)        # scattered rows: large strides, some left to the slices
    rp = np.concatenate([[0], np.cumsum(wide)])
    start = np.minimum(np.arange(5000) * 4, 20000)
    col = np.concatenate([s + np.sort(rng.choice(120, k, replace=False)) for s, k in zip(start, wide)])
    ms = [_blocks(gpu, few, 92), gpu.Matrix.from_csr(20120, 5000, rp, col, rng.uniform(0.1, 1.0, rp[-1])),
          _blocks(gpu, np.full(60000, 4), 93), _fine(gpu, rng.integers(0, 9, 9001), 1000, 94)]
    xs = [torch.randn((n, (m.n_src + 3) // 4 * 4), device="cuda")[:, :m.n_src] for n, m in zip(nfs, ms)]
    ys = [torch.full((n, m.n_dst), float("nan"), device="cuda") for n, m in zip(nfs, ms)]
    B = gpu.Batch(ms, list(nfs))
    for _ in range(2):
        B.apply(xs, ys)
        for m, x, y in zip(ms, xs, ys):
            assert torch.equal(y, gpu.apply_f32split(m, x, fields_per_pass=0, unroll=1, variant=4))
            assert m.device_status() == 0
            y.fill_(float("nan"))
