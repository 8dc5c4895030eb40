"""First applies of a matrix, which build the layouts: in any order of the
kernel variants, and from several host threads at once. Rows of more than 32
entries, which the staged kernels leave to the sliced layout, are among them;
every split kernel gives the same bits."""
import threading

import numpy as np
import pytest

from test_gpu_apply_shapes import LONG, SHORT, _check_split, _reference, _rows_matrix

pytestmark = pytest.mark.gpu


def _lens(seed):
    return np.random.default_rng(seed).choice(LONG + 4 * SHORT, 700).astype(np.int64)


@pytest.mark.parametrize("first", ["segmented", "prepare", "staged", "direct", "hilo"])
def test_any_variant_first(gpu, oracle, first):
    import torch
    nf = 6
    X = np.random.default_rng(2).standard_normal((nf, 4000)).astype(np.float32)
    xs = torch.tensor(X, device="cuda")
    M = _rows_matrix(gpu, _lens(1), 4000, 3)
    if first == "prepare":
        M.prepare(3)
    elif first == "hilo":
        gpu.apply_f32split_hilo(M, xs)
    else:
        v, u = {"segmented": (5, 32), "staged": (3, 4), "direct": (0, 4)}[first]
        gpu.apply_f32split(M, xs, fields_per_pass=0, unroll=u, variant=v)
    ys = {}
    for v, u in ((3, 4), (1, 4), (2, 4), (0, 4), (4, 1), (5, 32)):
        y = torch.full((nf, M.n_dst), float("nan"), device="cuda")
        ys[v] = gpu.apply_f32split(M, xs, y, fields_per_pass=0, unroll=u, variant=v).cpu().numpy()
    _check_split(ys[3], *_reference(M, oracle, X))
    for v, y in ys.items():
        assert np.array_equal(y, ys[3]), v


@pytest.mark.parametrize("nf", [1, 6, 20])
def test_first_applies_from_several_threads(gpu, nf):
    """Eight threads, each on its own stream, start on a matrix without layouts:
    default, staged, segmented and FP64 applies side by side."""
    import torch
    X = torch.randn((nf, 4000), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    X64 = X.double()
    calls = [lambda M, y: gpu.apply_f32split(M, X, y),
             lambda M, y: gpu.apply_f32split(M, X, y, fields_per_pass=0, unroll=4, variant=3),
             lambda M, y: gpu.apply_f32split(M, X, y, fields_per_pass=0, unroll=32, variant=5),
             lambda M, y: gpu.apply_f64(M, X64, y)]
    for seed in range(6):
        M = _rows_matrix(gpu, _lens(10 + seed), 4000, 20 + seed)
        out = [torch.full((nf, M.n_dst), float("nan"), device="cuda", dtype=torch.float64 if q % 4 == 3 else torch.float32)
               for q in range(8)]
        torch.cuda.synchronize()
        start = threading.Barrier(8)

        def work(q):
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(30)
                calls[q % 4](M, out[q])
                torch.cuda.current_stream().synchronize()

        th = [threading.Thread(target=work, args=(q,)) for q in range(8)]
        for t in th:
            t.start()
        for t in th:
            t.join()
        want = gpu.apply_f32split(M, X, fields_per_pass=0, unroll=1, variant=4)
        want64 = gpu.apply_f64(M, X64)
        for q in range(8):
            assert torch.equal(out[q], want64 if q % 4 == 3 else want), (seed, q)
        assert M.device_status() == 0


@pytest.mark.parametrize("nf,direct", [(3, True), (40, True), (400, False)])
def test_default_choice_before_and_after_the_layouts(gpu, nf, direct):
    """The default kernel choice read from a matrix without layouts is the one
    its applies use: rows of every length class, 8 staged launches, 40 fields
    of half a million entries (more than 12 and less than 32 million)."""
    lens = np.repeat(np.arange(1, 33), 960)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.arange(len(lens)) // 4  # neighbouring rows share their sources: every block is staged
    col = np.arange(rp[-1]) - np.repeat(rp[:-1] - start, lens)
    M = gpu.Matrix.from_csr(int(col.max()) + 1, len(lens), rp, col, np.full(rp[-1], 0.5))
    ch = gpu.get_kernel_choice(M, nf)
    M.prepare(2)
    assert gpu.get_kernel_choice(M, nf) == ch
    assert ch["cached"] is False and (ch["variant"] == 4) is direct


@pytest.mark.parametrize("nf", [1, 5, 40])
def test_renumbered_apply_under_capture(gpu, nf):
    """A split apply whose sources are gathered into scratch first, captured in a
    graph (the scratch is then the graph's) and replayed on new fields."""
    import torch
    n_src, n_dst = 20003, 9000
    rng = np.random.default_rng(61)
    perm = rng.permutation(n_src)
    lens = rng.integers(1, 8, n_dst)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.minimum(np.arange(n_dst) * n_src // n_dst, n_src - 8)
    col = np.concatenate([np.sort(perm[s:s + n]) for s, n in zip(start, lens)])
    M = gpu.Matrix.from_csr(n_src, n_dst, rp, col, rng.uniform(0.1, 1.0, rp[-1]))
    M.prepare(2)
    assert M.stats()["source_renumbered"]
    x = torch.zeros((nf, n_src), device="cuda")
    y = torch.empty((nf, n_dst), device="cuda")
    for v, u in ((None, None), (3, 4)):
        kw = {} if v is None else dict(fields_per_pass=0, unroll=u, variant=v)
        gpu.apply_f32split(M, x, y, **kw)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            gpu.apply_f32split(M, x, y, **kw)
        for k in range(3):
            x.copy_(torch.randn((nf, n_src), device="cuda", generator=torch.Generator(device="cuda").manual_seed(k)))
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, gpu.apply_f32split(M, x))


@pytest.mark.parametrize("nf", [6, 30])
def test_one_matrix_on_two_streams(gpu, nf):
    """Staged applies of one matrix, their largest class on the caller's stream and the
    others on shared ones, from two streams in turn."""
    import torch
    M = _rows_matrix(gpu, _lens(30), 4000, 31)
    M.prepare(2)
    streams = [torch.cuda.Stream() for _ in range(2)]
    xs = [torch.randn((nf, 4000), device="cuda") for _ in range(2)]
    want = [gpu.apply_f32split(M, x, fields_per_pass=0, unroll=1, variant=4) for x in xs]
    torch.cuda.synchronize()
    ys = [[torch.full((nf, M.n_dst), float("nan"), device="cuda") for _ in range(8)] for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(8):
        for q, s in enumerate(streams):
            with torch.cuda.stream(s):
                gpu.apply_f32split(M, xs[q], ys[q][k], fields_per_pass=0, unroll=4, variant=3 if k % 2 else 1)
    torch.cuda.synchronize()
    for q in range(2):
        for y in ys[q]:
            assert torch.equal(y, want[q])


def test_autotuned_choice_of_small_work(gpu):
    """Small work of more than eight fields: whatever is chosen (the direct kernel's own
    form is among the candidates) gives the same bits and is kept."""
    import torch
    M = _rows_matrix(gpu, np.random.default_rng(40).choice(SHORT, 1000), 900, 41)
    x = torch.randn((12, 900), device="cuda")
    want = gpu.apply_f32split(M, x)
    y = torch.empty_like(want)
    best = gpu.autotune_f32split(M, x, y)
    assert torch.equal(gpu.apply_f32split(M, x), want)
    assert gpu.get_kernel_choice(M, 12)["cached"] is True and best is not None
