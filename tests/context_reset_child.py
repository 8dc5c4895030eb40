"""Child of tests/test_gpu_context_reset.py: the same calls before and after
the device's primary context is reset (what cudaDeviceReset does), on new
handles, with the same results. Device memory comes from the driver API, so
nothing but the library keeps state across the reset."""
import ctypes as C
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path[:0] = [ROOT, os.path.join(ROOT, "helm-project_gb300")]

import numpy as np  # noqa: E402

import axgb  # noqa: E402
from axgb import grids  # noqa: E402

cu = C.CDLL("libcuda.so.1")


def drv(name, *args):
    rc = getattr(cu, name)(*args)
    assert rc == 0, (name, rc)


def renumbered():
    """A matrix whose split applies gather the sources into scratch first."""
    n_src, n_dst = 20003, 9000
    rng = np.random.default_rng(51)
    perm = rng.permutation(n_src)
    lens = rng.integers(1, 8, n_dst)
    rp = np.concatenate([[0], np.cumsum(lens)])
    start = np.minimum(np.arange(n_dst) * n_src // n_dst, n_src - 8)
    col = np.concatenate([np.sort(perm[s:s + n]) for s, n in zip(start, lens)])
    return axgb.Matrix.from_csr(n_src, n_dst, rp, col, rng.uniform(0.1, 1.0, rp[-1]))


def apply_all(M, nf):
    x = np.random.default_rng(1).standard_normal((nf, M.n_src)).astype(np.float32)
    y = np.empty((nf, M.n_dst), np.float32)
    dx, dy = C.c_uint64(), C.c_uint64()
    drv("cuMemAlloc_v2", C.byref(dx), C.c_size_t(x.nbytes))
    drv("cuMemAlloc_v2", C.byref(dy), C.c_size_t(y.nbytes))
    drv("cuMemcpyHtoD_v2", dx, x.ctypes.data_as(C.c_void_p), C.c_size_t(x.nbytes))
    out = []
    for v, u in ((3, 4), (1, 4), (2, 4), (0, 4), (4, 1), (5, 32)):
        rc = axgb.lib().axgb_apply_f32split_tuned(M.handle, C.c_void_p(dx.value), C.c_int64(M.n_src), C.c_void_p(dy.value),
                                                  C.c_int64(M.n_dst), C.c_int64(nf), v, 0, u, None)
        assert rc == 0, axgb.last_error()
        drv("cuMemcpyDtoH_v2", y.ctypes.data_as(C.c_void_p), dy, C.c_size_t(y.nbytes))
        out.append(y.copy())
    drv("cuMemFree_v2", dx)
    drv("cuMemFree_v2", dy)
    return out


def everything(handles):
    axgb.init(0)
    A = axgb.Mesh.from_grid(grids.cubed_sphere(96))
    B = axgb.Mesh.from_grid(grids.regular_latlon(720, 360))
    M = axgb.generate_weights(A, B, {"method": "conservative"})
    csr = M.to_csr()  # large enough for the threaded export
    R = renumbered()
    out = [csr[k] for k in sorted(csr)] + apply_all(M, 40) + apply_all(R, 12)
    handles += [A, B, M, R]
    return out


if __name__ == "__main__":
    kept = []
    first = everything(kept)
    if sys.argv[1] == "destroyed":  # every handle is given up before the reset, or none
        kept.clear()
    drv("cuDevicePrimaryCtxReset_v2", 0)
    again = everything([])
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
    print("same", flush=True)
    os._exit(0)  # the old handles' memory went with the context
