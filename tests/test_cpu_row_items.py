"""The FP64 apply's map from warps to (tile of fields, slice of rows)
(helm-project_gb300/csrc/row_items.hpp), compiled alone with g++ and walked
over the whole blocks a launch starts, the surplus warps of its last block
included: every item is taken once, and no warp that goes on lies past the
slices, where the row order ends."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "helm-project_gb300", "csrc")


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("items") / "libitems.so")
    subprocess.run([gxx, "-std=c++20", "-O2", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "native", "row_items_harness.cpp"), "-o", out], check=True)
    lib = C.CDLL(out)
    P = C.POINTER(C.c_int)
    lib.row_items_walk.argtypes = [C.c_longlong] * 5 + [P, P]
    lib.row_items_walk.restype = C.c_longlong

    def run(n_long, F, n_slices, nrhs, tile):
        long_hits = np.zeros(max(1, n_long * -(-nrhs // F)), np.int32)
        hits = np.zeros(n_slices * -(-nrhs // tile), np.int32)
        bad = lib.row_items_walk(n_long, F, n_slices, nrhs, tile, *(a.ctypes.data_as(P) for a in (long_hits, hits)))
        return bad, long_hits, hits

    return run


@pytest.mark.parametrize("n_long", [0, 1, 5, 64])
@pytest.mark.parametrize("n_slices", [1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 16384])
def test_every_item_once_and_none_past_the_rows(walk, n_long, n_slices):
    for F, nrhs, tile in [(1, 1, 4), (2, 2, 4)] + [(4, n, t) for t in (4, 8, 16, 64)
                                                   for n in (3, 4, 5, 7, 8, 9, 15, 16, 17, 63, 64, 65, 130)]:
        bad, long_hits, hits = walk(n_long, F, n_slices, nrhs, tile)
        assert bad == 0, (F, nrhs, tile)
        assert np.all(hits == 1), (F, nrhs, tile)
        assert n_long == 0 or np.all(long_hits == 1), (F, nrhs, tile)
