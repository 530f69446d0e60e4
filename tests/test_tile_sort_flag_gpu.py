"""Buckets that were not filled as counted: the tile sort raises the table flag, leaves those buckets alone, and every
other bucket is either in order or untouched, never half of each, although blocks of the same launch read the
flag while it is raised. The sort is compiled by itself (no call of the library fills a bucket wrongly)."""

from __future__ import annotations

import ctypes
import importlib
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
FLAGS, TABLE, WORDS = 1, 2, 16


@pytest.fixture(scope="module")
def tile_sort(tmp_path_factory, cuda_device):
    build = importlib.import_module("us3d_b200.build")
    so = tmp_path_factory.mktemp("sort") / "probe.so"
    flags = [f for f in build.NVCC_FLAGS if f != "-lineinfo"]
    subprocess.run([build._nvcc(), *flags, "-cudart", "shared", "-I", str(build.CSRC_DIR), "-I", str(build.INCLUDE_DIR),
                    str(ROOT / "tests" / "tile_sort_probe.cu"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so), mode=ctypes.RTLD_LOCAL).tile_sort
    fn.argtypes = [ctypes.c_int64] * 2 + [ctypes.c_void_p] * 8
    return fn


@pytest.mark.parametrize("n_elems", [4000, 1 << 21])  # with and without packed keys
@pytest.mark.parametrize("wrong", [[], [0], [2500], list(range(0, 5000, 50))])
def test_wrong_fills_are_flagged(wrong, n_elems, tile_sort, cuda_device):
    rng = np.random.default_rng(len(wrong))
    T = 5000
    size = rng.integers(0, 400, T)
    size[wrong] = 200
    start = np.concatenate([[0], np.cumsum(size)]).astype(np.int32)
    n = int(start[-1])
    tile = np.repeat(np.arange(T), size)
    keys = (rng.integers(0, 1 << 31, n).astype(np.uint64) << np.uint64(32)) | rng.integers(0, n_elems, n).astype(np.uint64)
    cursor = size.copy()
    cursor[wrong] -= rng.integers(1, 3, len(wrong))
    d = lambda a, t: torch.as_tensor(np.ascontiguousarray(a).view(t)).to(cuda_device)  # noqa: E731
    t_start, t_count, t_cursor = d(start, np.int32), d(size.astype(np.int32), np.int32), d(cursor.astype(np.int32), np.int32)
    t_keys, inst = d(keys, np.int64), torch.arange(n, dtype=torch.int32, device=cuda_device)
    gid, sorted_inst = (torch.full((n,), -1, dtype=torch.int32, device=cuda_device) for _ in range(2))
    header = torch.zeros(WORDS, dtype=torch.int64, device=cuda_device)
    torch.cuda.synchronize()
    rc = tile_sort(T, n_elems, *(x.data_ptr() for x in (t_start, header, t_keys, inst, gid, sorted_inst, t_count,
                                                        t_cursor)))
    assert rc == 0
    assert int(header[FLAGS]) == (TABLE if wrong else 0)
    got = gid.cpu().numpy()
    order = np.lexsort((keys, tile))
    want = (keys[order] & np.uint64(0xFFFFFFFF)).astype(np.int32)
    same = np.bincount(tile, got == want, T) == size
    left = np.bincount(tile, got == -1, T) == size
    assert (same | left).all() and left[wrong].all()
    if not wrong:
        assert same.all()
        np.testing.assert_array_equal(sorted_inst.cpu().numpy(), order)
    # once raised, the flag turns the whole sort away
    gid.fill_(-1)
    header[FLAGS] = TABLE
    torch.cuda.synchronize()
    assert tile_sort(T, n_elems, *(x.data_ptr() for x in (t_start, header, t_keys, inst, gid, sorted_inst, t_count,
                                                          t_cursor))) == 0
    assert (gid == -1).all()
