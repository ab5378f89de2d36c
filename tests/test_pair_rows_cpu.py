"""Rows that the CTA-pair kernel loads: all rows of a tile, and none behind the last row block that the sort filled
(sorted activations may be allocated at tokens*topk + experts*tile_m - topk rows, no more)."""
import ctypes
import random
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "flydsl_b200" / "csrc"


@pytest.fixture(scope="module")
def pair_rows(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("pair_rows")
    (d / "f.cpp").write_text('#include "gemm_args.cuh"\n'
                             'extern "C" int f(int blocks, int tile_m, int rank) '
                             '{ return flymoe::pair_rows(blocks, tile_m, rank); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), "-I",
                    str(Path(nvcc).resolve().parents[1] / "include"), str(d / "f.cpp"), "-o", str(d / "f.so")], check=True)
    return ctypes.CDLL(str(d / "f.so")).f


@pytest.mark.parametrize("tile_m", [64, 128])
def test_a_tiles_rows_are_loaded_once_and_nothing_else(pair_rows, tile_m):
    rng = random.Random(tile_m)
    for _ in range(200):
        counts = [rng.choice((0, 1, 63, 64, 65, 128, 129, 192, 255, 256, 257, 300)) for _ in range(rng.randint(1, 6))]
        blocks = [(c + tile_m - 1) // tile_m for c in counts]
        valid_rows = sum(blocks) * tile_m
        loaded, first = [], 0
        for nb in blocks:                                   # an expert's blocks, cut into tiles of 256 rows
            for b in range(0, nb, 256 // tile_m):
                tile_blocks = min(256 // tile_m, nb - b)
                for rank in (0, 1):
                    n = pair_rows(tile_blocks, tile_m, rank)
                    assert n % tile_m == 0
                    start = (first + b) * tile_m + rank * 128
                    loaded += range(start, start + n)
            first += nb
        assert loaded == list(range(valid_rows))
