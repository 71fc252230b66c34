"""The tensor-core launch plan, checked on the CPU: every (tile, K stage) belongs to exactly one worker, TMEM and scratch
sizes hold (scratch within what a runtime sets aside), for row counts at tile edges, single groups and long rows, few and
many tiles."""
import ctypes as C
import os
import subprocess
import tempfile

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def shim():
    out = os.path.join(tempfile.mkdtemp(prefix="q4gemm"), "shim.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out, os.path.join(ROOT, "tests", "gemm_plan_shim.cpp")])
    lib = C.CDLL(out)
    lib.shim_gemm_plan.argtypes = [C.c_uint32] * 4
    return lib


@pytest.mark.parametrize("m", [1, 17, 32, 33, 128, 129, 256, 257, 333, 1000, 2048])
def test_every_stage_of_every_tile_once(shim, m):
    for k in (64, 128, 192, 1024, 5120, 17408):
        for row_tiles in (1, 2, 20, 41, 73, 74, 75, 136, 147, 148, 149, 221, 970):
            assert shim.shim_gemm_plan(m, k, row_tiles, 74) == 0, (m, k, row_tiles)
