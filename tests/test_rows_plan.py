"""The short-batch kernel's cut of a launch into runs of quads (csrc/q4_decomp.h), followed on the CPU: every quad of every
tile is taken by exactly one warp, and what a warp that finishes a shared tile expects -- how many contributions, in
which scratch slots -- is what the other warps do."""
import ctypes as C
import os
import subprocess
from collections import defaultdict

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("shim") / "libdecomp.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "decomp_shim.cpp")], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("k", [64, 192, 512, 1600, 5120, 5184, 17408])
@pytest.mark.parametrize("tiles", [1, 3, 64, 320, 533, 2176, 15520])
@pytest.mark.parametrize("cap,mp", [(102, 2), (78, 2), (48, 2), (51, 4), (24, 4), (26, 8), (12, 8), (13, 16)])  # what a block holds
def test_every_quad_once_and_shares_agree(shim, k, tiles, cap, mp):
    sms = 148
    cpt = (k // 64 + 1) // 2
    longest = C.c_uint32(0)
    parts = shim.shim_rows_plan(cpt, tiles, sms, cap, mp, C.byref(longest))
    assert 1 <= parts <= 32 and longest.value <= cap
    run = shim.shim_rows_run(tiles, longest.value, parts, sms)
    slots = shim.shim_rows_part_slots(cpt, parts, run)
    assert run >= 1
    for part in range(parts):
        lo, hi = shim.shim_rows_part_begin(cpt, parts, part), shim.shim_rows_part_begin(cpt, parts, part + 1)
        assert lo % 4 == 0 and lo < hi and hi - lo <= longest.value
        quads = (hi - lo + 3) // 4
        seen = defaultdict(list)
        taken = 0
        for worker in range(sms // parts * 16):
            u = min(worker * run, tiles * quads)
            end = min(u + run, tiles * quads)
            while u < end:
                tile = u // quads
                stop = min(end, (tile + 1) * quads)
                taken += stop - u
                seen[tile].append(worker - tile * quads // run)
                u = stop
        assert taken == tiles * quads
        for tile in range(tiles):
            assert seen[tile] == list(range(shim.shim_rows_shares(tile, quads, run)))
            assert len(seen[tile]) <= slots


@pytest.mark.parametrize("cap", [78, 48])  # aligned, byte-addressed
def test_single_rows_fit_the_scratch_a_runtime_sets_aside(shim, cap):
    """8 MB of partial sums (two padded rows, fp32) and 16384 tile counters hold any single row of up to 8192 inputs and 2^18
    outputs, so that a decode call does not allocate."""
    longest = C.c_uint32(0)
    for k in (64, 512, 1600, 4096, 5120, 6144, 8192):
        cpt = (k // 64 + 1) // 2
        for tiles in list(range(1, 400)) + list(range(400, 16384, 97)) + [16384]:
            parts = shim.shim_rows_plan(cpt, tiles, 148, cap, 2, C.byref(longest))
            slots = shim.shim_rows_part_slots(cpt, parts, shim.shim_rows_run(tiles, longest.value, parts, 148))
            assert parts * slots * 2 * tiles * 64 <= 8 << 20, (k, tiles)


def test_a_launch_with_more_quads_than_32_bits_is_refused(shim):
    longest = C.c_uint32(0)
    assert shim.shim_rows_plan(136, 0xFFFFFFF, 148, 92, 2, C.byref(longest)) == 0
