"""The short-batch kernel's cut of a launch into runs of quads (csrc/q4_decomp.h), followed on the CPU: every quad of every
item is taken by exactly one warp, and what a warp that finishes a shared item expects -- how many contributions, in
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
@pytest.mark.parametrize("cap,mp,tw", [(92, 2, 1), (31, 4, 1), (16, 8, 1), (21, 8, 2), (8, 16, 1)])
def test_every_quad_once_and_shares_agree(shim, k, tiles, cap, mp, tw):
    sms = 148
    cpt = (k // 64 + 1) // 2
    longest = C.c_uint32(0)
    parts = shim.shim_rows_plan_for(cpt, tiles, sms, cap, tw, mp, C.byref(longest))
    assert 1 <= parts <= 32 and longest.value <= cap
    items = (tiles + tw - 1) // tw
    run = shim.shim_rows_run(items, longest.value, parts, sms)
    slots = shim.shim_rows_part_slots(cpt, parts, run)
    assert run >= 1
    for part in range(parts):
        lo, hi = shim.shim_rows_part_begin(cpt, parts, part), shim.shim_rows_part_begin(cpt, parts, part + 1)
        assert lo % 4 == 0 and lo < hi and hi - lo <= longest.value
        quads = (hi - lo + 3) // 4
        seen = defaultdict(list)
        taken = 0
        for worker in range(sms // parts * 16):
            u = min(worker * run, items * quads)
            end = min(u + run, items * quads)
            while u < end:
                item = u // quads
                stop = min(end, (item + 1) * quads)
                taken += stop - u
                seen[item].append(worker - item * quads // run)
                u = stop
        assert taken == items * quads
        for item in range(items):
            assert seen[item] == list(range(shim.shim_rows_shares(item, quads, run)))
            assert len(seen[item]) <= slots


@pytest.mark.parametrize("cap", [78, 48])  # aligned, byte-addressed
def test_single_rows_fit_the_scratch_a_runtime_sets_aside(shim, cap):
    """8 MB of partial sums (two padded rows, fp32) and 16384 tile counters hold any single row of up to 8192 inputs and 2^18
    outputs, so that a decode call does not allocate."""
    longest = C.c_uint32(0)
    for k in (64, 512, 1600, 4096, 5120, 6144, 8192):
        cpt = (k // 64 + 1) // 2
        for tiles in list(range(1, 400)) + list(range(400, 16384, 97)) + [16384]:
            parts = shim.shim_rows_plan_for(cpt, tiles, 148, cap, 1, 2, C.byref(longest))
            slots = shim.shim_rows_part_slots(cpt, parts, shim.shim_rows_run(tiles, longest.value, parts, 148))
            assert parts * slots * 2 * tiles * 64 <= 8 << 20, (k, tiles)


def test_a_launch_with_more_quads_than_32_bits_is_refused(shim):
    longest = C.c_uint32(0)
    assert shim.shim_rows_plan_for(136, 0xFFFFFFF, 148, 92, 1, 2, C.byref(longest)) == 0
