"""The CTA-pair tensor-core GEMM at the sizes where it can go wrong: activation rows and weight rows around tile edges, odd
numbers of affine groups, tiles cut along K between workers, several projections of different alignment in one launch,
and the fused gate/up form with ragged rows. Tolerances are the ones of the path: the oracle that rounds weights to bf16
differs only by the order of fp32 sums (2e-4), and by last-place flips of the bf16 hidden rows in the MLP (5e-4)."""
import numpy as np
import pytest

from helpers import upload_matrix

pytestmark = pytest.mark.gpu

SEED = 20261


@pytest.mark.parametrize("m,k,rows,offsets", [
    (17, 64, (1, 255), (0, 2)),          # one group: a stage of one group; fewest stages
    (32, 192, (256, 257), (8, 0)),       # odd number of groups
    (33, 320, (128, 513, 40), (0, 6, 2)),
    (128, 1088, (300,), (15,)),          # two accumulators, odd byte offset
    (129, 1024, (511, 64), (0, 0)),
    (257, 704, (700,), (2,)),            # two activation tiles
    (40, 17408, (300,), (0,)),           # few tiles, long rows: cut into many parts
    (520, 2112, (3000, 2500), (2, 0)),   # whole tiles, then a tail cut into runs of any length
])
def test_tile_edges(runtime, oracle, m, k, rows, offsets):
    bits = oracle.synth_bf16(SEED, 5000 + m, m * k)
    x = oracle.bf16_to_f32(bits).reshape(m, k)
    trips = [oracle.synth_q4(SEED, 100 * m + i, n, k) for i, n in enumerate(rows)]
    jobs = [upload_matrix(runtime, *t, offset=o) for t, o in zip(trips, offsets)]
    outs = runtime.q4_affine_matmul_mapped_batch(bits, m, jobs)
    again = runtime.q4_affine_matmul_mapped_batch(bits, m, jobs)
    added = runtime.q4_affine_matmul_add_mapped_batch(bits, m, jobs, [np.full((m, n), 2.0, dtype=np.float32) for n in rows])
    for out, rep, add, t, n in zip(outs, again, added, trips, rows):
        assert oracle.rel_l2(out, oracle.matmul_bf16_tiles(x, *t, n, threads=8)) <= 2e-4
        assert np.array_equal(out, rep)  # parts of cut tiles are added in a fixed order
        assert np.allclose(add, out + 2.0, rtol=0, atol=1e-5)


@pytest.mark.parametrize("m,k,inter,n,offset", [(17, 192, 64, 65, 0), (100, 512, 192, 300, 2), (300, 1024, 1088, 130, 8)])
def test_fused_gate_up_ragged(runtime, oracle, m, k, inter, n, offset):
    bits = oracle.synth_bf16(SEED, 6000 + m, m * k)
    x = oracle.bf16_to_f32(bits).reshape(m, k)
    gate, up, down = (oracle.synth_q4(SEED, 200 * m + i, r, c) for i, (r, c) in enumerate(((inter, k), (inter, k), (n, inter))))
    jobs = [upload_matrix(runtime, *t, offset=offset) for t in (gate, up, down)]
    out = runtime.q4_affine_mlp_mapped_batch(bits, m, *jobs)
    h = oracle.swiglu(oracle.matmul_bf16_tiles(x, *gate, inter), oracle.matmul_bf16_tiles(x, *up, inter))
    h = oracle.bf16_to_f32(oracle.f32_to_bf16(h)).reshape(m, inter)
    assert oracle.rel_l2(out, oracle.matmul_bf16_tiles(h, *down, n, threads=8)) <= 5e-4
