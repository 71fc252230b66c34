"""The short-batch kernel's byte-addressed instance: tensors at any byte offset, any whole number of affine groups, single
rows that add to their output, and activations that are not finite. Bar: relative L2 <= 1e-5 of the 64-bit result, as for
aligned tensors (group sums are exact integers, about 1e-7 is seen)."""
import numpy as np
import pytest

from helpers import upload_in_one_shard, upload_matrix

pytestmark = pytest.mark.gpu

SEED = 20262


@pytest.mark.parametrize("offset", [1, 2, 3, 4, 6, 8, 11, 12, 14, 15])
@pytest.mark.parametrize("m", [2, 9])
def test_every_offset(runtime, oracle, m, offset):
    n, k = 75, 1536
    trip = oracle.synth_q4(SEED, offset, n, k)
    job = upload_matrix(runtime, *trip, offset=offset)
    assert "rows_i8" in runtime.describe_dispatch(0, m, k, [job])
    x = np.random.default_rng(offset).standard_normal((m, k)).astype(np.float32)
    out = runtime.q4_affine_matmul_mapped_batch(x.reshape(-1), m, [job])[0]
    assert oracle.rel_l2(out, oracle.matmul_f64(x, *trip, n)) <= 1e-5


@pytest.mark.parametrize("k", [64, 128, 192, 448, 576, 1600, 5184, 17408 + 64])
@pytest.mark.parametrize("m,offset", [(2, 0), (5, 2), (8, 13), (15, 6)])
def test_any_number_of_groups(runtime, oracle, m, offset, k):
    """Odd group counts leave half a last chunk, and every parameter row has a boundary of its own; the three tensors of
    both projections lie back to back in one shard, so their offsets differ too."""
    shapes = (33, 500)
    trips = [oracle.synth_q4(SEED, 40 + i, n, k) for i, n in enumerate(shapes)]
    jobs = upload_in_one_shard(runtime, trips, offset)
    x = np.random.default_rng(k + m).standard_normal((m, k)).astype(np.float32)
    for _ in range(2):
        outs = runtime.q4_affine_matmul_mapped_batch(x.reshape(-1), m, jobs)
        for out, trip, n in zip(outs, trips, shapes):
            assert oracle.rel_l2(out, oracle.matmul_f64(x, *trip, n)) <= 1e-5


@pytest.mark.parametrize("k,offset", [(512, 0), (704, 2), (17408, 2), (4096, 6)])
def test_single_row_that_adds(runtime, oracle, k, offset):
    n = 301
    trip = oracle.synth_q4(SEED, 60, n, k)
    job = upload_matrix(runtime, *trip, offset=offset)
    x = np.random.default_rng(k).standard_normal((1, k)).astype(np.float32)
    res = np.random.default_rng(k + 1).standard_normal((1, n)).astype(np.float32)
    out = runtime.q4_affine_matmul_add_mapped_batch(x.reshape(-1), 1, [job], [res.copy()])[0]
    assert oracle.rel_l2(out, oracle.matmul_f64(x, *trip, n) + res) <= 1e-5


@pytest.mark.parametrize("offset", [0, 2])
def test_outliers_and_non_finite_inputs(runtime, oracle, offset):
    """A channel a million times the rest costs the other groups no precision (its own group: the test below); an infinity or a
    NaN reaches every result of its own row and no other row."""
    n, k, m = 96, 1024, 5
    trip = oracle.synth_q4(SEED, 70, n, k)
    x = np.random.default_rng(3).standard_normal((m, k)).astype(np.float32)
    x[0, 100] = 1e6
    trip[1][:, 1] = 0  # the outlier's group has scale and bias zero: what is left are the ordinary inputs
    trip[2][:, 1] = 0
    job = upload_matrix(runtime, *trip, offset=offset)
    x[1] *= np.float32(1e37)
    x[2] *= np.float32(1e-30)
    x[3, 777] = np.inf
    x[4, 5] = np.nan
    out = runtime.q4_affine_matmul_mapped_batch(x.reshape(-1), m, [job])[0]
    ref = oracle.matmul_f64(x[:3], *trip, n)
    for r in range(3):
        assert oracle.rel_l2(out[r], ref[r]) <= 1e-5, r
    assert not np.isfinite(out[3:]).any()


@pytest.mark.parametrize("m,offset", [(1, 0), (2, 0), (4, 2), (8, 2), (12, 6)])
def test_fp32_inputs_keep_their_bits(runtime, oracle, m, offset):
    """fp32 inputs in four digits: what is left is the fp32 accumulation of K / 64 groups, two roundings of 2^-24 each, which
    add up to about sqrt(2 K / 64) 2^-24 / sqrt(3) = 1.9e-7 (three digits alone would leave 3e-7)."""
    n, k = 256, 1024
    trip = oracle.synth_q4(SEED, 80, n, k)
    job = upload_matrix(runtime, *trip, offset=offset)
    x = np.random.default_rng(m).standard_normal((m, k)).astype(np.float32)
    out = runtime.q4_affine_matmul_mapped_batch(x.reshape(-1), m, [job])[0]
    assert oracle.rel_l2(out.reshape(m, n), oracle.matmul_f64(x, *trip, n)) <= 1.9e-7


def _zero_weight_at(trip, index):
    """Weight zero (q = 8, bias = -8 scale) for input `index` of every group, in every row; the other weights stay live."""
    w, s, b = trip
    word, shift = index // 8, np.uint32(4 * (index % 8))
    w[:, word::8] = (w[:, word::8] & ~(np.uint32(15) << shift)) | (np.uint32(8) << shift)
    b[:] = (s + np.uint16(3 << 7)) ^ np.uint16(0x8000)  # bf16: three more in the exponent, sign flipped
    return trip


@pytest.mark.parametrize("spread", [1e3, 1e4, 1e5])
@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("m,k,offset", [(1, 5120, 0), (1, 5120, 2), (2, 5120, 2), (3, 5184, 0), (8, 5120, 2), (13, 5120, 2), (15, 5184, 6)])
def test_a_large_input_with_zero_weight_costs_its_neighbours_little(runtime, oracle, m, k, offset, bf16, spread):
    """One input far above its 63 neighbours, whose own weight is zero: what is left of its group is the neighbours' sum. Bar:
    that of the path, 1e-5. The step of four digits is 2^-30 of the power of two above the large input and inputs are off by
    0.29 of it (rms) against a standard deviation of 1, in one group of K / 64: 2^-30 * 131072 * 0.29 / sqrt(80) = 4e-6 at
    a spread of 1e5. Residual form, so that single rows take this kernel at every size."""
    n = 200
    trip = _zero_weight_at(oracle.synth_q4(SEED, 90, n, k), 37)
    job = upload_matrix(runtime, *trip, offset=offset)
    x = np.random.default_rng(m).standard_normal((m, k)).astype(np.float32)
    x[:, 64 + 37] = spread
    given = x.reshape(-1)
    if bf16:
        given = oracle.f32_to_bf16(given)
        x = oracle.bf16_to_f32(given).reshape(m, k)
    out = runtime.q4_affine_matmul_add_mapped_batch(given, m, [job], [np.zeros((m, n), dtype=np.float32)])[0].reshape(m, n)
    ref = oracle.matmul_f64(x, *trip, n)
    for r in range(m):
        assert oracle.rel_l2(out[r], ref[r]) <= 1e-5, r


@pytest.mark.parametrize("n", [40, 5120, 16368, 16400])
@pytest.mark.parametrize("offset", [0, 2])
def test_single_rows_take_one_kernel_up_to_lm_head(runtime, oracle, n, offset):
    """A plain single row takes the kernel that the residual form takes, so both give the same bits, and neither size nor offset
    changes how its inputs are held (bar: as above, 1e-5 with one input of 1e4 and a weight of zero beside it)."""
    k = 512
    trip = _zero_weight_at(oracle.synth_q4(SEED, 92, n, k), 37)
    job = upload_matrix(runtime, *trip, offset=offset)
    x = np.random.default_rng(n).standard_normal((1, k)).astype(np.float32)
    x[0, 37] = 1e4
    bits = oracle.f32_to_bf16(x.reshape(-1))
    for given, held in ((x.reshape(-1), x), (bits, oracle.bf16_to_f32(bits).reshape(1, k))):
        out = runtime.q4_affine_matvec_mapped_batch(given, [job])[0]
        added = runtime.q4_affine_matmul_add_mapped_batch(given, 1, [job], [np.zeros((1, n), dtype=np.float32)])[0]
        assert np.array_equal(out, added.reshape(-1))
        assert oracle.rel_l2(out, oracle.matmul_f64(held, *trip, n)) <= 1e-5
