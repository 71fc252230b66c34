"""Calls whose buffers share memory: an output over the activation, and projections of one call that write or add to the same
output. Launches that read and write such memory at once would race, so the results must be those of separate buffers and of calls
made one after the other, up to the order of fp32 sums."""
import pytest

pytestmark = pytest.mark.gpu

SEED = 20265


def _job(rt, tensor, n, k, offset):
    from qwen38_metal_b200.runtime import MappedQ4AffineJob

    w = rt.alloc_shard(n * (k // 2) + offset)
    s = rt.alloc_shard(n * (k // 64) * 2 + offset)
    b = rt.alloc_shard(n * (k // 64) * 2 + offset)
    job = MappedQ4AffineJob(w, offset, s, offset, b, offset, n, offset % 4 == 0)
    rt.synth_q4(SEED, tensor, 0.02, 0, n, k, job)
    return job


@pytest.mark.parametrize("m", [1, 4, 9, 40])
@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("add", [True, False])
def test_output_over_the_activation(runtime, oracle, m, offset, add):
    import torch

    from qwen38_metal_b200 import capi

    k = 2048
    job = _job(runtime, offset, k, k, offset)
    stream = torch.cuda.current_stream().cuda_stream
    flags = capi.FLAG_ACCUMULATE if add else 0
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(m), device="cuda")
    out = x.clone()
    runtime.matmul_batch_device(x.data_ptr(), capi.Q4B_F32, m, k, [job], [out.data_ptr()], flags, stream)
    runtime.device_status()
    for _ in range(3):
        same = x.clone()
        runtime.matmul_batch_device(same.data_ptr(), capi.Q4B_F32, m, k, [job], [same.data_ptr()], flags, stream)
        runtime.device_status()
        # (up to 15 rows another kernel takes the call: fp32 sums in another order)
        assert oracle.rel_l2(same.cpu().numpy(), out.cpu().numpy()) <= (2e-6 if m < 16 else 0.0)


@pytest.mark.parametrize("m", [1, 4, 9, 40])
@pytest.mark.parametrize("add", [True, False])
def test_projections_that_share_an_output(runtime, m, add):
    import torch

    from qwen38_metal_b200 import capi

    n, k = 3000, 1024
    jobs = [_job(runtime, 10 + i, n, k, (0, 2, 0)[i]) for i in range(3)]
    stream = torch.cuda.current_stream().cuda_stream
    flags = capi.FLAG_ACCUMULATE if add else 0
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    start = [torch.randn(m, n, generator=gen, device="cuda") for _ in range(2)]

    def outputs():
        return [s.clone() for s in start]

    want = outputs()
    for job, o in zip(jobs, (want[0], want[1], want[0])):
        runtime.matmul_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, [job], [o.data_ptr()], flags, stream)
    runtime.device_status()
    for _ in range(3):
        got = outputs()
        runtime.matmul_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, jobs, [got[0].data_ptr(), got[1].data_ptr(), got[0].data_ptr()], flags, stream)
        runtime.device_status()
        for a, b in zip(got, want):
            # (which projections share a launch decides how K is cut: fp32 sums in another order)
            assert float((a - b).double().norm() / b.double().norm()) <= 2e-6
