"""Device calls captured in a CUDA graph: what they hold on to stays valid when later calls on the same runtime need more
scratch than there was at the time of the capture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20263


def _jobs(rt, rows, k, offset=0):
    from qwen38_metal_b200.runtime import MappedQ4AffineJob

    jobs = []
    for i, n in enumerate(rows):
        w = rt.alloc_shard(n * (k // 2) + offset)
        s = rt.alloc_shard(n * (k // 64) * 2 + offset)
        b = rt.alloc_shard(n * (k // 64) * 2 + offset)
        job = MappedQ4AffineJob(w, offset, s, offset, b, offset, n, offset % 4 == 0)
        rt.synth_q4(SEED, i, 0.02, 0, n, k, job)
        jobs.append(job)
    return jobs


# (captured call, larger call): single rows and short batches share the tile sums of the short-batch kernel, prompt rows
# the converted activation and the cut tiles of the tensor-core GEMM
@pytest.mark.parametrize("small,large", [
    ((1, (5120,), 5120, 0), (16, (131072,), 1024, 0)),
    ((1, (17408, 17408), 5120, 2), (16, (131072,), 1024, 0)),
    ((3, (700, 40), 1600, 0), (16, (131072,), 1024, 0)),
    ((40, (2048, 48), 5120, 0), (2100, (17408,), 5120, 0)),
])
def test_captured_call_survives_a_call_that_outgrows_its_scratch(small, large):
    import torch

    from qwen38_metal_b200 import capi
    from qwen38_metal_b200.runtime import CudaRuntime

    rt = CudaRuntime(0)
    stream = torch.cuda.Stream()

    def prepare(m, rows, k, offset):
        gen = torch.Generator(device="cuda").manual_seed(m)
        x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
        return x, m, k, _jobs(rt, rows, k, offset), [torch.zeros(m, n, device="cuda") for n in rows]

    def call(state):
        x, m, k, jobs, outs = state
        rt.matmul_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, jobs, [o.data_ptr() for o in outs], 0, stream.cuda_stream)

    try:
        a, b = prepare(*small), prepare(*large)
        torch.cuda.synchronize()
        call(a)
        rt.device_status()
        first = [o.clone() for o in a[4]]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            call(a)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        call(b)
        rt.device_status()
        assert torch.cuda.mem_get_info()[0] < free - (4 << 20)  # scratch did grow
        other = [o.clone() for o in b[4]]
        for _ in range(2):
            for o in a[4]:
                o.zero_()
            torch.cuda.synchronize()
            graph.replay()
            rt.device_status()
            for o, ref in zip(a[4], first):
                assert torch.equal(o, ref)
            call(b)  # and the larger call is not disturbed either
            rt.device_status()
            for o, ref in zip(b[4], other):
                assert torch.equal(o, ref)
        assert all(np.isfinite(o.cpu().numpy()).all() and float(o.abs().sum()) > 0 for o in first)
    finally:
        rt.close()


def test_first_calls_do_not_allocate():
    """A single row never allocates, and of prompt rows only the converted activation does (once for all calls of its size): the
    scratch for tiles cut between SM pairs is bounded and set aside with the runtime."""
    import torch

    from qwen38_metal_b200 import capi
    from qwen38_metal_b200.runtime import CudaRuntime

    rt = CudaRuntime(0)
    stream = torch.cuda.current_stream().cuda_stream
    try:
        calls = []
        for m, rows, k, offset in ((1, (5120,), 5120, 0), (1, (6144, 1024, 1024), 5120, 2), (600, (256,), 5120, 0), (600, (5000, 300), 5120, 2), (200, (19000,), 5120, 0)):
            x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
            calls.append((x, m, k, _jobs(rt, rows, k, offset), [torch.zeros(m, n, device="cuda") for n in rows]))
        free = []
        for x, m, k, jobs, outs in calls:
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])
            rt.matmul_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, jobs, [o.data_ptr() for o in outs], 0, stream)
            rt.device_status()
        free.append(torch.cuda.mem_get_info()[0])
        assert free[0] == free[1] == free[2]  # single rows
        assert 0 <= free[2] - free[3] <= 16 << 20  # 600 x 5120 bf16, rounded up
        assert free[3] == free[4] == free[5]
    finally:
        rt.close()
