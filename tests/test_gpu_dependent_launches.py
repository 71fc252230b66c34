"""Programmatic dependent launches: a kernel may start while the one in front still runs, so each has to wait before it reads what
came before. A row of calls whose intermediate buffers are used again and again must give the bits that the same calls give
with the device idle between them."""
import pytest

pytestmark = pytest.mark.gpu

SEED = 20264


def _job(rt, tensor, n, k, offset):
    from qwen38_metal_b200.runtime import MappedQ4AffineJob

    w = rt.alloc_shard(n * (k // 2) + offset)
    s = rt.alloc_shard(n * (k // 64) * 2 + offset)
    b = rt.alloc_shard(n * (k // 64) * 2 + offset)
    job = MappedQ4AffineJob(w, offset, s, offset, b, offset, n, offset % 4 == 0)
    rt.synth_q4(SEED, tensor, 0.02, 0, n, k, job)
    return job


@pytest.mark.parametrize("m", [1, 5, 40])
@pytest.mark.parametrize("captured", [False, True])
def test_a_row_of_calls_reads_what_the_call_before_wrote(runtime, m, captured):
    import torch

    from qwen38_metal_b200 import capi

    k, inter, vocab, rounds = 1024, 2048, 3000, 12
    gate, up, down, head = (_job(runtime, i, n, c, o) for i, (n, c, o) in enumerate(((inter, k, 0), (inter, k, 2), (k, inter, 0), (vocab, k, 2))))
    f32 = lambda *shape: torch.zeros(*shape, device="cuda")
    x, h = torch.zeros(m, k, dtype=torch.bfloat16, device="cuda"), torch.zeros(m, inter, dtype=torch.bfloat16, device="cuda")
    g, u, d = f32(m, inter), f32(m, inter), f32(m, k)
    tokens, values = torch.zeros(rounds, m, dtype=torch.int32, device="cuda"), f32(rounds, m)
    seen = [f32(m, k) for _ in range(rounds)]
    start = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(m), device="cuda").to(torch.bfloat16)
    stream = torch.cuda.Stream()
    raw = stream.cuda_stream

    def rows(wait):
        idle = (lambda: torch.cuda.synchronize()) if wait else (lambda: None)
        with torch.cuda.stream(stream):
            x.copy_(start)
            for i in range(rounds):
                runtime.matmul_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, [gate, up], [g.data_ptr(), u.data_ptr()], 0, raw)
                idle()
                runtime.swiglu_device(g.data_ptr(), u.data_ptr(), m * inter, 0, h.data_ptr(), raw)
                idle()
                runtime.matmul_batch_device(h.data_ptr(), capi.Q4B_BF16, m, inter, [down], [d.data_ptr()], 0, raw)
                idle()
                seen[i].copy_(d)
                runtime.rms_unit_bf16_device(d.data_ptr(), m, k, 1e-6, x.data_ptr(), raw)
                idle()
                runtime.argmax_batch_device(x.data_ptr(), capi.Q4B_BF16, m, k, head, 0, tokens[i].data_ptr(), values[i].data_ptr(), raw)
                idle()

    torch.cuda.synchronize()
    rows(wait=True)
    runtime.device_status()
    expected = [t.clone() for t in seen] + [tokens.clone(), values.clone()]
    assert len({float(t.double().sum()) for t in seen}) == rounds  # every round has other data
    run = lambda: rows(wait=False)
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            rows(wait=False)
        run = graph.replay
    for _ in range(3):
        for t in seen + [tokens, values, x, h, g, u, d]:
            t.zero_()
        torch.cuda.synchronize()
        run()
        runtime.device_status()
        for got, ref in zip(seen + [tokens, values], expected):
            assert torch.equal(got, ref)


@pytest.mark.parametrize("m,offset", [(1, 0), (1, 2), (4, 0), (8, 2)])
def test_calls_wait_for_weights_that_the_caller_can_write(runtime, m, offset):
    """Asking for a shard's address makes the calls that use it wait for the kernel in front before they read weights. A copy of
    the caller's into the shard, directly in front of the call, is what the call computes with."""
    import torch

    from qwen38_metal_b200 import capi

    n, k = 512, 1024
    job, other = _job(runtime, 20, n, k, offset), _job(runtime, 21, n, k, offset)
    x = torch.randn(m, k, generator=torch.Generator(device="cuda").manual_seed(m), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def call(j):
        out = torch.zeros(m, n, device="cuda")
        runtime.matmul_batch_device(x.data_ptr(), capi.Q4B_F32, m, k, [j], [out.data_ptr()], 0, stream)
        return out

    first, second = call(job), call(other)
    assert "weights_ahead=1" in runtime.describe_dispatch(capi.Q4B_F32, m, k, [job])
    fresh = [torch.from_numpy(runtime.read_shard(b, 0, b.length)).cuda() for b in (other.weights, other.scales, other.biases)]
    torch.cuda.synchronize()

    class Raw:  # a shard as torch sees memory
        def __init__(self, buf):
            self.__cuda_array_interface__ = {"shape": (buf.length,), "typestr": "|u1", "data": (runtime.shard_pointer(buf), False), "version": 3}

    shards = [torch.as_tensor(Raw(b), device="cuda") for b in (job.weights, job.scales, job.biases)]
    for s, f in zip(shards, fresh):
        torch.add(f, 0, out=s)  # a kernel, not a copy
    again = call(job)
    runtime.device_status()
    assert "weights_ahead=0" in runtime.describe_dispatch(capi.Q4B_F32, m, k, [job])
    assert "weights_ahead=1" in runtime.describe_dispatch(capi.Q4B_F32, m, k, [other])
    assert torch.equal(again, second) and not torch.equal(first, second)
