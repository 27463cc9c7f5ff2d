"""The benchmark's flow from host buffers to host buffers: results as a synchronous pass gives them, in buffers that are not
filled again before they can be read, and no device memory taken once two steps' buffers are there."""
import pytest
import torch

import bench

pytestmark = pytest.mark.gpu


def test_host_pipeline_takes_no_memory_and_keeps_its_results():
    dev = torch.device("cuda:0")
    n = 1 << 20
    pinned = {"x": torch.zeros(n).pin_memory(), "y": torch.arange(n, dtype=torch.float32).pin_memory()}
    busy = torch.randn(2048, 2048, device=dev)

    def fn(t):
        z = t["x"] + t["y"]                          # outputs and scratch of every step come from the allocator
        for _ in range(8):
            busy @ busy                              # the host queues a step well before the device has done it
        return z * 2, z.long()

    p = bench.HostPipeline(fn, pinned, (torch.empty(n), torch.empty(n, dtype=torch.int64)), dev)
    for _ in range(4):
        p.step()
    p.drain()
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats(dev)["num_device_alloc"]
    seen = []
    for i in range(40):
        out = p.step()
        seen.append(out)
        if i >= 2:                                   # step i began when the results of step i - 2 had arrived in these buffers
            assert out[0] is seen[i - 2][0]
    assert torch.cuda.memory_stats(dev)["num_device_alloc"] == before
    p.drain()
    torch.cuda.synchronize()
    want = torch.arange(n, dtype=torch.float32)
    for doubled, whole in p.results:
        assert torch.equal(doubled, want * 2) and torch.equal(whole, want.long())
