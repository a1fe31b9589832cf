"""The Katsevich filter under capture, with buffers that overlap in part (the copy is then a node of
the graph)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 5, -1000])
def test_captured_overlapping_buffers(shift):
    import torch

    from fastcone_b200 import ops
    from fastcone_b200.geometry import ConeGeometry

    g = ConeGeometry.helical((48, 48, 40), 1.0, (96, 24), 1.0, 150.0, 300.0, 3, 80, 24.0)
    p = torch.rand(g.proj_shape, device="cuda")
    plan = ops.KatsevichPlan(g)
    buf = torch.zeros(p.numel() + 2000, device="cuda")
    a = buf[1000:1000 + p.numel()].view(g.proj_shape)
    b = buf[1000 + shift:1000 + shift + p.numel()].view(g.proj_shape)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.copy_(p)
        plan(a, out=b)
    ref = plan(p.clone())
    for _ in range(2):
        buf.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(b, ref) or float((b - ref).norm() / ref.norm()) < 1e-6
