"""Calls of one handle queued on several streams."""
import pytest
import torch

from platoanalyze_b200 import capi
from platoanalyze_b200.problem import EllipticProblem
from platoanalyze_b200.workloads import cantilever, splitmix_uniform

pytestmark = pytest.mark.gpu


def _setup(size, count):
    p = EllipticProblem(cantilever(*size))
    z = p.to_dev(splitmix_uniform(p.num_nodes, 3, 0.2, 1.0))
    g = torch.Generator(device="cuda").manual_seed(7)
    us = [torch.rand(p.num_dofs, generator=g, device="cuda", dtype=torch.float64) for _ in range(count)]
    return p, z, us


@pytest.mark.parametrize("size", [(7, 3, 2), (40, 20, 20), (100, 50, 50)], ids=str)
def test_calls_queued_on_two_streams(size):
    """Calls that follow one another on different streams without a wait of the caller's give the bits of the
    same calls on one stream (fixed orders of all sums)."""
    p, z, us = _setup(size, 12)
    calls = [lambda u: p.vf_value(u, z), lambda u: p.sf_gradient_u(u, z), lambda u: p.sf_gradient_z(u, z),
             lambda u: p.apply_operator(z, u, capi.OPERATOR_MATRIX_FREE)]
    want = [calls[k % 4](u) for k, u in enumerate(us)]
    torch.cuda.synchronize()
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for k, u in enumerate(us):
        with torch.cuda.stream(streams[2 * k % 3]):
            p.set_stream(streams[2 * k % 3])
            got.append(calls[k % 4](u))
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_a_captured_call_between_others():
    """A call under stream capture, after one on the default stream and before others: its replays and they agree."""
    p, z, us = _setup((40, 20, 20), 3)
    want = [p.vf_value(u, z) for u in us]
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    u = us[1].clone()
    with torch.cuda.graph(graph, stream=side):
        p.set_stream(torch.cuda.current_stream())
        out = p.vf_value(u, z)
    p.set_stream(torch.cuda.current_stream())
    first = p.vf_value(us[0], z)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(first, want[0]) and torch.equal(out, want[1])
    u.copy_(us[2])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[2]) and torch.equal(p.vf_value(us[0], z), want[0])
