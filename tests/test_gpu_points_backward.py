"""A backward pass that wants only the points' gradient leaves the parameters'
alone: with power and rotation on the host, where fetching theirs would wait
for the GPU, it makes no synchronisation and can be captured into a graph."""
import pytest

from cantucci_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def estimate(cg):
    import torch
    from cantucci_gb300.autograd import mandelbulb_de
    p = torch.as_tensor(W.uniform_points(5003, seed=2)).cuda().requires_grad_(True)
    w = torch.linspace(-1, 1, 5003, device="cuda")

    def run(power_grad=False, rot_grad=False):
        power = torch.tensor(8.3, requires_grad=power_grad)
        rot = torch.tensor([0.1, -0.2, 0.3], requires_grad=rot_grad)
        inputs = [p] + [t for t in (power, rot) if t.requires_grad]
        return torch.autograd.grad(mandelbulb_de(p, power, rot, 15, 2.5), inputs, w)

    return run


def test_points_only_makes_no_synchronisation(estimate):
    import torch
    estimate()
    torch.cuda.synchronize()
    torch.cuda.set_sync_debug_mode("error")
    try:
        estimate()
    finally:
        torch.cuda.set_sync_debug_mode("default")


def test_points_only_is_captured(estimate):
    import torch
    (ref,) = estimate()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        estimate()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        (got,) = estimate()
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int32), ref.view(torch.int32))


@pytest.mark.parametrize("power_grad,rot_grad", [(True, False), (False, True), (True, True)])
def test_each_parameter_alone(estimate, power_grad, rot_grad):
    import torch
    _, gpow, grot = estimate(True, True)
    got = estimate(power_grad, rot_grad)[1:]
    ref = [g for g, want in ((gpow, power_grad), (grot, rot_grad)) if want]
    assert [g.shape for g in got] == [g.shape for g in ref]
    assert all(torch.equal(a, b) and a.device.type == "cpu" for a, b in zip(got, ref))
