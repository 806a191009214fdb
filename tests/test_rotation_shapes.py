"""Rotations that are not one scalar per angle are refused before anything is
launched (no GPU needed)."""
import pytest
import torch

from cantucci_gb300 import fit
from cantucci_gb300.autograd import mandelbulb_de

POINTS = torch.zeros((4, 3))


def calls():
    cam = fit.camera(8, 8)
    return {"mandelbulb_de": lambda rot: mandelbulb_de(POINTS, torch.tensor(8.0), rot),
            "depth_render": lambda rot: fit.depth_render(torch.tensor(8.0), rot, cam),
            "surface_loss": lambda rot: fit.surface_loss(torch.tensor(8.0), rot, POINTS)}


@pytest.mark.parametrize("call", sorted(calls()))
@pytest.mark.parametrize("shape,error", [((1, 3), ValueError), ((3, 2), ValueError),
                                         ((1, 1, 3), ValueError), ((), TypeError)])
def test_rotation_shape_refused(call, shape, error):
    with pytest.raises(error):
        calls()[call](torch.zeros(shape))


def test_accepted_rotations_give_their_angles():
    from cantucci_gb300.autograd import angles
    for shape in ((3,), (3, 1), (3, 1, 1)):
        assert angles(torch.tensor([0.5, -1.5, 2.0], requires_grad=True).reshape(shape)) == [
            0.5, -1.5, 2.0]
