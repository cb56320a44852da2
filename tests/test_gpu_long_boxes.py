"""The 3D filter on boxes with more planes than a grid's z dimension has blocks."""
import pytest
import torch

from entity_gb300.inputs import GridSpec, empty_field
from entity_gb300.sim import Context
from oracle.oracle import Oracle
from tests.helpers import random_currents

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [(4, 9, 65535), (5, 4, 65537), (40, 4, 66001)])
def test_filter_of_long_boxes(n, real):
    g = GridSpec(dim=3, n=n, order=2, real=real)
    o, ctx = Oracle(g), Context(g)
    Jo, buff = random_currents(g, 7), empty_field(g, 3)
    o.fill_ghosts(Jo, False, 0, 3)
    Jg = Jo.cuda()
    for _ in range(2):
        o.filter_pass(Jo, buff)
        o.fill_ghosts(Jo, False, 0, 3)
    ctx.filter_currents(Jg, empty_field(g, 3, "cuda"), 2)
    torch.cuda.synchronize()
    assert torch.equal(Jo, Jg.cpu())
    ctx.close()
