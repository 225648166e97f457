"""fnum_plan_set_shape's resident blocks on variant 9: the one- and two-angle kernel runs with one block
per SM where that is asked for, the tensor-core kernel has one anyway.  Where a block runs does not
change its arithmetic: equal images."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows

pytestmark = pytest.mark.gpu

PITCH = 0.3048e-3


@pytest.mark.parametrize("na,most", [(1, 2), (2, 2), (3, 1)])
def test_resident_blocks(gpu, na, most):
    import torch
    rng = np.random.default_rng(71)
    ne, nt, side = 64, 512, 90
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(side) - (side - 1) / 2.0) * PITCH / 2
    pz = 5e-3 + np.arange(side) * PITCH / 2
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    plan = das.PWPlan(px, pz, nt, ne, 20e6, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, windows.hann(),
                      f_numbers.grating.angle_lb(60.0, 1.5))
    plan.set_kernel_variant(9)
    rf = torch.tensor(rng.standard_normal((na, ne, nt)), dtype=torch.float32, device=gpu)
    assert plan.info()["blocks_per_sm"] == most
    ref = plan.execute(rf).clone()
    for ask in (1, 2, 7, 0):
        plan.set_shape(ask, 0)
        assert plan.info()["blocks_per_sm"] == (min(ask, most) if ask else most)
        assert torch.equal(plan.execute(rf), ref)
    plan.close()
