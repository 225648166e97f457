"""Device memory of plane-wave plans: one of the per-voxel kernel holds no window table until a gradient
needs it, and where the device has no room for a whole table the plan makes do with a part of it."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows

pytestmark = pytest.mark.gpu

PITCH, FB = 0.3048e-3, [4e6, 4.02e6]


def _plan(ne, px, kernel="fused"):
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    return das.PWPlan(px, np.array([9.1e-3, 21.3e-3]), 64, ne, 20e6, np.deg2rad([-5.0, 0.0, 5.0]), arr.width, arr.pitch,
                      1540.0, FB, 0.0, windows.hann(), f_numbers.constant(0.0), kernel=kernel)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _grid(n):
    return 0.031e-3 + (np.arange(n) - n // 2) * 3.3 * PITCH


def test_plain_kernel_plan_has_no_table(gpu):
    import torch
    rng = np.random.default_rng(79)
    px = _grid(200)                         # 1024 elements: a table of 840 MB
    G = torch.tensor(rng.standard_normal((200, 2)) + 1j * rng.standard_normal((200, 2)), dtype=torch.complex64,
                     device=gpu)
    rf = torch.tensor(rng.standard_normal((3, 1024, 64)), dtype=torch.float32, device=gpu)
    fused = _plan(1024, px)
    fused.execute(rf)
    want, _ = fused.adjoint(G, dc=False)
    fused.close()
    before = _free()
    plan = _plan(1024, px, "plain")
    assert before - _free() < 400 << 20
    plan.execute(rf)
    got, _ = plan.adjoint(G, dc=False)      # takes the table
    assert before - _free() > 800 << 20
    assert torch.equal(got, want)
    plan.close()


def test_plan_where_the_table_does_not_fit(gpu):
    import torch
    rng = np.random.default_rng(83)
    px = _grid(60)                          # 4096 elements: a table of 4 GB
    rf = torch.tensor(rng.standard_normal((3, 4096, 64)), dtype=torch.float32, device=gpu)
    plan = _plan(4096, px)
    want = plan.execute(rf).clone()
    plan.close()
    hold = torch.empty(_free() - (2 << 30), dtype=torch.uint8, device=gpu)
    try:
        plan = _plan(4096, px)
        img = plan.execute(rf).clone()
        plan.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    # the bins may be split into other ranges: two images within 1e-5 of the exact one each
    assert float(torch.linalg.vector_norm(img - want)) <= 2e-5 * float(torch.linalg.vector_norm(want))
