"""Images kept apart (one per angle) share a launch of the tensor-core kernel, whose operands are fp16
pairs under a power-of-two scale.  The scale is each angle's own: an image is as accurate by itself
as alone, however loud the others are (the bound of test_gpu_pw_tc.py)."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH, FS = 0.3048e-3, 20e6


def test_images_of_angles_far_apart_in_level(gpu):
    import torch
    rng = np.random.default_rng(37)
    ne, nt, nx, nz, win, fn = 48, 384, 6, 33, windows.hann(), f_numbers.constant(1.31)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(nx) - (nx - 1) / 2.0) * 0.513e-3
    pz = 4.013e-3 + np.arange(nz) * 0.2503e-3
    angles = np.deg2rad(np.linspace(-9.0, 9.0, 5))
    rf = rng.standard_normal((5, ne, nt)) * np.array([1.0, 1e-10, 1e5, 0.0, 1e-4])[:, None, None]
    rf = rf.astype(np.float32)
    plan = das.PWPlan(px, pz, nt, ne, FS, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win, fn,
                      compound=False)
    img = plan.execute(torch.tensor(rf, device=gpu)).cpu().numpy()
    plan.close()
    for a in range(5):
        o = O.das_pw_mex(px, pz, rf[a].T.astype(np.float64), FS, angles[a], arr.width, arr.pitch, 1540.0,
                         (2e6, 7e6), 0.0, win.spec(), fn.spec(), "on")[0].T
        assert np.linalg.norm(img[a] - o) <= TOL * np.linalg.norm(o), a
