"""The tensor-core plane-wave kernel (variant 9) where its tiling can go wrong: element counts
around its groups of 8 and its element passes, angles around its passes, ragged grids, columns
beside the array whose apertures are empty, and images per angle.

The error against the FP64 oracle: the receive and the transmit recurrence round once a bin,
relative 1.5 2^-24 each, over 32 bins between exact anchors (2 x 2.9e-6 at the stretch's end),
the phasor polynomials 1e-7 and the operand split 2^-21 = 4.8e-7: below 1e-5 of the image."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

PITCH = 0.3048e-3
FN = f_numbers.grating.angle_lb(60.0, 1.5)
TOL = 1e-5


def _setup(gpu, ne, na, nt, nx, nz, dx, win, compound, seed=41):
    import torch
    rng = np.random.default_rng(seed)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(nx) - (nx - 1) / 2.0) * dx
    pz = 4e-3 + np.arange(nz) * 0.2503e-3
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    plan = das.PWPlan(px, pz, nt, ne, 20e6, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win, FN,
                      compound=compound)
    return plan, arr, px, pz, angles, rf, torch.tensor(rf, device=gpu)


@pytest.mark.parametrize("ne,na,nt,nx,nz,dx,win,compound", [
    (2, 1, 256, 1, 2, 1.03e-4, windows.boxcar(), True),
    (7, 3, 300, 5, 33, 2.07e-4, windows.hann(), True),
    (33, 2, 512, 9, 31, 1.313e-3, windows.tukey(0.5), True),         # columns beside the array
    (64, 9, 384, 3, 64, 4.01e-4, windows.triangular(), True),
    (97, 16, 640, 7, 36, 4.013e-3, windows.hann(), True),            # two element passes
    (130, 17, 256, 6, 20, 5.01e-3, windows.boxcar(), True),
    (200, 25, 512, 5, 40, 9.07e-3, windows.tukey(0.2), True),        # four element passes, 32 angles a pass
    (48, 33, 256, 4, 16, 1.07e-3, windows.hann(), True),             # two angle passes
    (41, 10, 384, 6, 35, 1.07e-3, windows.hann(), False),
    (100, 35, 256, 4, 18, 3.07e-3, windows.triangular(), False),
])
def test_image_matches_oracle(gpu, ne, na, nt, nx, nz, dx, win, compound):
    plan, arr, px, pz, angles, rf, rf_d = _setup(gpu, ne, na, nt, nx, nz, dx, win, compound)
    plan.set_kernel_variant(9)
    img = plan.execute(rf_d).cpu().numpy()
    o = np.stack([O.das_pw_mex(px, pz, rf[a].T.astype(np.float64), 20e6, angles[a], arr.width, arr.pitch, 1540.0,
                               (2e6, 7e6), 0.0, win.spec(), FN.spec(), "on")[0].T for a in range(na)])
    if compound:
        o = o.sum(axis=0, keepdims=True)
    assert np.linalg.norm(img - o) <= TOL * np.linalg.norm(o)
    plan.close()



@pytest.mark.parametrize("ne,na,nt,nx,nz,dx,win,compound", [
    (2, 1, 300, 5, 33, 2.07e-4, windows.boxcar(), True),
    (65, 1, 700, 4, 31, 1.513e-3, windows.hann(), True),             # two passes of 64 elements
    (131, 2, 512, 6, 33, 4.03e-3, windows.tukey(0.5), True),
    (40, 2, 384, 3, 20, 1.07e-3, windows.triangular(), False),
])
def test_few_angles_match_oracle(gpu, ne, na, nt, nx, nz, dx, win, compound):
    """One and two angles (FP32 recurrences); the same bound, without the operand split."""
    test_image_matches_oracle(gpu, ne, na, nt, nx, nz, dx, win, compound)
