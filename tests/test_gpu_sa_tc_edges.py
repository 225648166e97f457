"""The synthetic-aperture tensor-core kernel (variant 2) where its tiling can go wrong: elements
around its groups of 8 and around the 64 up to which it keeps two bins' phasors, bins narrower
and wider than half of the accumulator, columns beside the array whose apertures are empty,
bands of one and of several ranges, and unequal windows and F-numbers.

The error against the FP64 oracle: the phasor recurrence rounds once a bin, relative 1.5 2^-24,
over 32 bins between exact anchors (2.9e-6 at the stretch's end) and enters transmit and receive
factors; the operand split adds 2^-21 = 4.8e-7: below 1e-5 of the image."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, normalizations, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
LB, C12 = f_numbers.grating.angle_lb(60, 1.5), f_numbers.constant(1.2)


@pytest.mark.parametrize("ne,nt,nx,nz,dx,wt,wr,ft,fr", [
    (2, 200, 3, 4, 1.03e-4, windows.boxcar(), windows.boxcar(), C12, C12),
    (9, 300, 5, 33, 2.07e-4, windows.hann(), windows.hann(), LB, LB),
    (63, 400, 5, 20, 4.03e-3, windows.tukey(0.5), windows.tukey(0.5), LB, LB),        # columns beside the array
    (64, 700, 4, 40, 4.01e-4, windows.boxcar(), windows.boxcar(), C12, C12),
    (65, 700, 4, 40, 4.01e-4, windows.boxcar(), windows.boxcar(), C12, C12),
    (72, 360, 6, 35, 9.01e-4, windows.boxcar(), windows.hann(), C12, LB),
    (121, 360, 3, 12, 7.01e-4, windows.triangular(), windows.tukey(0.2), LB, C12),
    (128, 300, 5, 10, 5.07e-3, windows.hann(), windows.hann(), C12, C12),
])
def test_image_matches_oracle(gpu, ne, nt, nx, nz, dx, wt, wr, ft, fr):
    import torch
    rng = np.random.default_rng(17)
    arr = synth.LinearArray(ne, 0.3e-3, 0.918 * 0.3e-3)
    px = (np.arange(nx) - (nx - 1) / 2.0) * dx
    pz = 3e-3 + np.arange(nz) * 0.7503e-3
    rf = rng.standard_normal((ne, ne, nt)).astype(np.float32)
    on = normalizations.on()
    plan = das.SAPlan(px, pz, nt, ne, 40e6, arr.width, arr.pitch, 1540.0, [2e6, 9e6], 8.5, wt, wr, ft, fr, on, on)
    plan.set_kernel_variant(2)
    img = plan.execute(torch.tensor(rf, device=gpu))[0].cpu().numpy().T
    ref, _, _, _ = O.das_sa_mex(px, pz, np.transpose(rf, (2, 1, 0)).astype(np.float64), 40e6, arr.width, arr.pitch,
                                1540.0, (2e6, 9e6), 8.5, wt.spec(), wr.spec(), ft.spec(), fr.spec(), "on", "on")
    assert np.linalg.norm(img - ref) <= TOL * np.linalg.norm(ref)
    plan.close()
