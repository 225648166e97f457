"""One and two angles (variant 9) where F, and with it every aperture, is the same over a chunk of 64
bins: the weights are then applied after the sum over the bins instead of at each one.  Constant
F, F constant in pieces that end inside chunks, bands shorter than a chunk and shapes of 16 bins
between exact phases, against the FP64 oracle within the bound of test_gpu_pw_tc.py."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH, FS = 0.3048e-3, 20e6


class _Steps(f_numbers.f_number):
    """F in pieces of `n` bins."""

    def __init__(self, n):
        self.n = n

    def compute_values(self, p):
        return (0.9 + 0.4 * ((np.arange(np.size(p)) // self.n) % 3)).reshape(np.shape(p))

    def spec(self):
        raise NotImplementedError

    def string(self):
        return "steps_%d" % self.n


@pytest.mark.parametrize("ne,na,nt,nx,nz,win,fn,compound,bins", [
    (2, 1, 96, 3, 5, windows.boxcar(), f_numbers.constant(0.7), True, 0),
    (65, 1, 700, 5, 33, windows.hann(), f_numbers.constant(1.5), True, 0),
    (131, 2, 512, 6, 33, windows.tukey(0.5), f_numbers.constant(0.8), True, 16),
    (40, 2, 384, 3, 20, windows.triangular(), f_numbers.constant(0.0), False, 0),
    (70, 1, 900, 5, 35, windows.hann(), _Steps(150), True, 0),
    (70, 2, 900, 5, 35, windows.boxcar(), _Steps(97), False, 16),
])
def test_image_matches_oracle(gpu, ne, na, nt, nx, nz, win, fn, compound, bins):
    import torch
    rng = np.random.default_rng(47)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(nx) - (nx - 1) / 2.0) * 0.913e-3
    pz = 4.013e-3 + np.arange(nz) * 0.2503e-3
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    plan = das.PWPlan(px, pz, nt, ne, FS, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win, fn,
                      compound=compound)
    plan.set_kernel_variant(9)
    plan.set_shape(0, bins)
    w = torch.empty((nx, nz), dtype=torch.float32, device=gpu)
    img = plan.execute(torch.tensor(rf, device=gpu), weights=w).cpu().numpy()
    info = plan.info()
    plan.close()
    band = O.band_mex(pz, nt, ne, FS, arr.width, arr.pitch, 1540.0, (2e6, 7e6), 0.0)
    F = fn.compute_values(O.pitch_over_lambda(band, arr.pitch, FS, 1540.0))
    o = [O.das_pw_mex(px, pz, rf[a].T.astype(np.float64), FS, angles[a], arr.width, arr.pitch, 1540.0,
                      (2e6, 7e6), 0.0, win.spec(), F, "on") for a in range(na)]
    ref = np.stack([x[0].T for x in o])
    if compound:
        ref = ref.sum(axis=0, keepdims=True)
    assert np.linalg.norm(img - ref) <= TOL * np.linalg.norm(ref)
    np.testing.assert_allclose(w.cpu().numpy(), o[0][1].T, rtol=1e-5)
    # the counted terms are the apertures' elements
    W = np.stack([O._aperture_weights(("boxcar", 0.0), px[i], pz, F, band, ne, arr.pitch) for i in range(nx)])
    assert info["active_terms"] == int((W > 0).sum()) * na
