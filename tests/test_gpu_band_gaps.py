"""F-numbers that empty a tile's apertures at some bins and not at others: the tensor-core kernels
keep phasors and products of a bin while the next one is formed, and the next one need not be its
neighbour.  A user's f_number class may return any values, and distance.constant with a small
upper bound is not monotone either.

F = 1e6 opens an aperture only within micrometres of an element's centre, and no column lies that
near to one.  A bin after a gap starts from exact phasors, so the bound of bands without gaps
holds: the recurrences round once a bin, 1.5 2^-24 relative over at most 32 bins (2.9e-6) and enter
two factors, and the operand split adds 4.8e-7: below 1e-5 of the image."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, normalizations, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH = 0.3e-3


class _Gaps(f_numbers.f_number):
    """F = `value`, and 1e6 at the bins of a gap."""

    def __init__(self, gap, value=1.0):
        self.gap, self.value = gap, value

    def compute_values(self, p):
        k = np.arange(np.size(p))
        if self.gap == "alternating":
            closed = k % 2 == 1
        elif self.gap == "one":
            closed = (k >= k.size // 2) & (k < k.size // 2 + 5)
        else:                                   # every third bin open, and neither end of the band
            closed = k % 3 != 1
        return np.where(closed, 1e6, self.value).reshape(np.shape(p))

    def spec(self):
        raise NotImplementedError

    def string(self):
        return "gaps_%s" % self.gap


def _grid(nx, nz):
    return 0.071e-3 + (np.arange(nx) - nx // 2) * 0.401e-3, 4e-3 + np.arange(nz) * 0.7503e-3


@pytest.mark.parametrize("ne,wt,wr,ft,fr", [
    (64, windows.boxcar(), windows.boxcar(), "alternating", "alternating"),
    (65, windows.boxcar(), windows.boxcar(), "alternating", "alternating"),
    (96, windows.hann(), windows.hann(), "one", "one"),
    (96, windows.boxcar(), windows.hann(), "one", "third"),
    (128, windows.hann(), windows.hann(), "third", "third"),
    (128, windows.boxcar(), windows.boxcar(), "alternating", "open"),
])
def test_synthetic_aperture(gpu, ne, wt, wr, ft, fr):
    rng = np.random.default_rng(23)
    nx, nz, nt, fs = 5, 9, 220, 40e6
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px, pz = _grid(nx, nz)
    fn = [f_numbers.constant(1.2) if f == "open" else _Gaps(f) for f in (ft, fr)]
    rf = np.transpose(rng.standard_normal((ne, ne, nt)).astype(np.float32), (2, 1, 0)).astype(np.float64)
    on = normalizations.on()
    img, _, _ = das.gpu_bf_saft_rf(px, pz, rf, fs, arr.width, arr.pitch, 1540.0, [2e6, 9e6], 8.5, wt, wr, fn[0],
                                   fn[1], on, on)
    band = O.band_mex(pz, nt, ne, fs, arr.width, arr.pitch, 1540.0, (2e6, 9e6), 8.5)
    F = [f.compute_values(O.pitch_over_lambda(band, arr.pitch, fs, 1540.0)) for f in fn]
    ref, _, _, info = O.das_sa_mex(px, pz, rf, fs, arr.width, arr.pitch, 1540.0, (2e6, 9e6), 8.5, wt.spec(),
                                   wr.spec(), F[0], F[1], "on", "on")
    assert info["zero_weight_bins"] > 0
    assert np.linalg.norm(img - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("na,gap", [(1, "third"), (2, "alternating"), (3, "alternating"), (5, "one"), (17, "third")])
def test_plane_wave(gpu, na, gap):
    import torch
    rng = np.random.default_rng(29)
    ne, nx, nz, nt, fs = 70, 5, 35, 300, 20e6
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px, pz = _grid(nx, nz)
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    fn, win = _Gaps(gap), windows.hann()
    plan = das.PWPlan(px, pz, nt, ne, fs, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win, fn)
    plan.set_kernel_variant(9)
    img = plan.execute(torch.tensor(rf, device=gpu))[0].cpu().numpy().T
    band = O.band_mex(pz, nt, ne, fs, arr.width, arr.pitch, 1540.0, (2e6, 7e6), 0.0)
    F = fn.compute_values(O.pitch_over_lambda(band, arr.pitch, fs, 1540.0))
    ref = sum(O.das_pw_mex(px, pz, rf[a].T.astype(np.float64), fs, angles[a], arr.width, arr.pitch, 1540.0,
                           (2e6, 7e6), 0.0, win.spec(), F, "on")[0] for a in range(na))
    assert np.linalg.norm(img - ref) <= TOL * np.linalg.norm(ref)
    plan.close()
