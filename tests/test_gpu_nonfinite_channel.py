"""A channel that delivers NaN or Inf.  An element outside a voxel's aperture has no part in its
value, so such a channel spoils the voxels whose aperture holds it (at some bin with a weight) and
no others: those equal the image without the channel, within the bounds of test_gpu_pw_tc.py.
The kernels form sums over groups of 8 elements with zero weights at the apertures' edges, where
0 times NaN must not get in."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH, FS = 0.3048e-3, 20e6


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("ne,na,nx,nz,win,compound", [
    (40, 1, 7, 35, windows.boxcar(), True),
    (70, 1, 6, 20, windows.hann(), True),
    (40, 2, 5, 33, windows.hann(), False),
    (70, 2, 6, 20, windows.tukey(0.5), True),
    (40, 3, 6, 33, windows.boxcar(), False),
    (70, 17, 5, 20, windows.hann(), False),
    (70, 5, 6, 33, windows.hann(), True),
])
def test_other_voxels_keep_their_values(gpu, ne, na, nx, nz, win, compound, bad):
    import torch
    rng = np.random.default_rng(31)
    nt, fn = 384, f_numbers.constant(1.31)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(nx) - (nx - 1) / 2.0) * 0.913e-3
    pz = 4.013e-3 + np.arange(nz) * 0.2503e-3
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    e0 = ne // 2 + 3
    clean = rf.copy()
    rf[0, e0, 100] = bad
    clean[0, e0] = 0.0
    plan = das.PWPlan(px, pz, nt, ne, FS, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win, fn,
                      compound=compound)
    img = plan.execute(torch.tensor(rf, device=gpu)).cpu().numpy()
    plan.close()
    band = O.band_mex(pz, nt, ne, FS, arr.width, arr.pitch, 1540.0, (2e6, 7e6), 0.0)
    F = np.full(band.K, 1.31)
    held = np.zeros((nx, nz), dtype=bool)
    for i in range(nx):
        w = O._aperture_weights(win.spec(), px[i], pz, F, band, ne, arr.pitch)       # [K, z, E]
        held[i] = (w[:, :, e0] > 0).any(axis=0)
    assert held.any() and not held.all()
    o = np.stack([O.das_pw_mex(px, pz, clean[a].T.astype(np.float64), FS, angles[a], arr.width, arr.pitch, 1540.0,
                               (2e6, 7e6), 0.0, win.spec(), fn.spec(), "on")[0].T for a in range(na)])
    if compound:
        o = o.sum(axis=0, keepdims=True)
    assert not np.isfinite(img[0][held]).any()
    spoiled = np.zeros(img.shape, dtype=bool)
    spoiled[0] = held                               # the other angles' images do not see the channel
    got, want = img[~spoiled], o[~spoiled]
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)
