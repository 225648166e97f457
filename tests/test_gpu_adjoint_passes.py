"""The adjoint kernel's angle passes of 24 (17 to 24, 33 to 48 angles, ...) entry by entry:
dL/dX*_j = sum_v conj(A_vj) G_v against the images A_j of single spectrum entries, at the first and
last angle of a pass, bins around the chunks of 8 and several slices.  The bound is
test_gpu_pw_adj_tc.py's."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows

pytestmark = pytest.mark.gpu

PITCH = 0.3048e-3


@pytest.mark.parametrize("ne,na,nt,nx,nz,win", [
    (20, 17, 300, 7, 3, windows.boxcar()),
    (33, 24, 256, 5, 41, windows.hann()),
    (130, 33, 128, 6, 29, windows.tukey(0.5)),
    (24, 20, 200, 91, 92, windows.hann()),
    (64, 48, 90, 4, 33, windows.triangular()),
])
def test_entries_match_images(gpu, ne, na, nt, nx, nz, win):
    import torch
    rng = np.random.default_rng(29)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px = (np.arange(nx) - (nx - 1) / 2.0) * 0.513e-3
    pz = 5e-3 + np.arange(nz) * 0.2503e-3
    angles = np.deg2rad(np.linspace(-9.0, 9.0, na))
    plan = das.PWPlan(px, pz, nt, ne, 20e6, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, win,
                      f_numbers.grating.angle_lb(60.0, 1.5))
    plan.set_kernel_variant(9)
    G = torch.tensor(rng.standard_normal((nx, nz)) + 1j * rng.standard_normal((nx, nz)), dtype=torch.complex64,
                     device=gpu)
    g, _ = plan.adjoint(G, dc=False)
    tol = 3 * -(-min(nx * nz, 8192) // 8) * 2.0 ** -23 + 1e-5
    img = torch.empty((1, nx, nz), dtype=torch.complex64, device=gpu)
    K = plan.n_bins
    X = torch.zeros((ne, K, na), dtype=torch.complex64, device=gpu)
    for e, k, a in [(ne // 2, 0, 0), (ne // 2, K - 1, na - 1), (ne // 2 - 1, 7, 15), (0, 8, 16),
                    (ne - 1, K - 8, min(23, na - 1)), (ne // 3, K - 9, min(24, na - 1))]:
        X.zero_()
        X[e, k, a] = 1.0
        plan.set_spectra(X)
        A = plan.execute_beamform(img)[0].to(torch.complex128)
        want = (torch.conj(A) * G.to(torch.complex128)).sum().item()
        scale = (A.abs() * G.abs().double()).sum().item()
        assert abs(g[e, k, a].item() - want) <= tol * scale, (e, k, a)
    plan.close()
