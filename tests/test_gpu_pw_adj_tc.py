"""The adjoint kernel entry by entry: dL/dX*_j = sum_v conj(A_vj) G_v against the images A_j of
single spectrum entries, where its tiling can go wrong: columns shorter than a group of 8 voxels,
several slices, element passes, angle passes of 8 and 16 and their remainders.

The bound is relative to sum_v |A_vj| |G_v|: the tensor cores' FP32 accumulation rounds each of
the three additions a group of 8 voxels (up to 1024 groups of a slice) by at most 2^-24 2 of the
partial sum, the images carry 1e-5 (see test_gpu_pw_tc.py)."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, synth, windows

pytestmark = pytest.mark.gpu

PITCH = 0.3048e-3


@pytest.mark.parametrize("ne,na,nt,nx,nz,win", [
    (20, 3, 300, 7, 3, windows.boxcar()),
    (33, 8, 256, 5, 41, windows.hann()),
    (130, 9, 300, 6, 29, windows.tukey(0.5)),
    (64, 17, 256, 4, 33, windows.triangular()),
    (24, 5, 200, 91, 92, windows.hann()),
    (257, 2, 256, 3, 17, windows.hann()),
])
def test_entries_match_images(gpu, ne, na, nt, nx, nz, win):
    import torch
    rng = np.random.default_rng(23)
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
    X = torch.zeros((ne, plan.n_bins, na), dtype=torch.complex64, device=gpu)
    K = plan.n_bins
    for e, k, a in [(ne // 2, 0, 0), (ne // 2, K - 1, na - 1), (ne // 2 - 1, K // 2, na // 2), (0, 0, na - 1),
                    (ne - 1, 1, 0), (ne // 3, K // 3, na - 1)]:
        X.zero_()
        X[e, k, a] = 1.0
        plan.set_spectra(X)
        A = plan.execute_beamform(img)[0].to(torch.complex128)
        want = (torch.conj(A) * G.to(torch.complex128)).sum().item()
        scale = (A.abs() * G.abs().double()).sum().item()
        assert abs(g[e, k, a].item() - want) <= tol * scale, (e, k, a)
    plan.close()
