"""Window tables of long arrays: beyond 256 elements a column holds those that its tile's apertures
reach, which for a narrow aperture is a small part of the array, and a table beyond 4 GB (synthetic
aperture: 256 MB) holds the frame's columns in turns, refilled between launches.  Bounds as in
test_gpu_pw_tc.py (images) and, between sums over the same voxels in other slices, the operand split
2^-21 and three FP32 additions a group of 8 voxels, each within 2^-23 of the partial sum."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, normalizations, synth, windows
from oracle import coracle as CO
from oracle import fnum_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH, FS, FB = 0.3048e-3, 20e6, [4e6, 4.02e6]


def _plan(ne, na, nt, px, pz, win, fn, fb, compound=True):
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    return arr, angles, das.PWPlan(px, pz, nt, ne, FS, angles, arr.width, arr.pitch, 1540.0, fb, 0.0, win, fn,
                                   compound=compound)


def _check(gpu, ne, na, nt, px, pz, win, fn, fb, compound):
    import torch
    rng = np.random.default_rng(53)
    arr, angles, plan = _plan(ne, na, nt, px, pz, win, fn, fb, compound)
    plan.set_kernel_variant(9)
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    img = plan.execute(torch.tensor(rf, device=gpu)).cpu().numpy()
    plan.close()
    ix, iz = (v.ravel().astype(np.int32) for v in np.meshgrid(np.arange(px.size), np.arange(pz.size), indexing="ij"))
    ref = [CO.pw_mex(px, pz, rf[a:a + 1], FS, angles[a:a + 1], arr.width, arr.pitch, 1540.0, tuple(fb), 0.0,
                     win.spec(), fn.spec(), "on", ix, iz)[0].reshape(px.size, pz.size) for a in range(na)]
    ref = np.stack(ref)
    if compound:
        ref = ref.sum(axis=0, keepdims=True)
    assert np.linalg.norm(img - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("ne,na,dx,win,compound", [
    (257, 1, 0.5, windows.hann(), True),
    (512, 2, 7.3, windows.tukey(0.5), False),
    (300, 3, 0.5, windows.hann(), True),
    (512, 3, 40.0, windows.boxcar(), True),           # a tile's columns see disjoint elements
    (1100, 17, 21.7, windows.triangular(), False),
    (300, 5, 111.3, windows.hann(), True),            # columns beside the array
    (4096, 1, 411.3, windows.hann(), True),           # tables nearly as wide as the array
])
def test_narrow_apertures(gpu, ne, na, dx, win, compound):
    px = 0.031e-3 + (np.arange(11) - 5) * dx * PITCH
    pz = 3.013e-3 + np.arange(37) * 0.2503e-3
    _check(gpu, ne, na, 64, px, pz, win, f_numbers.grating.angle_lb(60.0, 1.5),
           [3e6, 4e6] if ne < 1000 else FB, compound)


# all of 4096 elements in every aperture: 67 MB a column
NE, PX, PZ = 4096, 0.031e-3 + (np.arange(67) - 33) * 17.3 * PITCH, np.array([9.1e-3, 21.3e-3])


@pytest.mark.parametrize("na,compound", [(1, True), (3, True), (3, False)])
def test_table_in_turns(gpu, na, compound):
    _check(gpu, NE, na, 64, PX, PZ, windows.hann(), f_numbers.constant(0.0), FB, compound)


def test_adjoint_in_turns(gpu):
    """The gradient of a frame is the sum of those of its halves, whose tables fit."""
    import torch
    rng = np.random.default_rng(59)
    G = torch.tensor(rng.standard_normal((PX.size, PZ.size)) + 1j * rng.standard_normal((PX.size, PZ.size)),
                     dtype=torch.complex64, device=gpu)
    g = []
    for s in (slice(None), slice(0, 35), slice(35, None)):
        _, _, plan = _plan(NE, 3, 64, PX[s], PZ, windows.hann(), f_numbers.constant(0.0), FB)
        g.append(plan.adjoint(G[s].contiguous(), dc=False)[0].to(torch.complex128))
        plan.close()
    err = torch.linalg.vector_norm(g[0] - g[1] - g[2]) / torch.linalg.vector_norm(g[0])
    assert float(err) <= 2.0 ** -21 + 3 * -(-PX.size * PZ.size // 8) * 2.0 ** -23


@pytest.mark.parametrize("win", [windows.boxcar(), windows.hann()])
def test_synthetic_aperture_in_turns(gpu, win):
    import torch
    rng = np.random.default_rng(61)
    ne, nt, on, fn = 128, 64, normalizations.on(), f_numbers.constant(0.8)
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px, pz = 0.031e-3 + (np.arange(4071) - 2035) * 9.13e-6, np.array([9.1e-3])
    cols = np.array([0, 2100, 4059, 4063, 4064, 4067, 4070], dtype=np.int32)
    rf = rng.standard_normal((ne, ne, nt)).astype(np.float32)
    plan = das.SAPlan(px, pz, nt, ne, FS, arr.width, arr.pitch, 1540.0, [4e6, 4.3e6], 0.0, win, win, fn, fn, on, on)
    plan.set_kernel_variant(2)
    img = plan.execute(torch.tensor(rf, device=gpu))[0].cpu().numpy()
    plan.close()
    ref, _, _, _ = CO.sa_mex(px, pz, rf, FS, arr.width, arr.pitch, 1540.0, (4e6, 4.3e6), 0.0, win.spec(), win.spec(),
                             fn.spec(), fn.spec(), "on", "on", cols, np.zeros_like(cols))
    assert np.linalg.norm(img[cols, 0] - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("ne,na,nx,nz,dx", [(300, 3, 21, 13, 0.5), (512, 9, 9, 37, 40.0), (400, 2, 130, 70, 2.9),
                                            (1100, 20, 9, 37, 40.0)])
def test_adjoint_of_narrow_apertures(gpu, ne, na, nx, nz, dx):
    """dL/dX*_j = sum_v conj(A_vj) G_v against the images of single spectrum entries, also of elements
    that no aperture reaches (zero)."""
    import torch
    rng = np.random.default_rng(67)
    px = 0.031e-3 + (np.arange(nx) - nx // 2) * dx * PITCH
    pz = 3.013e-3 + np.arange(nz) * 0.1503e-3
    _, _, plan = _plan(ne, na, 64, px, pz, windows.hann(), f_numbers.grating.angle_lb(60.0, 1.5), FB)
    G = torch.tensor(rng.standard_normal((nx, nz)) + 1j * rng.standard_normal((nx, nz)), dtype=torch.complex64,
                     device=gpu)
    g, _ = plan.adjoint(G, dc=False)
    tol = 3 * -(-min(nx * nz, 8192) // 8) * 2.0 ** -23 + 1e-5
    img = torch.empty((1, nx, nz), dtype=torch.complex64, device=gpu)
    X = torch.zeros((ne, plan.n_bins, na), dtype=torch.complex64, device=gpu)
    K = plan.n_bins
    for e, k, a in [(ne // 2, 0, 0), (ne // 2 - 1, K - 1, na - 1), (ne // 2 + 9, K // 2, 0), (0, 0, na - 1),
                    (ne - 1, 1, 0), (127, K // 3, 0), (128, 0, na - 1)]:
        X.zero_()
        X[e, k, a] = 1.0
        plan.set_spectra(X)
        A = plan.execute_beamform(img)[0].to(torch.complex128)
        want = (torch.conj(A) * G.to(torch.complex128)).sum().item()
        scale = (A.abs() * G.abs().double()).sum().item()
        assert abs(g[e, k, a].item() - want) <= tol * scale, (e, k, a)
    plan.close()


def test_batch_with_a_table_in_turns(gpu):
    """Such a frame keeps its own launches in a batch, beside the persistent ones: the images are those
    of the plans by themselves, bit for bit."""
    import torch
    rng = np.random.default_rng(89)
    plans = [_plan(NE, 3, 64, PX, PZ, windows.hann(), f_numbers.constant(0.0), FB)[2],
             _plan(64, 5, 300, PX[:9], PZ, windows.hann(), f_numbers.constant(1.1), [3e6, 5e6])[2],
             _plan(300, 3, 200, PX[:9], PZ, windows.boxcar(), f_numbers.constant(1.5), [3e6, 5e6])[2]]
    rfs = [torch.tensor(rng.standard_normal(s), dtype=torch.float32, device=gpu)
           for s in ((3, NE, 64), (5, 64, 300), (3, 300, 200))]
    want = [p.execute(rf).clone() for p, rf in zip(plans, rfs)]
    images = [torch.full_like(w, float("nan")) for w in want]
    batch = das.Batch(plans, rfs, images, n_streams=2)
    assert batch.persistent() == (2, 1)
    for _ in range(2):
        for im in images:
            im.fill_(float("nan"))
        batch.execute()
        torch.cuda.synchronize()
        assert all(torch.equal(im, w) for im, w in zip(images, want))
    batch.close()
    for p in plans:
        p.close()
