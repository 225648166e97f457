"""Frames of more columns than a launch has blocks in y and z (65535): the window tables have a block
per (column, row)."""
import numpy as np
import pytest

from f_number_gb300 import das, f_numbers, normalizations, synth, windows
from oracle import coracle as CO

pytestmark = pytest.mark.gpu

TOL = 1e-5
PITCH, FS, NX = 0.3048e-3, 20e6, 65543
PX = (np.arange(NX) - (NX - 1) / 2.0) * 2.03e-8
PZ = np.array([2.013e-3])
COLS = np.array([0, 5, 32771, 65534, 65535, 65536, 65542], dtype=np.int32)
WIN, FN = windows.hann(), f_numbers.constant(0.831)


@pytest.mark.parametrize("na", [1, 3])
def test_plane_wave(gpu, na):
    import torch
    rng = np.random.default_rng(41)
    ne, nt = 6, 96
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    angles = np.zeros(1) if na == 1 else np.deg2rad(np.linspace(-9.0, 9.0, na))
    rf = rng.standard_normal((na, ne, nt)).astype(np.float32)
    plan = das.PWPlan(PX, PZ, nt, ne, FS, angles, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, WIN, FN)
    plan.set_kernel_variant(9)
    img = plan.execute(torch.tensor(rf, device=gpu))[0].cpu().numpy()
    ref, _, _ = CO.pw_mex(PX, PZ, rf, FS, angles, arr.width, arr.pitch, 1540.0, (2e6, 7e6), 0.0, WIN.spec(),
                          FN.spec(), "on", COLS, np.zeros_like(COLS))
    assert np.linalg.norm(img[COLS, 0] - ref) <= TOL * np.linalg.norm(ref)
    plan.close()


def test_synthetic_aperture(gpu):
    import torch
    rng = np.random.default_rng(43)
    ne, nt, on = 6, 96, normalizations.on()
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    rf = rng.standard_normal((ne, ne, nt)).astype(np.float32)
    plan = das.SAPlan(PX, PZ, nt, ne, FS, arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0, WIN, WIN, FN, FN, on, on)
    plan.set_kernel_variant(2)
    img = plan.execute(torch.tensor(rf, device=gpu))[0].cpu().numpy()
    ref, _, _, _ = CO.sa_mex(PX, PZ, rf, FS, arr.width, arr.pitch, 1540.0, (2e6, 7e6), 0.0, WIN.spec(), WIN.spec(),
                             FN.spec(), FN.spec(), "on", "on", COLS, np.zeros_like(COLS))
    assert np.linalg.norm(img[COLS, 0] - ref) <= TOL * np.linalg.norm(ref)
    plan.close()
