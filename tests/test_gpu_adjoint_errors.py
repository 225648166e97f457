"""The error word of a plan and the gradients: fnum_pw_adjoint reports what its own kernels recorded, a
bit that an earlier call left does not fail it, and an overflow of the segment scratch in its
derivative pass does.  A probe built against the plan's definition sets the word, and makes the
scratch look too short (the kernel then keeps within it and records the overflow)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from f_number_gb300 import _lib, build, das, f_numbers, synth, windows

pytestmark = pytest.mark.gpu

PITCH = 0.3048e-3
SOURCE = r"""
#include "fnum_host.cpp"
extern "C" __attribute__((visibility("default"))) int probe_set_bits(fnum_plan* p, unsigned long long bits) {
  return (int)cudaMemcpy(p->counters + 2, &bits, sizeof(bits), cudaMemcpyHostToDevice);
}
extern "C" __attribute__((visibility("default"))) int probe_set_cap(fnum_plan* p, int cap) {
  const int old = p->pw.seg_cap;
  if (cap >= 2 && cap <= old) p->pw.seg_cap = cap;
  return old;
}
extern "C" __attribute__((visibility("default"))) unsigned long long probe_timeout_bit() { return fnum::ERR_TC_TIMEOUT; }
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("probe")
    src, lib = d / "plan_probe.cpp", d / "plan_probe.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O1", "-std=c++17", "-Xcompiler", "-fPIC,-fvisibility=hidden",
                                                  "-shared", "-cudart", "static", "-I", build.CSRC, "-I",
                                                  os.path.join(build.ROOT, "include"), "-o", str(lib), str(src),
                                                  build.LIB], check=True)
    L = C.CDLL(str(lib))
    L.probe_set_bits.argtypes = [C.c_void_p, C.c_ulonglong]
    L.probe_set_cap.argtypes = [C.c_void_p, C.c_int]
    L.probe_timeout_bit.restype = C.c_ulonglong
    return L


def _plan(gpu):
    import torch
    rng = np.random.default_rng(73)
    ne, na, nt, nx, nz = 40, 3, 300, 7, 20
    arr = synth.LinearArray(ne, PITCH, 0.918 * PITCH)
    px, pz = (np.arange(nx) - (nx - 1) / 2.0) * 0.513e-3, 5e-3 + np.arange(nz) * 0.2503e-3
    plan = das.PWPlan(px, pz, nt, ne, 20e6, np.deg2rad([-5.0, 0.0, 5.0]), arr.width, arr.pitch, 1540.0, [2e6, 7e6], 0.0,
                      windows.hann(), f_numbers.grating.angle_lb(60.0, 1.5))
    plan.execute(torch.tensor(rng.standard_normal((na, ne, nt)), dtype=torch.float32, device=gpu))
    G = torch.tensor(rng.standard_normal((nx, nz)) + 1j * rng.standard_normal((nx, nz)), dtype=torch.complex64,
                     device=gpu)
    return plan, G


def test_earlier_bits_do_not_fail_the_adjoint(gpu, probe):
    import torch
    plan, G = _plan(gpu)
    want, _ = plan.adjoint(G, dc=False)
    for dc in (False, True):
        assert probe.probe_set_bits(plan._ptr, probe.probe_timeout_bit()) == 0
        with pytest.raises(_lib.FNumError):
            plan.info()
        got, _ = plan.adjoint(G, dc=dc)
        assert torch.linalg.vector_norm(got - want) <= 1e-6 * torch.linalg.vector_norm(want)
        plan.info()
    plan.close()


def test_overflow_fails_the_derivative_pass(gpu, probe):
    plan, G = _plan(gpu)
    cap = probe.probe_set_cap(plan._ptr, 2)
    with pytest.raises(_lib.FNumError):
        plan.adjoint(G, dc=True)
    assert cap > 2
    plan.close()
