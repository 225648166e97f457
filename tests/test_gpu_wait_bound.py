"""The device waits of the tensor-core beamformers end: a wait for an arrival that never comes gives
up after WAIT_NS of the global timer, records the timeout and raises the abort flag, later waits
then end at once, and the context stays usable.  The probe is one warp; its first wait has an
arrival, its second has none."""
import ctypes as C
import os
import subprocess

import pytest

from f_number_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fnum_tc_beam.cuh"
using namespace fnum;
using namespace fnum::tcx;
// out: answer and nanoseconds of three waits, the abort flag, the error word
__global__ void probe(unsigned long long* out, unsigned long long* err) {
  __shared__ uint64_t bars[2];
  __shared__ int flag;
  volatile int* abort_flag = &flag;
  const uint32_t b = smem_u32(bars);
  if (threadIdx.x == 0) {
    flag = 0;
    mbar_init(b, 1);
    mbar_init(b + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arrive(b);
    for (int i = 0; i < 3; ++i) {
      const unsigned long long t0 = global_ns();
      out[2 * i] = p5_wait(i ? b + 8 : b, 0u, 0u, abort_flag, err) ? 1 : 0;
      out[2 * i + 1] = global_ns() - t0;
    }
    out[6] = (unsigned long long)flag;
  }
}
extern "C" unsigned long long wait_ns() { return WAIT_NS; }
extern "C" unsigned long long timeout_bit() { return ERR_TC_TIMEOUT; }
extern "C" int run(unsigned long long* host) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 8 * sizeof(*d));
  if (e == cudaSuccess) e = cudaMemset(d, 0, 8 * sizeof(*d));
  if (e == cudaSuccess) {
    probe<<<1, 32>>>(d, d + 7);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(host, d, 8 * sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


def test_wait_without_an_arrival_ends(gpu, tmp_path):
    src, lib = tmp_path / "wait_probe.cu", tmp_path / "wait_probe.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-cudart",
                                                  "static", "-I", build.CSRC, "-I",
                                                  os.path.join(build.ROOT, "include"), "-o", str(lib), str(src)],
                   check=True)
    L = C.CDLL(str(lib))
    L.wait_ns.restype = L.timeout_bit.restype = C.c_ulonglong
    out = (C.c_ulonglong * 8)()
    assert L.run(out) == 0
    ok = [out[0], out[2], out[4]]
    ns = [out[1], out[3], out[5]]
    limit = L.wait_ns()
    assert ok == [1, 0, 0]
    assert ns[0] < limit // 4
    # the timer is read every 64 tests of a fraction of a millisecond each
    assert limit <= ns[1] <= limit + 500_000_000
    assert ns[2] < limit // 4
    assert out[6] == 1 and out[7] == L.timeout_bit()
    import torch
    assert float(torch.ones(8, device=gpu).sum()) == 8.0
