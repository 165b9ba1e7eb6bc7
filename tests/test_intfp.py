"""The integer forms of FP64 sums, differences and products (csrc/sbfs_intfp.cuh) give the hardware's values bit for
bit wherever they do not give up: on the host's build of the file, and on the GPU's."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "simplebubblyflowsolver_gb300", "csrc")
FORMS = """
#include "sbfs_intfp.cuh"
using namespace sbfs::intfp;
SBFS_IF void form(int op, double a, double b, double &s, double &t, u32 &bad) {
  t = 0.;
  switch (op) {
    case 0: s = add<true>(a, b, bad); break;
    case 1: s = add<false>(a, b, bad); break;
    case 2: s = sub<true>(a, b, bad); break;
    case 3: addsub<true>(a, b, s, t, bad); break;
    case 4: addsub<false>(a, b, s, t, bad); break;
    case 5: s = addp(a, b, bad); break;
    case 6: s = mul<true>(a, b, bad); break;
    case 8: addsub<false, true>(a, b, s, t, bad); break;
    default: s = mul<false>(a, b, bad);
  }
}
"""
HOST = FORMS + """
extern "C" void run(int op, int n, const double *a, const double *b, double *s, double *t, unsigned *bad) {
  for (int i = 0; i < n; ++i) { bad[i] = 0; form(op, a[i], b[i], s[i], t[i], bad[i]); }
}
"""
DEVICE = FORMS + """
#include <cuda_runtime.h>
__global__ void k(int op, int n, const double *a, const double *b, double *s, double *t, unsigned *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned g = 0;
  double x, y;
  form(op, a[i], b[i], x, y, g);
  s[i] = x, t[i] = y, bad[i] = g;
}
extern "C" int run(int op, int n, const double *a, const double *b, double *s, double *t, unsigned *bad) {
  double *d;
  unsigned *g;
  if (cudaMalloc(&d, 32ull * n) || cudaMalloc(&g, 4ull * n)) return 1;
  cudaMemcpy(d, a, 8ull * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, 8ull * n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(op, n, d, d + n, d + 2 * n, d + 3 * n, g);
  cudaMemcpy(s, d + 2 * n, 8ull * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(t, d + 3 * n, 8ull * n, cudaMemcpyDeviceToHost);
  const int e = cudaMemcpy(bad, g, 4ull * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(g);
  return e;
}
"""
OPS = ["add_zero", "add", "sub_zero", "addsub_zero", "addsub", "addp", "mul_zero", "mul", "addsub_sticky"]


def _build(tmp, device):
    src, lib = os.path.join(tmp, "forms.cu" if device else "forms.cpp"), os.path.join(tmp, "forms.so")
    with open(src, "w") as f:
        f.write(DEVICE if device else HOST)
    if device:
        from simplebubblyflowsolver_gb300.build import ARCH, nvcc
        cmd = [nvcc(), *ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I" + CSRC, src, "-o", lib, "-lcudart"]
    else:
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + CSRC, src, "-o", lib]
    subprocess.run(cmd, check=True, capture_output=True)
    return ctypes.CDLL(lib)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("intfp")), False)


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("intfp_gpu")), True)


def _operands(n=400000):
    """pairs at every exponent difference, with trailing zeros and runs of ones (ties, carries), near-equal pairs
    (cancellation), zeros of either sign, and the whole range of patterns (denormals, infinities, NaN)"""
    rng = np.random.default_rng(11)
    frac = rng.integers(0, 1 << 52, (2, n), dtype=np.uint64)
    kind = rng.integers(0, 8, (2, n))
    frac = np.where(kind == 0, frac & np.uint64(0xfffff00000000), frac)
    frac = np.where(kind == 1, 0, frac)
    frac = np.where(kind == 2, frac | np.uint64(0xfffffffffff00), frac)
    frac = np.where(kind == 3, frac & np.uint64(0xfffffffffff80), frac)
    ea = rng.integers(1003, 1043, n)
    eb = np.where(np.arange(n) % 2 == 0, ea + rng.integers(-2, 3, n), ea + rng.integers(-65, 66, n))
    wild = np.arange(n) % 16 == 0
    ea, eb = np.where(wild, rng.integers(0, 2048, n), ea), np.where(wild, rng.integers(0, 2048, n), eb)
    sign = rng.integers(0, 2, (2, n)).astype(np.uint64) << np.uint64(63)
    u = sign | (np.stack((ea, eb)).astype(np.uint64) << np.uint64(52)) | frac
    near = rng.integers(0, 16, n) == 0
    u[1] = np.where(near, (u[0] + rng.integers(0, 5, n).astype(np.uint64)) ^ sign[1], u[1])
    for row in (0, 1):
        u[row] = np.where(rng.integers(0, 64, n) == 0, sign[row], u[row])
    return u[0].view(np.float64), u[1].view(np.float64)


def _check(lib, op):
    a, b = _operands()
    if op == "addp":
        a, b = np.abs(a), np.abs(b)
    n = a.size
    s, t, bad = np.empty(n), np.empty(n), np.empty(n, dtype=np.uint32)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, s, t, bad)]
    assert not lib.run(OPS.index(op), n, *p)
    with np.errstate(all="ignore"):
        want = {"a": a + b, "s": a - b, "m": a * b}["s" if op.startswith("sub_") else op[0]]
        diff = a - b
    ok = bad == 0
    assert np.array_equal(s[ok].view(np.uint64), want[ok].view(np.uint64))
    if op.startswith("addsub"):
        assert np.array_equal(t[ok].view(np.uint64), diff[ok].view(np.uint64))
    # what it must leave to the FP64 unit, and what it must not
    assert not ok[~np.isfinite(a) | ~np.isfinite(b)].any()
    plain = (np.abs(np.log2(np.abs(a / np.where(b == 0, 1, b)))) < 10) & (np.abs(want) > 1e-6 * np.abs(a)) & \
        (np.abs(diff) > 1e-6 * np.abs(a)) & (np.abs(a) > 1e-30) & (np.abs(a) < 1e30)
    assert plain.sum() > n / 4 and ok[plain].all()
    if op.endswith("_sticky"):  # never given up for lost bits
        plain = (np.abs(a) > 1e-30) & (np.abs(a) < 1e30) & (np.abs(b) > 0) & (np.abs(b) < 1e-4 * np.abs(a))
        assert plain.sum() > n / 16 and ok[plain].all()
    if op.endswith("_zero"):
        assert ok[(a == 0) & (b == 0) & ~np.signbit(a) & ~np.signbit(b)].all()


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("op", OPS)
def test_host_build_gives_the_hosts_bits(host, op):
    host.run.restype = None
    _check(host, op)


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("op", OPS)
def test_device_build_gives_the_hosts_bits(device, op):
    device.run.restype = ctypes.c_int
    _check(device, op)
