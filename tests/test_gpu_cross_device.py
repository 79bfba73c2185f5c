"""The device text of the forward's per-event screen (cross_bit, bats_gb300/csrc/common.cuh: a chain of predicates in PTX) gives the
answers of its host text, which tests/test_cross_screen.py proves conservative: on states with a root next to either end of the
window, on the edges of the ranges in which claims are made, and on operands of every class, NaN and infinities among them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300.build import ARCH_FLAGS, nvcc_path  # noqa: E402
from tests._float_model import F, expf_range, states_with_root_near  # noqa: E402
from tests.test_cross_screen import ROOT, SCREEN, _build, _claims  # noqa: E402
from tests.test_screen_source import _wild  # noqa: E402

pytestmark = pytest.mark.gpu

DEVICE = r"""
#include "common.cuh"
using namespace bats;
// The windows in memory first, as the forward kernels have them from their producers.
__global__ void windows(const float* es, const float* en, SolveConst k, int n, CrossWindow* w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) w[i] = cross_window(0.0f, 0.0f, es[i], en[i], k);
}
template <bool CONV>
__global__ void bits(const float* a, const float* b, const CrossWindow* w, SolveConst k, int n, unsigned* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = cross_bit<CONV>(a[i], b[i], w[i], k, 1u << (i & 31));
}
extern "C" int screen(int conv, const float* a, const float* b, const float* es, const float* en, float c, float e_max, int n,
                      void* w, unsigned* out) {
    SolveConst k{};
    k.c = c;
    k.tau = 1.0f;
    k.e_max = e_max;
    k.inv_c = c > 0.0f ? 1.0f / c : 0.0f;
    k.fast = c > 0.0f;
    set_screen_const(k);
    windows<<<(n + 255) / 256, 256>>>(es, en, k, n, (CrossWindow*)w);
    if (conv) bits<true><<<(n + 255) / 256, 256>>>(a, b, (CrossWindow*)w, k, n, out);
    else bits<false><<<(n + 255) / 256, 256>>>(a, b, (CrossWindow*)w, k, n, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    d = tmp_path_factory.mktemp("device_screen")
    src, so = d / "screen.cu", d / "screen.so"
    src.write_text(DEVICE)
    subprocess.run([nvcc_path(), *ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(ROOT, "bats_gb300", "csrc"), "-o", str(so), str(src)], check=True)
    fn = ctypes.CDLL(str(so)).screen
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4 + [ctypes.c_float] * 2 + [ctypes.c_int] + [ctypes.c_void_p] * 2
    return fn


@pytest.mark.parametrize("conv", [False, True], ids=["fc", "conv"])
def test_device_answers_are_the_hosts(cuda, device, tmp_path_factory, conv):
    exe = _build(tmp_path_factory.mktemp("host_screen"), "screen", SCREEN)
    rng = np.random.default_rng(31)
    n, tau = 100_000, F(0.26)
    t = (rng.uniform(0.1, 8.2, n) * np.float64(tau)).astype(F)
    e_lo, e_hi = expf_range(t, tau)
    delta = np.exp(rng.uniform(np.log(1e-9), 0.0, n))
    u = rng.uniform(-40.0, 24.0, n) * 2.0 ** -20
    cases = []
    for c in (F(0.7), F(5.0), F(2.0 ** -20), F(2.0 ** -61), F(2.0 ** 60), F(0.0)):
        a, b = states_with_root_near(e_lo.astype(np.float64), u, delta, c if c > 0 else F(1.0))
        cases += [(a, b, np.zeros(n, F), e_lo, c, np.inf), (a, b, e_hi, np.full(n, np.inf, F), c, np.inf), (a, b, e_hi, e_lo, c, 40.0)]
        a, b = _wild(rng, n), _wild(rng, n)
        cases += [(a, b, e_hi, _wild(rng, n), c, np.inf), (a, b, _wild(rng, n), e_lo, c, 7.5)]
        edge = np.asarray([2.0 ** -50, 2.0 ** 60, -2.0 ** 60, np.nextafter(F(2.0 ** 60), F(np.inf)), 0.0, -0.0, 1e-38, 1e-45], F)
        b = edge[rng.integers(0, edge.size, n)] * rng.choice(np.asarray([1, 1, 1 + 2.0 ** -23, 2.0 ** -70], F), n)
        cases.append((edge[rng.integers(0, edge.size, n)], b.astype(F), e_hi, e_lo, c, np.inf))
    claimed = 0
    for a, b, es, en, c, e_max in cases:
        host = [np.ascontiguousarray(v, F) for v in (a, b, es, en)]
        dev = [torch.as_tensor(v).cuda() for v in host]
        w, out = torch.empty((n, 8), device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        assert device(int(conv), *(v.data_ptr() for v in dev), float(c), float(e_max), n, w.data_ptr(), out.data_ptr()) == 0
        bits = out.cpu().numpy().view(np.uint32)
        claim = _claims(exe, conv, *host, c, F(e_max)).astype(bool)
        assert np.array_equal(bits, np.where(claim, 0, np.uint32(1) << (np.arange(n) & 31).astype(np.uint32)))
        claimed += int(claim.sum())
    assert claimed > 100_000
