"""The exact tracers' and the polylines' quotients and roots against the IEEE
operations, bit pattern against bit pattern: zeros keep their sign, and a NaN
comes out only where the operations give one.  A line in a field whose zero
component is -0 stays at the coordinate -0 it starts from, as in the
restatement of the reference."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

from fastqsl_gb300 import _build
from fastqsl_gb300 import params as P
from test_gpu_trace import run_dropin

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "qsl_scott.cuh"
#include "path.cu"
using namespace qsl;
__device__ bool same(float a, float b) { return isnan(a) ? isnan(b) : __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(double a, double b) {
    return isnan(a) ? isnan(b) : __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ bool unit_ok(const float* r) {
    const float nb = sqrtf(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const float3 u = unit_exact(v3(r[0], r[1], r[2]));
    return same(u.x, r[0] / nb) && same(u.y, r[1] / nb) && same(u.z, r[2] / nb);
}
__device__ bool quotient_ok(const float* r) { return same(div_const_exact(r[0], 0.002f, 1.f / 0.002f), r[0] / 0.002f); }
// the twist sum of one step of length 1, from -0 (which keeps the sign of a zero term)
__device__ bool twist_ok(const float* r) {
    TraceJob<FieldSoA> J;
    Lane<true> L;
    L.len = 0.0;
    L.tw = -0.0;
    L.pend_dl = 1.f;
    L.pend_td = r[0];
    Pending<FieldSoA> pending{J, L, true, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.f};
    for (int st = 0; st < 4; ++st) pending(st);
    pending.done();
    return same(L.tw, -0.0 + (double)r[0] / 4.0 / kRefPi * 1.0);
}
__device__ bool path_ok(const float* r) {
    const double a = (double)r[0] * 1.1, s = (double)r[1] * r[1] + (double)r[2] * r[2];
    return same(over_sqrt(a, s), __ddiv_rn(a, __dsqrt_rn(s))) && same(sixth(a), __ddiv_rn(a, 6.0));
}
__global__ void k_probe(int kind, const float* r, long long n, unsigned long long* bad) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < n; i += step) {
        const float* v = r + 3 * i;
        const bool ok = kind == 0 ? unit_ok(v) : kind == 1 ? quotient_ok(v) : kind == 2 ? twist_ok(v) : path_ok(v);
        if (!ok) atomicAdd(bad, 1ull);
    }
}
extern "C" int probe(int kind, const float* r, long long n, unsigned long long* bad) {
    k_probe<<<1216, 128>>>(kind, r, n, bad);
    return cudaDeviceSynchronize();
}
"""
KINDS = ["unit", "quotient", "twist", "path"]


@pytest.fixture(scope="module")
def probe(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("sign_probe")
    src, lib = d / "probe.cu", d / "probe.so"
    src.write_text(SOURCE)
    subprocess.run([_build.NVCC, *_build.COMMON, *_build.ARCH, "-fmad=false", "-shared", "-cudart", "static", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    return ctypes.CDLL(str(lib)).probe


@pytest.mark.parametrize("values", ["zeros", "plain", "short", "every"])
@pytest.mark.parametrize("kind", KINDS)
def test_bits_equal_the_ieee_operations(probe, kind, values):
    n = 1 << 21
    g = torch.Generator(device="cuda").manual_seed(23)
    r = torch.randn(n, 3, generator=g, device="cuda")
    e = torch.rand(n, 3, generator=g, device="cuda")
    if values == "zeros":    # of either sign, on one, two or all components
        r = torch.where(e < 0.3, torch.zeros_like(r), torch.where(e < 0.6, torch.full_like(r, -0.0), r))
    elif values == "short":  # few significant bits
        r = torch.round(r * 8.0)
    elif values == "every":  # every kind of float
        r = torch.randint(-(1 << 31), (1 << 31) - 1, (n, 3), generator=g, device="cuda", dtype=torch.int64)
        r = r.to(torch.int32).view(torch.float32)
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert probe(KINDS.index(kind), ctypes.c_void_p(r.contiguous().data_ptr()), ctypes.c_longlong(n),
                 ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0


@pytest.mark.parametrize("kind", ["rk4", "rkf45"])
def test_a_line_at_minus_zero(cuda, oracle_port, kind):
    shape = (12, 14, 16)
    x, y, z = np.meshgrid(*[np.arange(k, dtype=np.float32) for k in shape], indexing="ij")
    B = [np.full(shape, -0.0, np.float32), (0.2 + 0.01 * z).astype(np.float32), (1.0 + 0.02 * y).astype(np.float32)]
    g = np.random.default_rng(2)
    n = 64
    ys, zs = g.uniform(2.0, 8.0, n).astype(np.float32), g.uniform(2.0, 12.0, n).astype(np.float32)
    xs = np.where(np.arange(n) % 2, np.float32(-0.0), np.float32(0.0)).astype(np.float32)
    prm = P.reference_rk4() if kind == "rk4" else P.reference_rkf45()
    ref = oracle_port.trace_all("port32cr", *B, xs, ys, zs, s_len=0.125, tol_coef=0.5, params=prm)
    got = run_dropin(kind, *B, xs, ys, zs, 0.125, 0.5)
    # (the Fehlberg sums have terms of both signs and end at +0)
    assert kind != "rk4" or (np.signbit(ref["end_x"]).any() and not np.signbit(ref["end_x"]).all())
    for k in ("end_x", "start_x"):
        assert np.array_equal(got[k].view(np.int32), ref[k].view(np.int32)), k
