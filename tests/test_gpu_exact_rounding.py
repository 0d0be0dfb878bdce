"""The exact tracers' float forms of the reference's double arithmetic against
the double arithmetic itself, bit for bit: the corner weights
(weights_exact) at fractions of every kind a sample can have, the step
controller's power (step_scale_exact) at every float near its range, the
offsets and quotients by constants, and a vector over its norm (unit_exact)
against the IEEE square root and divisions."""
import ctypes
import subprocess

import pytest
import torch

from fastqsl_gb300 import _build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "qsl_scott.cuh"
using namespace qsl;
__device__ bool same(float a, float b) { return a == b || (isnan(a) && isnan(b)); }
__global__ void k_weights(const float* r, long long n, unsigned long long* bad) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < n; i += step) {
        const float rx = r[3 * i], ry = r[3 * i + 1], rz = r[3 * i + 2], rxy = rx * ry;
        const double ox = 1.0 - (double)rx, oy = 1.0 - (double)ry, oz = 1.0 - (double)rz;
        const float e[8] = {(float)(ox * oy * oz), (float)(ox * oy * (double)rz), (float)(ox * (double)ry * oz),
                            (float)(ox * (double)ry * (double)rz), (float)((double)rx * oy * oz),
                            (float)((double)rx * oy * (double)rz), (float)((double)rxy * oz), rxy * rz};
        float w[8];
        weights_exact(rx, ry, rz, w);
        bool ok = true;
        for (int q = 0; q < 8; ++q) ok &= same(w[q], e[q]);
        if (!ok) atomicAdd(bad, 1ull);
    }
}
__global__ void k_scale(unsigned first, long long n, unsigned long long* bad) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < n; i += step) {
        const float q = __uint_as_float(first + (unsigned)i);
        if (!same(step_scale_exact(q), pow_cr((float)((double)q / 11.09), 0.2f))) atomicAdd(bad, 1ull);
    }
}
__global__ void k_unit(const float* r, long long n, unsigned long long* bad) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < n; i += step) {
        const float x = r[3 * i], y = r[3 * i + 1], z = r[3 * i + 2];
        const float nb = sqrtf(x * x + y * y + z * z);
        const float3 u = unit_exact(v3(x, y, z));
        if (!(same(u.x, x / nb) && same(u.y, y / nb) && same(u.z, z / nb))) atomicAdd(bad, 1ull);
    }
}
__global__ void k_constants(const float* r, long long n, unsigned long long* bad) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < n; i += step) {
        const float x = r[i];
        bool ok = same(add_const_exact(x, PlusMilli{}), (float)((double)x + 0.001));
        ok &= same(-add_const_exact(-x, PlusMilli{}), (float)((double)x - 0.001));
        ok &= same(div_const_exact(x, 0.002f, 1.f / 0.002f), x / 0.002f);
        ok &= same(sixth_exact(x), (float)(1.0 / 6.0 * (double)x));
        const double td = (double)(0.25f * x), q = td * kInvPi, m = __fma_rn(-q, kRefPi, td);
        const double w = over_4pi(x, __fma_rn(m, kInvPi * (1.0 + 0x1p-20), q), __fma_rn(m, kInvPi * (1.0 - 0x1p-20), q));
        ok &= w == (double)x / 4.0 / kRefPi || isnan(w);
        if (!ok) atomicAdd(bad, 1ull);
    }
}
extern "C" int probe_unit(const float* r, long long n, unsigned long long* bad) {
    k_unit<<<1216, 128>>>(r, n, bad);
    return cudaDeviceSynchronize();
}
extern "C" int probe_constants(const float* r, long long n, unsigned long long* bad) {
    k_constants<<<1216, 128>>>(r, n, bad);
    return cudaDeviceSynchronize();
}
extern "C" int probe_weights(const float* r, long long n, unsigned long long* bad) {
    k_weights<<<1216, 128>>>(r, n, bad);
    return cudaDeviceSynchronize();
}
extern "C" int probe_scale(unsigned first, long long n, unsigned long long* bad) {
    k_scale<<<1216, 128>>>(first, n, bad);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_probe")
    src, lib = d / "probe.cu", d / "probe.so"
    src.write_text(SOURCE)
    subprocess.run([_build.NVCC, *_build.COMMON, *_build.ARCH, "-fmad=false", "-shared", "-cudart", "static", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    return ctypes.CDLL(str(lib))


def _fractions(kind, n):
    g = torch.Generator(device="cuda").manual_seed(11)
    u = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64)
    if kind.startswith("below"):  # c - floor(c) of coordinates below a size
        c = (u * float(kind[5:])).float()
        return c - c.floor()
    if kind.startswith("bits"):   # short fractions, whose products tie
        b = int(kind[4:])
        return (torch.floor(u * 2 ** b) / 2 ** b).float()
    if kind == "tiny":            # down to 2^-60: the error terms' underflow guard
        return (u * torch.pow(2.0, -60.0 * torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64))).float()
    if kind == "faces":           # pinned to a face on some axes
        return torch.where(u < 0.3, 0.0, torch.where(u < 0.5, 1.0, u)).float()
    return torch.where(u < 0.05, float("nan"), 3.0 * u - 1.0).float()  # extrapolating cells, and NaN


@pytest.mark.parametrize("kind", ["below1", "below64", "below1024", "bits1", "bits9", "bits16", "bits17", "bits18",
                                  "tiny", "faces", "outside"])
def test_exact_weights_equal_the_double_form(probe, kind):
    n = 1 << 22
    r = _fractions(kind, n).contiguous()
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert probe.probe_weights(ctypes.c_void_p(r.data_ptr()), ctypes.c_longlong(n), ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0


# every float of [2^-18, 2^25) (the float form covers [2^-16, 2^23]), the
# smallest and largest floats, infinity and NaN
@pytest.mark.parametrize("first,count", [(0x36800000, 0x4C000000 - 0x36800000), (0, 1 << 16), (0x7F7FFF00, 0x200)])
def test_exact_step_scale_equals_the_double_form(probe, first, count):
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert probe.probe_scale(ctypes.c_uint(first), ctypes.c_longlong(count), ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0


@pytest.mark.parametrize("kind", ["plain", "small", "uneven", "zeros", "extreme", "nodes"])
def test_exact_unit_vector_equals_the_library(probe, kind):
    n = 1 << 22
    g = torch.Generator(device="cuda").manual_seed(13)
    r = torch.randn(n, 3, generator=g, device="cuda")
    e = torch.rand(n, 3, generator=g, device="cuda")
    if kind == "small":
        r = r * 1e-6
    elif kind == "uneven":    # components far apart
        r = r * torch.pow(10.0, -25.0 * e)
    elif kind == "zeros":
        r = torch.where(e < 0.4, 0.0, r)
    elif kind == "extreme":   # squares that over- and underflow
        r = r * torch.pow(10.0, 60.0 * e[:, :1] - 40.0)
    elif kind == "nodes":     # few significant bits
        r = torch.round(r * 8.0)
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert probe.probe_unit(ctypes.c_void_p(r.contiguous().data_ptr()), ctypes.c_longlong(n),
                            ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0


@pytest.mark.parametrize("kind", ["coordinates", "near0", "powers", "all"])
def test_exact_constants_equal_the_double_form(probe, kind):
    n = 1 << 22
    g = torch.Generator(device="cuda").manual_seed(17)
    u = torch.rand(n, generator=g, device="cuda")
    if kind == "coordinates":
        x = 600.0 * u - 4.0
    elif kind == "near0":
        x = (u - 0.5) * 0.01
    elif kind == "powers":
        x = torch.round(u * 512.0) * torch.pow(2.0, -torch.floor(8.0 * torch.rand(n, generator=g, device="cuda")))
    else:                     # every kind of float
        x = torch.randint(-(1 << 31), (1 << 31) - 1, (n,), generator=g, device="cuda", dtype=torch.int64)
        x = x.to(torch.int32).view(torch.float32)
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert probe.probe_constants(ctypes.c_void_p(x.contiguous().data_ptr()), ctypes.c_longlong(n),
                                 ctypes.c_void_p(bad.data_ptr())) == 0
    assert bad.item() == 0
