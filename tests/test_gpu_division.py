"""The complex quotient of the resident solves' scalar recurrences against Smith's algorithm with
rounded divisions, which it stands in for, and against 64-bit mantissas on the host."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess
from pathlib import Path

import numpy
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include "fdfd_resident.cuh"
__global__ void k(const double* ab, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const fdfd::dcx a = {ab[4 * i], ab[4 * i + 1]}, b = {ab[4 * i + 2], ab[4 * i + 3]};
  const fdfd::dcx q = fdfd::cdiv(a, b), s = fdfd::ddiv(a, b);
  out[4 * i] = q.re;
  out[4 * i + 1] = q.im;
  out[4 * i + 2] = s.re;
  out[4 * i + 3] = s.im;
}
extern "C" int run(const double* ab, double* out, int n) {
  k<<<(n + 255) / 256, 256>>>(ab, out, n);
  return (int)cudaDeviceSynchronize();
}
'''


@pytest.fixture(scope='module')
def quotients(cuda, tmp_path_factory):
    import torch
    from meanas_b200 import build
    nvcc = build.nvcc()
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip('no nvcc to compile the test kernel with')
    d = tmp_path_factory.mktemp('division')
    (d / 'q.cu').write_text(SOURCE)
    csrc = Path(build.__file__).resolve().parent / 'csrc'
    subprocess.run([nvcc, *build.ARCH, '-O3', '-std=c++17', '-Xcompiler', '-fPIC', '-shared', f'-I{csrc}',
                    '-o', str(d / 'q.so'), str(d / 'q.cu')], check=True)
    lib = C.CDLL(str(d / 'q.so'))

    def run(a, b):
        ab = torch.as_tensor(numpy.stack([a.real, a.imag, b.real, b.imag], 1), device=cuda).contiguous()
        out = torch.empty_like(ab)
        torch.cuda.synchronize()
        assert lib.run(C.c_void_p(ab.data_ptr()), C.c_void_p(out.data_ptr()), C.c_int(len(a))) == 0
        out = out.cpu().numpy()
        return out[:, :2], out[:, 2:]
    return run


def _errors(q, a, b):
    """|q - a / b| / |a / b| in units of 2^-53, formed with 64-bit mantissas."""
    L = numpy.longdouble
    ar, ai, br, bi = (v.astype(L) for v in (a.real, a.imag, b.real, b.imag))
    # a - q b relative to |a|, with q b exact to 2^-64
    qr, qi = q[:, 0].astype(L), q[:, 1].astype(L)
    er, ei = ar - (qr * br - qi * bi), ai - (qr * bi + qi * br)
    scale = numpy.maximum(abs(ar), abs(ai))
    size = numpy.sqrt((ar / scale) ** 2 + (ai / scale) ** 2)
    return (numpy.sqrt((er / scale) ** 2 + (ei / scale) ** 2) / size).astype(float) * 2.0 ** 53


def _complex(re, im):
    return re + 1j * im


@pytest.mark.parametrize('spread', [0, 10, 440])
def test_errors_are_those_of_rounded_divisions(quotients, spread):
    rng = numpy.random.default_rng(1)
    n = 400000

    def numbers():
        z = _complex(rng.standard_normal(n), rng.standard_normal(n))
        z[::3] = _complex(rng.standard_normal((n + 2) // 3) * 2.0 ** rng.uniform(-30, 0, (n + 2) // 3),
                          rng.standard_normal((n + 2) // 3))
        return z * 2.0 ** numpy.floor(rng.uniform(-spread, spread, n))
    a, b = numbers(), numbers()
    a[1::3] = (b * (1 + 1e-3 * rng.standard_normal(n)))[1::3]  # quotients close to the real axis
    q, s = quotients(a, b)
    eq, es = _errors(q, a, b), _errors(s, a, b)
    # rounding r, d (r's share of at most 1/2 and its own), the numerators (r's share of at most
    # 0.71 and their own) and the quotients: 4.21 roundings to first order
    assert max(eq.max(), es.max()) <= 4.3
    assert numpy.sqrt((eq ** 2).mean()) <= 1.01 * numpy.sqrt((es ** 2).mean())


def test_other_numbers_are_divided(quotients):
    """Beyond 2^+-450, zeros, infinities and NaN: the bits of the rounded divisions."""
    rng = numpy.random.default_rng(2)
    edge = numpy.array([0.0, -0.0, 5e-324, 2.0 ** -1022, 2.0 ** -451, 2.0 ** 451, 1.7e308, numpy.inf, -numpy.inf, numpy.nan])
    v = numpy.stack(numpy.meshgrid(*[edge] * 4, indexing='ij'), -1).reshape(-1, 4)
    with numpy.errstate(all='ignore'):
        a = numpy.empty(len(v), complex)
        b = numpy.empty(len(v), complex)
    a.real, a.imag, b.real, b.imag = v.T
    q, s = quotients(a, b)
    assert numpy.array_equal(numpy.isnan(q), numpy.isnan(s))
    assert numpy.array_equal(q[~numpy.isnan(q)].view(numpy.int64), s[~numpy.isnan(s)].view(numpy.int64))
    # just inside and just outside of the range
    for e in (-452, -451, -450, -449, 448, 449, 450, 451):
        a = _complex(rng.standard_normal(1000), rng.standard_normal(1000)) * 2.0 ** e
        b = _complex(rng.standard_normal(1000), rng.standard_normal(1000))
        for x, y in ((a, b), (b, a), (a, a[::-1])):
            q, s = quotients(x, y)
            assert max(_errors(q, x, y).max(), _errors(s, x, y).max()) <= 4.3
