"""Kernels whose float64 work runs as float-float (csrc/ff.cuh): the shell sums of the
power spectrum, the whitenoise values and the k-space transfers of the adjoint."""
import ctypes

import numpy
import pytest

from oracle import pmesh_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def G():
    import fastpm_gb300
    return fastpm_gb300


def _modes(G, n, seed, scale=1.0):
    rng = numpy.random.RandomState(seed)
    v = (rng.normal(size=(n, n, n // 2 + 1)) + 1j * rng.normal(size=(n, n, n // 2 + 1))).astype('c8') * numpy.float32(scale)
    pm = G.ParticleMesh(BoxSize=50.0, Nmesh=[n] * 3)
    return pm, pm.complex_from(v), v.astype('c16')


def _sums(G, f1, f2, n):
    import torch
    from fastpm_gb300 import _lib
    s = torch.zeros((3, n // 2), dtype=torch.float64, device='cuda')
    _lib.call('fpm_power_accumulate', _lib.ptr(f1.data), _lib.ptr(f2.data) if f2 is not None else None, n, 50.0,
              _lib.ptr(s[0]), _lib.ptr(s[1]), _lib.ptr(s[2]), _lib.stream_ptr())
    return s.cpu().numpy()


def _freq(n):
    f = numpy.fft.fftfreq(n, 1.0 / n)
    return f.reshape(-1, 1, 1), f.reshape(1, -1, 1), numpy.arange(n // 2 + 1.0).reshape(1, 1, -1)


# values in float32's middle, squares past float32's range on either side, and zeros
@pytest.mark.parametrize('scale', [1.0, 1e-17, 1e-24, 1e15])
@pytest.mark.parametrize('n', [16, 24, 96])
def test_power_sums(G, n, scale):
    pm, f1, v1 = _modes(G, n, n, scale)
    _, f2, v2 = _modes(G, n, n + 1, scale)
    f1.value[1, 2, 3] = 0
    v1[1, 2, 3] = 0
    fx, fy, fz = _freq(n)
    q = fx ** 2 + fy ** 2 + fz ** 2
    d = numpy.floor(numpy.sqrt(q)).astype(int)
    w = numpy.where((fz == 0) | (fz == n // 2), 1.0, 2.0) * numpy.ones_like(q)
    ok = d < n // 2
    for other, vo in ((None, v1), (f2, v2)):
        k, p, c = _sums(G, f1, other, n)
        ref = [numpy.bincount(d[ok], weights=(x * w)[ok], minlength=n // 2)
               for x in (numpy.sqrt(q) * (2 * numpy.pi / 50.0), abs(v1 * vo.conj()), numpy.ones_like(q))]
        assert numpy.array_equal(c, ref[2])
        # a float64 sum of m positive terms: m 2^-53 of it, m < 15000 here
        numpy.testing.assert_allclose(k, ref[0], rtol=2e-12)
        numpy.testing.assert_allclose(p, ref[1], rtol=2e-12)


def test_power_not_finite(G):
    n = 16
    pm, f1, v1 = _modes(G, n, 3)
    f1.value[2, 1, 0] = float('inf')   # shell 2
    p = _sums(G, f1, None, n)[1]
    assert not numpy.isfinite(p[2]) and numpy.isfinite(numpy.delete(p, 2)).all()


@pytest.mark.parametrize('unitary', [False, True])
@pytest.mark.parametrize('n', [16, 48])
def test_whitenoise_rounds_as_float64(G, n, unitary):
    ref = pmesh_np.whitenoise([n] * 3, 99, unitary=unitary)
    got = G.ParticleMesh(BoxSize=1.0, Nmesh=[n] * 3).generate_whitenoise(99, unitary=unitary).numpy()
    for a, b in ((got.real, ref.real), (got.imag, ref.imag)):
        # half an ulp of the float32 result, and the 2^-36 of the float-float value (modulus up to about 6)
        assert (abs(a - b) <= 2.0 ** -24 * abs(b) * 1.01 + 6 * 2.0 ** -36).all()


@pytest.mark.parametrize('scale', [-1.0, 1e-9])   # 1e-9: the FP64 form
@pytest.mark.parametrize('n', [16, 24, 64, 96])
def test_kspace_combine(G, n, scale):
    from fastpm_gb300 import _lib
    pw = [(1, 0, 0), (0, 1, 1), (0, 0, 2)]
    lap = [1, 1, 0]
    fields = [_modes(G, n, 7 + s) for s in range(3)]
    pm = fields[0][0]
    out = G.ComplexField(pm)
    ptrs, keep = _lib.ptr_array([f[1].data for f in fields])
    _lib.call('fpm_kspace_combine', ptrs, 3, (ctypes.c_int * 9)(*[x for p in pw for x in p]), (ctypes.c_int * 3)(*lap),
              _lib.ptr(out.data), n, 50.0, scale, _lib.stream_ptr())
    fx, fy, fz = _freq(n)
    a = [(8 * numpy.sin(2 * numpy.pi * f / n) - numpy.sin(4 * numpy.pi * f / n)) * n / 300.0 for f in (fx, fy, fz)]
    q = fx ** 2 + fy ** 2 + fz ** 2
    k2 = numpy.where(q == 0, numpy.inf, q * (2 * numpy.pi / 50.0) ** 2)
    ref, size = 0, 0
    for (_, _, v), p, l in zip(fields, pw, lap):
        t = scale * v * (1j * a[0]) ** p[0] * (1j * a[1]) ** p[1] * (1j * a[2]) ** p[2] / (k2 if l else 1.0)
        ref, size = ref + t, size + abs(t)
    # float32 rounding of the result; sin(pi) is 1e-16 in the reference, 0 in the table
    err = abs(out.numpy() - ref)
    assert (err <= 2.0 ** -23 * abs(ref) + 2.0 ** -40 * (size + abs(scale))).all()


def test_kspace_combine_infinity(G):
    from fastpm_gb300 import _lib
    pm, f, v = _modes(G, 16, 1)
    f.value[1, 1, 1] = complex(float('inf'), 1.0)
    out = G.ComplexField(pm)
    ptrs, keep = _lib.ptr_array([f.data])
    _lib.call('fpm_kspace_combine', ptrs, 1, (ctypes.c_int * 3)(0, 0, 0), (ctypes.c_int * 1)(0), _lib.ptr(out.data), 16,
              50.0, 2.0, _lib.stream_ptr())
    got = out.numpy()
    assert got[1, 1, 1] == complex(float('inf'), 2.0)
    v[1, 1, 1] = 0
    got[1, 1, 1] = 0
    numpy.testing.assert_array_equal(got, (2 * v).astype('c8'))
