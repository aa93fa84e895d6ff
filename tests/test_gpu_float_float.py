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


@pytest.mark.parametrize('unitary', [False, True])
@pytest.mark.parametrize('n', [16, 48])
def test_whitenoise_rounds_as_float64(G, n, unitary):
    ref = pmesh_np.whitenoise([n] * 3, 99, unitary=unitary)
    got = G.ParticleMesh(BoxSize=1.0, Nmesh=[n] * 3).generate_whitenoise(99, unitary=unitary).numpy()
    for a, b in ((got.real, ref.real), (got.imag, ref.imag)):
        # half an ulp of the float32 result, and the 2^-36 of the float-float value (modulus up to about 6)
        assert (abs(a - b) <= 2.0 ** -24 * abs(b) * 1.01 + 6 * 2.0 ** -36).all()
