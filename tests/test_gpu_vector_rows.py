"""The vector forms of the scatter paint and the separate-mesh readout at mesh
edges."""
import numpy
import pytest

from oracle import pmesh_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def G():
    import fastpm_gb300
    return fastpm_gb300


# one particle in every cell of an edge row: windows that end in, straddle and
# wrap past the 16-byte quads
@pytest.mark.parametrize('window', ['cic', 'tsc'])
@pytest.mark.parametrize('n', [16, 24])
def test_vector_paint_and_readout_at_quad_edges(G, n, window):
    import torch
    rng = numpy.random.RandomState(n)
    x = rng.uniform(size=(4 * n, 3)) * [1.0, n, 1.0] + [0, 0, 0]
    x[:, 2] = (numpy.arange(4 * n) // 4 + rng.uniform(size=4 * n)) % n   # every z cell
    pos = torch.from_numpy((x / n * 10.0).astype('f4')).cuda()
    pm = G.ParticleMesh(BoxSize=10.0, Nmesh=[n] * 3, resampler=window)
    real = pm.paint(pos, mass=2.0)
    opm = pmesh_np.ParticleMesh(BoxSize=10.0, Nmesh=[n] * 3, resampler=window)
    oreal = opm.paint(pos.cpu().numpy().astype('f8'), mass=2.0)
    # positions: float32 cell units below n, so offsets are n 2^-24 off; some 20 particles a cell
    numpy.testing.assert_allclose(real.numpy(), numpy.asarray(oreal.value), atol=20 * 2 * 3 * n * 2.0 ** -23)
    val = real.readout(pos)
    oval = oreal.readout(pos.cpu().numpy().astype('f8'))
    top = float(real.value.max())
    numpy.testing.assert_allclose(val.cpu().numpy(), oval, atol=top * 27 * n * 2.0 ** -22)
    # what lies outside the window does not count, be it infinite
    one = G.RealField(pm)
    one.value[0, 0, :] = float('inf')
    one.value[0, 0, 4:7] = 1.0
    p5 = torch.tensor([[0.0, 0.0, 5.0 / n * 10.0]], device='cuda')
    row = pm.paint(p5).value[0, 0].cpu().numpy()
    got = float(one.readout(p5)[0]) if window == 'tsc' else 1.0
    assert numpy.isfinite(got) and numpy.count_nonzero(row) in (1, 3)
