"""The 2LPT state's own readout (fpm_lpt_readout) against the general one, and the
vector forms of the scatter paint and the separate-mesh readout at mesh edges."""
import numpy
import pytest

from oracle import pmesh_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def G():
    import fastpm_gb300
    return fastpm_gb300


# shift 0: lattice points are nodes; 0.25: they are not; -3: nodes, wrapped.
# 24^3 particles are whole warps, 17 (explicit) a ragged one
@pytest.mark.parametrize('shift, explicit', [(0.0, 0), (0.25, 0), (-3.0, 0), (0.0, 17), (0.0, 1000)])
def test_lpt_readout(G, shift, explicit):
    import torch
    from fastpm_gb300.force import _lpt_readout
    n = 24
    pm = G.ParticleMesh(BoxSize=60.0, Nmesh=[n] * 3)
    g = torch.Generator(device='cuda').manual_seed(4)
    meshes = torch.randn(3, n, n, n, generator=g, device='cuda')
    if explicit:
        Q = torch.rand(explicit, 3, generator=g, device='cuda', dtype=torch.float64) * 60.0
    else:
        Q = pm.generate_uniform_particle_grid(shift=shift)
    st = G.StateVector(G.Solver(pm, G.Planck15), Q)
    psi = torch.empty(len(Q), 3, device='cuda')
    _lpt_readout(pm, meshes, st, psi_out=psi)
    ref = torch.empty_like(psi)
    pm._readout([meshes[0], meshes[1], meshes[2]], [ref[:, 0], ref[:, 1], ref[:, 2]], [3, 3, 3], [1.0] * 3,
                q=st.q32, disp=None, lattice=st.lattice, resampler='cic')
    # eight products and their sum, each order: 8 roundings of values below 6
    assert float((psi - ref).abs().max()) <= 8 * 6 * 2.0 ** -24
    if shift == int(shift) and not explicit:
        assert torch.equal(psi, ref)
    first = torch.randn(len(Q), 3, generator=g, device='cuda')
    c1, c2 = (0.3, -2.0, 5.0), (0.01, 0.7, -1.0)
    for one in (False, True):
        out = [torch.full_like(psi, 9.0) for _ in range(3)]
        _lpt_readout(pm, meshes, st, psi1=None if one else first, out=out, c1=c1, c2=None if one else c2)
        for k in range(3):
            want = c1[k] * psi if one else c1[k] * first + c2[k] * psi
            assert torch.equal(out[k], want)


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
