"""The 2LPT state's own readout (fpm_lpt_readout) against the general one."""
import pytest

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
