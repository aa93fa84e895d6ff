"""The gradient stencil for aligned and for unaligned meshes: the same bits."""
import pytest

pytestmark = pytest.mark.gpu


# a single quad tile, a ragged one (24, 48), several z tiles per row (192), planes in pairs (512)
@pytest.mark.parametrize('n', [16, 24, 48, 192, 512])
def test_aligned_and_unaligned_force_meshes(n):
    import torch
    import fastpm_gb300 as G
    from fastpm_gb300 import _lib
    pm = G.ParticleMesh(BoxSize=30.0, Nmesh=[n] * 3)
    g = torch.Generator(device='cuda').manual_seed(n)
    rho = torch.rand(n ** 3 + 4, generator=g, device='cuda')
    ws = _lib.query('fpm_force_workspace', n)
    work = torch.zeros(ws, dtype=torch.uint8, device='cuda')
    out = {}
    for off in (0, 2):   # floats past a 16-byte boundary (the density must be 8-byte aligned)
        r = rho[off:off + n ** 3]
        r.copy_(torch.arange(n ** 3, device='cuda').float().mul_(0.37).sin_().add_(1.5))
        packed = torch.zeros(4 * n ** 3 + 4, device='cuda')[2 * off:2 * off + 4 * n ** 3]   # 16-byte aligned only when off
        _lib.call('fpm_force_mesh_packed', _lib.ptr(r), n, pm.L, 0.7, 0.45, _lib.ptr(packed), None, _lib.ptr(work), ws,
                  _lib.stream_ptr())
        blocked = torch.zeros(4 * n ** 3, device='cuda')
        if not off:
            _lib.call('fpm_force_mesh_blocked', _lib.ptr(r), n, pm.L, 0.7, 0.45, _lib.ptr(blocked), None, _lib.ptr(work),
                      ws, _lib.stream_ptr())
            h = n // 2
            b = blocked.view(h, h, h, 2, 2, 2, 4).permute(0, 3, 1, 4, 2, 5, 6).reshape(n, n, n, 4)
            assert torch.equal(b, packed.view(n, n, n, 4))
        f = [torch.zeros(n ** 3 + 4, device='cuda')[off:off + n ** 3] for _ in range(3)]
        _lib.call('fpm_force_mesh', _lib.ptr(r), n, pm.L, 0.7, 0.45, _lib.ptr(f[0]), _lib.ptr(f[1]), _lib.ptr(f[2]), None,
                  _lib.ptr(work), ws, _lib.stream_ptr())
        for d in range(3):
            assert torch.equal(packed.view(-1, 4)[:, d], f[d])
        out[off] = packed.clone()
    assert torch.equal(out[0], out[2])
