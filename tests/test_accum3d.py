"""accum_e2 with four z cells a thread against one cell a thread (which misaligned averages
run): every extent parity, both targets, a shortened x range.  The two may fuse different
products of a sum of squares: within 8 roundings of each value."""
import ctypes

import pytest

from lens_sensor_b200 import _native as N


@pytest.mark.gpu
@pytest.mark.parametrize('target', [1, 2])
@pytest.mark.parametrize('nx,ny,nz,nxt', [(5, 4, 3, 5), (7, 9, 33, 7), (8, 17, 64, 6), (9, 8, 126, 9), (6, 23, 127, 4),
                                          (6, 5, 129, 6), (4, 7, 160, 4), (5, 6, 255, 3)])
def test_four_cells_a_thread(target, nx, ny, nz, nxt):
    import torch
    from lens_sensor_b200 import engine as E
    P = E.pitch_of(nz)
    gen = torch.Generator(device='cuda').manual_seed(3)
    g = N.Grid3D()
    g.nx, g.ny, g.nz, g.pitch = nx, ny, nz, P
    one = torch.ones(512, device='cuda')
    for q, n in (('ax', nx), ('ay', ny), ('az', nz)):
        a = getattr(g, q)
        for tag, m in (('e', n), ('h', n - 1)):
            setattr(a, tag, N.Profile(one.data_ptr(), one.data_ptr(), one.data_ptr(), m, 0, 0))
    shapes = [(nx - 1, ny, nz), (nx, ny - 1, nz), (nx, ny, nz - 1)] + [(nx, ny, nz)] * 3
    keep = [torch.zeros((nx, ny, P), device='cuda') for _ in shapes]
    for c, (t, s) in enumerate(zip(keep, shapes)):
        t[:s[0], :s[1], :s[2]] = torch.randn(s, generator=gen, device='cuda')
        g.f[0][c] = t.data_ptr()
    g.ce_x = g.ce_y = g.ce_z = keep[3].data_ptr()
    g.src = N.Source(-1, None, None, None, 0, 0, 0)
    start = torch.rand(nx * ny * P, generator=gen, device='cuda')
    a, b = start.clone(), torch.empty(nx * ny * P + 1, device='cuda')[1:].copy_(start)
    assert a.data_ptr() % 16 == 0 and b.data_ptr() % 16 == 4
    lib = N.load()
    for t in (a, b):
        N.check(lib.lens_fdtd3d_accum_e2(ctypes.byref(g), target, nxt, ctypes.c_void_p(t.data_ptr()), None))
    torch.cuda.synchronize()
    assert float((a - b).abs().max()) <= 8 * 2.0 ** -24 * float(b.abs().max())
    same = (b == start)
    assert torch.equal(a[same], start[same])
