"""3D grids at the ends of the fused pass's x chunks, against the two streaming passes: grids
whose x absorbers meet (every x plane a strip plane; nothing written behind the last), and long
thin ones with as many chunks as there may be or as the chip holds at once."""
import numpy as np
import pytest

TOL = 2e-5   # of the vector field's norm, as the two forms are compared elsewhere (tests/test_gpu_parity.py)


def _grid(dims, lossy, fused):
    import torch
    from lens_sensor_b200 import engine as E
    from lens_sensor_b200.geometry import cpml_axis
    nx, ny, nz = dims
    dx = 30e-9
    dt = 0.5 * dx / (299792458.0 * np.sqrt(3))
    rng = np.random.default_rng(4)
    shapes = [(nx - 1, ny, nz), (nx, ny - 1, nz), (nx, ny, nz - 1)]
    ce = [(dt / (8.854e-12 * dx) * rng.uniform(0.4, 1.0, s)).astype(np.float32) for s in shapes]
    da = [rng.uniform(0.98, 1.0, s).astype(np.float32) for s in shapes] if lossy else None
    g = E.Grid3D(nx, ny, nz, dx, dt, ce, da, [cpml_axis(n, 10, 10, dx, dt) for n in dims], None, fused=fused)
    for q in g.FIELDS:
        v = g.view(q)
        v.copy_(torch.from_numpy((rng.standard_normal(tuple(v.shape)) / (1 if q[0] == 'e' else 377)).astype(np.float32)))
    return g


def _close(a, b):
    for names in ('ex ey ez', 'hx hy hz'):
        v = [[g.view(q).double() for q in names.split()] for g in (a, b)]
        norm = float(sum((t ** 2).sum() for t in v[1])) ** 0.5
        for x, y in zip(*v):
            assert float((x - y).norm()) <= TOL * norm


@pytest.mark.gpu
@pytest.mark.parametrize('dims,lossy', [((3, 24, 40), False), ((11, 33, 31), True), ((17, 48, 40), True), ((20, 40, 70), False)])
def test_x_all_absorber(dims, lossy):
    import torch
    from lens_sensor_b200 import engine as E
    nx, ny, nz = dims
    a, b = _grid(dims, lossy, True), _grid(dims, lossy, False)
    assert a.s.ax.e.lo == nx and a.s.ax.h.lo == nx - 1
    # the fused grid's two buffers with one more plane each, which has to stay as it is
    big = []
    for k in range(2):
        for c, q in enumerate(a.FIELDS):
            t = torch.full((nx + 1,) + a.bufs[k][q].shape[1:], 7.0, device='cuda')
            t[:nx] = a.bufs[k][q]
            a.bufs[k][q] = t[:nx]
            a.s.f[k][c] = t.data_ptr()
            big.append(t)
    tab = E.StepTable(0, 9, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    for g in (a, b):
        g.step(tab, 0, 9)
    torch.cuda.synchronize()
    a.check_flag()
    assert all(bool((t[nx] == 7.0).all()) for t in big)
    _close(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize('dims,lossy', [((1200, 30, 30), False), ((1000, 33, 40), True), ((301, 33, 65), False), ((2500, 8, 20), True),
                                        ((601, 65, 97), False)])
def test_long_and_thin(dims, lossy):
    import torch
    from lens_sensor_b200 import engine as E
    a, b = _grid(dims, lossy, True), _grid(dims, lossy, False)
    tab = E.StepTable(0, 9, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    for g in (a, b):
        g.step(tab, 0, 9)
    torch.cuda.synchronize()
    a.check_flag()
    _close(a, b)
