"""Launch counts of the step by step 2D spans (lens_te2d_step_launches / lens_tm2d_step_launches):
host arithmetic on descriptors whose pointers are never followed."""
import ctypes

import pytest

from lens_sensor_b200 import _native as N


def _grid(pol, nx, ny, ptr=16):
    g = N.TE2D() if pol == 's' else N.TM2D()
    g.nx, g.ny, g.pitch = nx, ny, (ny + 31) // 32 * 32
    for f in ('ez', 'hx', 'hy', 'ce_e', 'ce_h') if pol == 's' else ('ex', 'ey', 'hz', 'ca_x', 'ca_y'):
        setattr(g, f, ptr)
    for ax, n in ((g.ax, nx), (g.ay, ny)):
        ax.e, ax.h = N.Profile(16, 16, 16, n, 0, 0), N.Profile(16, 16, 16, n - 1, 0, 0)
    g.src = N.Source(-1, None, None, None, 0, 0, 0)
    return g


def _count(pol, nx, ny, epi=None, drive=False, n0=0, n=10, ptr=16):
    lib = N.load()
    fn = lib.lens_te2d_step_launches if pol == 's' else lib.lens_tm2d_step_launches
    tab = N.StepTable(16, 16, 16, 16, 0, 100)
    d = ctypes.byref(N.Drive2D()) if drive else None
    return fn(ctypes.byref(_grid(pol, nx, ny, ptr)), ctypes.byref(tab), ctypes.byref(epi) if epi is not None else None, d, n0, n)


def _epi(box=False, dft=None):
    e = N.Epi2D()
    e.iavg_n0 = 1 << 30
    if box:
        e.nbox, e.box_acc = 1, 16
        e.box[0] = (ctypes.c_int * 4)(1, 9, 1, 9)
    if dft:
        e.dft, (e.dft_n0, e.dft_n1) = 16, dft
    return e


@pytest.mark.parametrize('pol,nx,ny,plain,box,window', [
    ('s', 140, 96, 2, 2, 2), ('p', 140, 96, 2, 3, 3),           # one cell a thread; TM's epilogue is a launch
    ('s', 2900, 400, 2, 2, 2), ('s', 3500, 400, 2, 3, 2),       # wide: boxes are a launch, small ones from 1.2 M cells;
    ('s', 8000, 300, 2, 3, 2), ('p', 4000, 200, 2, 3, 3)])      # TE sums with the E pass that holds the field
def test_launches_of_a_step(pol, nx, ny, plain, box, window):
    assert _count(pol, nx, ny) == 10 * plain
    assert _count(pol, nx, ny, _epi(box=True)) == 10 * box
    assert _count(pol, nx, ny, _epi(dft=(4, 8))) == 6 * plain + 4 * window
    assert _count(pol, nx, ny, _epi(dft=(4, 8)), n0=4, n=4) == 4 * window
    one = 2 if pol == 's' else 3
    assert _count(pol, nx, ny, _epi(box=True), drive=True) == 10 * one       # driven steps: one cell a thread
    assert _count(pol, nx, ny, _epi(box=True), ptr=20) == 10 * one           # so with arrays off 16 bytes
    assert _count(pol, nx, ny, n=0) == 0
    assert _count(pol, nx, ny, n0=95) == -1                                  # beyond the table: refused


@pytest.mark.gpu
@pytest.mark.parametrize('pol,nx,ny', [('s', 140, 96), ('p', 140, 96), ('p', 4000, 200), ('s', 9001, 513)])
def test_grid_counts_what_its_spans_launch(pol, nx, ny):
    """Grid2D.launches against the counting entry, over short spans and a driven one (no rows driven)."""
    import torch
    from lens_sensor_b200 import engine as E
    from test_grid2d_resident import _grid as grid
    g = grid(pol, nx, ny, True, 5)
    fn = g.lib.lens_te2d_step_launches if pol == 's' else g.lib.lens_tm2d_step_launches
    tab = E.StepTable(7, 4, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    ep = E.Epi2D(g, boxes=[(2, nx // 3, 3, ny - 2)], dft=(8, 9))
    drive = type('D', (), {'s': N.Drive2D()})()
    for n, e, d in ((1, None, None), (3, ep, None), (2, ep, drive), (0, ep, None)):
        want = fn(ctypes.byref(g.s), ctypes.byref(tab.s), ctypes.byref(e.s) if e else None,
                  ctypes.byref(d.s) if d else None, 7, n)
        was = g.launches
        g.step(tab, 7, n, e, drive=d)
        assert g.launches - was == want
    was = g.launches
    with pytest.raises(N.LensError):
        g.step(tab, 7, 5, ep)
    assert g.launches == was
    torch.cuda.synchronize()
