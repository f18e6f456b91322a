"""Epilogue forms beyond the usual ones: the resident launch and the wide passes against the
one-cell-a-thread kernels."""
import ctypes

import pytest

from lens_sensor_b200 import _native as N
from test_grid2d_resident import FIELDS, _grid


def _tab(g, steps):
    from lens_sensor_b200 import engine as E
    return E.StepTable(7, steps, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))


def _one_cell(g, tab, n0, steps, epi):
    fn = g.lib.lens_te2d_step_driven if g.pol == 's' else g.lib.lens_tm2d_step_driven
    assert fn(ctypes.byref(g.s), ctypes.byref(tab.s), ctypes.byref(epi.s), ctypes.byref(N.Drive2D()), n0, steps, None) == 0


@pytest.mark.gpu
@pytest.mark.parametrize('pol', 'sp')
@pytest.mark.parametrize('windows', [((7, 15), (15, 23)), ((11, 23), (7, 15))])
def test_two_windows_on_one_array(pol, windows):
    """dft and dft_prev name the same sums (two windows of one phasor)."""
    import torch
    from lens_sensor_b200 import engine as E
    out = []
    for k in range(2):
        g = _grid(pol, 140, 96, True, 5)
        ep = E.Epi2D(g, dft=windows[0], prev=windows[1])
        ep.s.dft_prev = ep.s.dft
        tab = _tab(g, 16)
        if k == 0:
            g.step(tab, 7, 16, ep)
            assert g.launches == 1
        else:
            _one_cell(g, tab, 7, 16, ep)
        torch.cuda.synchronize()
        out.append(ep.dft)
    assert bool(out[1].any()) and torch.equal(*out)


@pytest.mark.gpu
@pytest.mark.parametrize('size', [('s', 140, 96), ('p', 140, 96), ('s', 3001, 401), ('p', 2703, 300)])
@pytest.mark.parametrize('resident', [True, False])
def test_boxes_beyond_the_grid(size, resident, monkeypatch):
    """Box ends anywhere in an int: the nodes of the grid that lie between them, none where they cross."""
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny = size
    lo, hi = -2 ** 31, 2 ** 31 - 1
    a, b = (_grid(pol, nx, ny, True, 5) for _ in range(2))
    tab = _tab(a, 6)
    monkeypatch.setattr(E, 'RS_MIN_STEPS', 4 if resident else 1 << 30)
    boxes = [(lo, 40, lo, hi), (10, lo, 0, ny), (nx - 9, hi, -5, ny + 5), (hi, lo, hi, lo)]
    ea, eb = E.Epi2D(a, boxes=boxes), E.Epi2D(b, boxes=[(0, 40, 0, ny), (0, 0, 0, 0), (nx - 9, nx, 0, ny), (0, 0, 0, 0)])
    a.step(tab, 7, 6, ea)
    _one_cell(b, tab, 7, 6, eb)
    torch.cuda.synchronize()
    x, y = ea.box_acc, eb.box_acc
    assert float(y[0]) > 0 and float(y[2]) > 0 and float(y[1]) == float(y[3]) == 0
    assert float((x - y).abs().max()) <= 1e-12 * float(y.abs().max())
    for q in FIELDS[pol]:
        assert torch.equal(getattr(a, q), getattr(b, q)), q
