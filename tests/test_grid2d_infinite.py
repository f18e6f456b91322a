"""Infinities and NaN in a field spread through the resident launch as through the step by step
kernels, whatever columns and rows they start from (a cell outside the strips has no psi to
make them NaN)."""
import pytest

from test_grid2d_resident import FIELDS, _grid


def _same(x, y):
    import torch
    return torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.nan_to_num(x, nan=0.0), torch.nan_to_num(y, nan=0.0))


@pytest.mark.gpu
@pytest.mark.parametrize('value', [float('inf'), -float('inf'), 3e38, float('nan')])
@pytest.mark.parametrize('size', [('s', 140, 96), ('p', 140, 96), ('s', 900, 431), ('p', 900, 431)])
def test_infinities_spread_alike(size, value, monkeypatch):
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny = size
    steps = 4
    a, b = (_grid(pol, nx, ny, True, 5) for _ in range(2))
    # in and beside the strips of either axis, at the source rows, in the lean rows, at band edges
    cells = [(5, 5), (30, 30), (13, 40), (nx // 2, 20), (nx // 2 + 9, ny - 30), (nx - 25, ny // 2), (nx // 3, 3), (70, ny // 2)]
    for g in (a, b):
        for q in FIELDS[pol]:
            for i, j in cells:
                g.view(q)[i, j] = value
    tab = E.StepTable(7, steps, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    ea, eb = (E.Epi2D(g, dft=(7, 7 + steps), dft_ex=pol == 'p', iavg_n0=7) for g in (a, b))
    a.step(tab, 7, steps, ea)
    assert a.launches == 1
    monkeypatch.setattr(E, 'RS_MIN_STEPS', 1 << 30)
    b.step(tab, 7, steps, eb)
    torch.cuda.synchronize()
    for q in FIELDS[pol]:
        assert _same(getattr(a, q), getattr(b, q)), q
    for q in b.psi:
        assert _same(a.psi[q], b.psi[q]), q
    for q in ('dft', 'iavg'):
        assert _same(getattr(ea, q), getattr(eb, q)), q
