"""Grids whose band plan differs with the number of detector boxes step on a resident launch with each."""
import pytest

from test_grid2d_resident import FIELDS, _grid


@pytest.mark.gpu
@pytest.mark.parametrize('size', [('p', 5200, 256), ('p', 5600, 230)])
def test_every_box_count_is_resident(size, monkeypatch):
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny = size
    steps = 12
    a, b = (_grid(pol, nx, ny, True, 5) for _ in range(2))
    tab = E.StepTable(7, steps, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    boxes = [(2, nx // 3, 3, ny - 2), (nx // 2, nx, 0, ny // 2), (5, 9, 5, 9), (nx - 40, nx, 0, ny)]
    for nbox in (0, 1, 2, 4):
        l0 = a.launches
        ea = E.Epi2D(a, boxes=boxes[:nbox])
        a.step(tab, 7, steps, ea)
        assert a.launches == l0 + 1, nbox
    a.check()
    with monkeypatch.context() as m:
        m.setattr(E, 'RS_MIN_STEPS', 1 << 30)
        for nbox in (0, 1, 2, 4):
            eb = E.Epi2D(b, boxes=boxes[:nbox])
            b.step(tab, 7, steps, eb)
    torch.cuda.synchronize()
    for q in FIELDS[pol]:
        assert torch.equal(getattr(a, q), getattr(b, q)), q
    assert float((ea.box_acc - eb.box_acc).abs().max()) <= 1e-12 * float(eb.box_acc.abs().max())
