"""Which spans Grid2D.step takes to the resident launch: never one that is faster step by step."""
import pytest

from lens_sensor_b200 import _native as N
from lens_sensor_b200 import engine as E


def test_sums_a_step():
    e = N.Epi2D()
    e.iavg_n0 = 1 << 30
    assert E.sums_a_step(e, 0, 8) == 0
    e.dft_n0, e.dft_n1 = 4, 20
    assert E.sums_a_step(e, 0, 8) == 0          # a window without sums
    e.dft = 16
    assert [E.sums_a_step(e, n, 8) for n in (0, 4, 12, 17, 40)] == [1, 1, 1, 0, 0]
    e.dft_ex, e.dft_prev, e.iavg = 16, 16, 16
    e.prev_n0, e.prev_n1, e.iavg_n0 = 4, 12, 4
    assert E.sums_a_step(e, 4, 8) == 4 and E.sums_a_step(e, 4, 16) == 4 and E.sums_a_step(e, 12, 8) == 3
    e.iavg_n0 = 1 << 30
    assert E.sums_a_step(e, 4, 4) == 3


def test_steps_rise_with_rows_and_sums():
    for pol, top in (('s', 3), ('p', 4)):
        for threads, bands in ((256, 147), (256, 430), (384, 147), (384, 430)):
            of = [[E.resident_steps(pol, r, threads, bands, s) for s in range(top + 1)] for r in range(2, 21, 2)]
            assert of[0] == [0] * (top + 1)
            for a, b in zip(of, of[1:]):
                assert all(x <= y for x, y in zip(a, b)), (pol, threads, bands, a, b)
            assert all(sum(a) >= sum(b) for a, b in zip(of[::-1], of[-2::-1]))
    assert E.resident_steps('s', 20, 384, 147, 7) == E.resident_steps('s', 20, 384, 147, 3)


@pytest.mark.gpu
@pytest.mark.parametrize('pol,steps,window,launches', [
    ('p', 24, True, 72), ('p', 24, False, 1), ('p', 4, False, 8), ('s', 12, True, 24), ('s', 60, True, 1)])
def test_spans_of_a_full_chip(pol, steps, window, launches):
    """2400 x 513 cells, bands of 18 rows: inside its windows step by step (TM at any length)."""
    import torch
    from test_grid2d_resident import _grid
    g = _grid(pol, 2400, 513, True, 5)
    assert g.rs_plan[0] >= 18 and g.rs_plan[1] == 384
    tab = E.StepTable(7, steps, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    w = (7, 7 + steps) if window else (1 << 28, 1 << 28)
    ep = E.Epi2D(g, dft=w, dft_ex=pol == 'p', prev=w, iavg_n0=w[0])
    g.step(tab, 7, steps, ep)
    torch.cuda.synchronize()
    assert g.launches == launches
