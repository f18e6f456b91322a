"""A resident grid launch whose wait ran out: what it leaves is plainly invalid."""
import ctypes

import pytest

from lens_sensor_b200 import _native as N
from test_grid2d_resident import FIELDS, _grid


@pytest.mark.gpu
@pytest.mark.parametrize('hold', [True, False])
def test_whole_bands_and_their_sums_are_nan(hold):
    """The second band withholds its first row: the bands' fields and sums are NaN over whole rows.
    hold: the DFT window meets the span (its sums sit in shared memory meanwhile)."""
    import torch
    from lens_sensor_b200 import engine as E
    g = _grid('p', 140, 95, True, 5)
    tab = E.StepTable(7, 20, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    w = (7, 27) if hold else (1 << 28, 1 << 28)
    ep = E.Epi2D(g, boxes=[(0, 9, 0, 95), (0, 140, 0, 95)], dft=w, dft_ex=True, prev=(9, 20), iavg_n0=7,
                 planes={'a': 1, 'b': 2})
    st = g.lib.lens_tm2d_resident_watchdog_test(ctypes.byref(g.s), ctypes.byref(tab.s), ctypes.byref(ep.s), 7, 20,
                                                E._ptr(g.rs_scratch), g.rs_scratch.numel(), E._ptr(g.rs_err), None)
    assert st == 0
    torch.cuda.synchronize()
    with pytest.raises(N.LensError):
        g.check()
    bad = torch.isnan(g.view('ey')).any(dim=1)
    assert bool(bad[:2].all())      # the first band waits for the row, the second has none of its neighbour's then
    for q in FIELDS['p']:
        v = torch.isnan(g.view(q))
        assert torch.equal(v.any(dim=1), v.all(dim=1)) and torch.equal(v.any(dim=1), bad[:v.shape[0]]), q
    for q in ('dft', 'dft_ex', 'prev'):
        v = torch.isnan(getattr(ep, q)[:, :95])
        assert torch.equal(v.all(dim=2).all(dim=1), bad) and torch.equal(v.any(dim=2).any(dim=1), bad), q
    v = torch.isnan(ep.iavg[:, :95])
    assert torch.equal(v.all(dim=1), bad) and torch.equal(v.any(dim=1), bad)
    assert bool(torch.isnan(ep.box_acc[:2]).all())
    assert bool(torch.isnan(ep.plane_acc[0, :, :95]).all())
    for q in FIELDS['p']:        # the padding stays as it was
        full = getattr(g, q).clone()
        full[:g.view(q).shape[0], :g.view(q).shape[1]] = 0
        assert not bool(full.any()), q


@pytest.mark.gpu
def test_check_waits_for_the_launch():
    """The error word of a launch on another stream is read after that launch."""
    import torch
    from lens_sensor_b200 import engine as E
    g = _grid('s', 140, 96, False, 5)
    tab = E.StepTable(7, 20, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(400_000_000)      # 0.2 s
        g.rs_err.fill_(1)                   # as a wait that ran out leaves it
    g.step(tab, 7, 20, stream=s)
    with pytest.raises(N.LensError):
        g.check()
