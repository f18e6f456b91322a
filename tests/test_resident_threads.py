"""Resident launches issued from two threads at once: a kernel that both use at different
shared memory sizes is planned and launched for each as alone."""
import threading

import pytest

from test_grid2d_resident import FIELDS, _grid


def _together(jobs):
    """Run the jobs side by side, each on a stream and thread of its own; their exceptions."""
    import torch
    errs, go = [], threading.Barrier(len(jobs))

    def run(job):
        try:
            go.wait()
            job(torch.cuda.Stream())
        except Exception as e:
            errs.append(e)
    torch.cuda.synchronize()
    ts = [threading.Thread(target=run, args=(j,)) for j in jobs]
    [t.start() for t in ts]
    [t.join() for t in ts]
    torch.cuda.synchronize()
    return errs


@pytest.mark.gpu
@pytest.mark.parametrize('pols', ['ss', 'sp'])
def test_grids_of_one_kernel(pols):
    """Equal sizes, one grid inside its DFT window (whose sums the launch holds in shared memory)."""
    import torch
    from lens_sensor_b200 import engine as E
    calls, n = 1500, 4
    gs = [_grid(p, 140, 96, True, 5) for p in pols]
    alone = [_grid(p, 140, 96, True, 5) for p in pols]
    tab = E.StepTable(7, calls * n, gs[0].dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    eps = [[E.Epi2D(v[0], dft=(7, 7 + calls * n)), None] for v in (gs, alone)]

    def job(g, ep):
        def run(s):
            for k in range(calls):
                g.step(tab, 7 + k * n, n, ep, s)
        return run
    errs = _together([job(g, ep) for g, ep in zip(gs, eps[0])])
    assert not errs, errs
    for g, b, ea, eb in zip(gs, alone, *eps):
        assert g.launches == calls      # one resident launch a call
        g.check()
        b.step(tab, 7, calls * n, eb)
        torch.cuda.synchronize()
        for q in FIELDS[g.pol]:
            assert torch.equal(getattr(g, q), getattr(b, q)), q
        if ea is not None:
            assert torch.equal(ea.dft, eb.dft)
