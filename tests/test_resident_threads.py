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


@pytest.mark.gpu
def test_groups_of_one_kernel():
    """Resident groups (lens_rs2d_run) of narrow TE and wide lossy TM instances, the same kernels at
    other shared memory sizes."""
    import torch
    from dataclasses import replace
    from lens_sensor_b200 import batch2d as B
    from lens_sensor_b200 import engine as E
    from lens_sensor_b200.workloads import sweep2d
    dev = E._device(None)
    specs = sweep2d(count=4)[0]
    te, tm = (next(s for s in specs if s.pol == p) for p in 'sp')
    sps = [replace(te, nx=160, ny=120), replace(tm, nx=160)]
    steps, cut = 3000, 2
    insts = [[B.Instance(sp, steps, torch.float32, dev, window=(10, steps)) for sp in sps] for _ in range(2)]
    tabs = [E.StepTable(0, steps, q.spec.dt, q.omega, q.omega, E.cw_envelope(q.spec.f0)) for q in insts[0]]
    groups = [B.ResidentGroup([q], dev) for q in insts[0]]

    def job(g, tab):
        def run(s):
            for n in range(0, steps, cut):
                g.step(tab, n, cut, s)
        return run
    errs = _together([job(g, t) for g, t in zip(groups, tabs)])
    assert not errs, errs
    for g, q, b, tab in zip(groups, *insts, tabs):
        g.check()
        one = B.ResidentGroup([b], dev)
        one.step(tab, 0, steps)
        torch.cuda.synchronize()
        for x, y in zip(q.f, b.f):
            assert torch.equal(x, y)
        assert torch.equal(q.dft, b.dft)
