"""Grid2D.step on the resident launch (lens_te2d_resident / lens_tm2d_resident) against
the step by step kernels: the same bits in every field, psi array, DFT sum and time
average (the FP64 box and plane sums to 1e-12: their additions come in another order),
over bands of one row to the longest, odd and narrow and wide grids, warps whose upper
lanes lie beyond the columns, no source, full-length x psi, and spans cut anywhere."""
import ctypes

import numpy as np
import pytest

from lens_sensor_b200 import _native as N

FIELDS = {'s': ('ez', 'hx', 'hy'), 'p': ('ex', 'ey', 'hz')}
SUMS = ('dft', 'dft_ex', 'prev', 'iavg')


def _grid(pol, nx, ny, lossy, seed, npml=10, source=True, full_x=False, pec=(1, 1, 1, 1)):
    """A grid of random coefficients around a solve's, random fields and psi."""
    import torch
    from lens_sensor_b200 import engine as E
    from lens_sensor_b200.geometry import cpml_axis
    dx = 25e-9
    dt = 0.5 * dx / (299792458.0 * np.sqrt(2))
    rng = np.random.default_rng(seed)
    u = lambda *s: rng.uniform(0.6, 1.0, s).astype(np.float32)
    c = dt / (8.854e-12 * dx)
    if pol == 's':
        coef = dict(ce_e=u(nx, ny), ce_h=c * u(nx, ny))
        coef['ce_h'][: nx // 2] = coef['ce_h'][0]       # repeated rows (the plain form) and rows of their own
        coef['ce_e'][: nx // 2] = coef['ce_e'][0]
    else:
        coef = dict(ca_x=c * u(nx - 1, ny), ca_y=c * u(nx, ny - 1))
        coef['ca_x'][: nx // 2] = coef['ca_x'][0]
        coef['ca_y'][: nx // 2] = coef['ca_y'][0]
        if lossy:
            coef.update(da_x=u(nx - 1, ny), da_y=u(nx, ny - 1))
            coef['da_x'][: nx // 2] = coef['da_x'][0]
            coef['da_y'][: nx // 2] = coef['da_y'][0]
    n = ny if pol == 's' else ny - 1
    src = dict(ix=npml + 2, amp=u(n), ph1=u(n), ph2=u(n)) if source else None
    g = E.Grid2D(pol, nx, ny, dx, dt, coef, cpml_axis(nx, npml, npml, dx, dt, kappa_max=1.5),
                 cpml_axis(ny, npml, npml, dx, dt), src, pec=pec, full_x=full_x)
    gen = torch.Generator(device='cuda').manual_seed(seed)
    r = lambda t, s: t.copy_(torch.randn(t.shape, generator=gen, device='cuda') * s)
    for q in FIELDS[pol]:
        r(g.view(q), 1.0 if q[0] == 'e' else 1 / 377)
    for q, t in g.psi.items():
        r(t, 0.1 if q[0] == 'h' else 0.1 / 377)
    return g


def _epi(g, steps, window):
    from lens_sensor_b200 import engine as E
    nx, ny = g.nx, g.ny
    w = (7 + steps // 4, 7 + steps) if window else (1 << 28, 1 << 28)
    return E.Epi2D(g, boxes=[(2, nx // 3, 3, ny - 2), (nx // 2, nx, 0, ny // 2 + 1)], dft=w, dft_ex=g.pol == 'p',
                   prev=(w[0], w[0] + steps // 3), iavg_n0=w[0] + 1, planes={'a': nx // 4, 'b': nx - 2, 'c': 13})


CASES = [  # pol, nx, ny, lossy, steps, window, options
    ('s', 60, 33, False, 24, True, {}), ('p', 60, 65, True, 24, True, {}), ('p', 61, 64, False, 24, True, {}),
    ('s', 140, 96, False, 40, True, {}), ('p', 301, 130, True, 40, True, {}), ('s', 301, 191, False, 40, False, {}),
    ('s', 700, 289, False, 24, True, {}), ('p', 900, 257, False, 24, True, {}), ('s', 1500, 431, False, 20, True, {}),
    ('p', 1201, 431, True, 20, True, {}), ('s', 2300, 480, False, 12, True, {}), ('p', 2650, 420, True, 12, False, {}),
    ('s', 800, 577, False, 16, True, {}), ('p', 900, 760, True, 12, True, {}), ('s', 2200, 768, False, 8, False, {}),
    ('s', 90, 70, False, 16, True, dict(full_x=True)), ('p', 90, 70, True, 16, True, dict(source=False)),
    ('s', 200, 100, False, 16, True, dict(pec=(0, 1, 0, 1))), ('p', 200, 100, True, 16, True, dict(pec=(1, 0, 1, 0))),
]


@pytest.mark.gpu
@pytest.mark.parametrize('case', CASES, ids=lambda c: f'{c[0]}-{c[1]}x{c[2]}')
def test_resident_grid_keeps_the_bits(case, monkeypatch):
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny, lossy, steps, window, kw = case
    a, b, c = (_grid(pol, nx, ny, lossy, 5, **kw) for _ in range(3))
    assert a.rs_scratch is not None
    tab = E.StepTable(7, steps, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    ea, eb, ec = (_epi(g, steps, window) for g in (a, b, c))
    a.step(tab, 7, steps, ea)
    cut = steps // 3 + 1
    c.step(tab, 7, cut, ec)
    c.step(tab, 7 + cut, 2, ec)                    # a short span: step by step
    c.step(tab, 9 + cut, steps - cut - 2, ec)
    monkeypatch.setattr(E, 'RS_MIN_STEPS', 1 << 30)
    b.step(tab, 7, steps, eb)
    torch.cuda.synchronize()
    a.check()
    assert bool(torch.isfinite(b.view(FIELDS[pol][0])).all())
    for other, eo in ((a, ea), (c, ec)):
        for q in FIELDS[pol]:
            assert torch.equal(getattr(other, q), getattr(b, q)), q
        for q in b.psi:
            assert torch.equal(other.psi[q], b.psi[q]), q
        for q in SUMS:
            if getattr(eb, q) is not None:
                assert torch.equal(getattr(eo, q), getattr(eb, q)), q
        for q in ('box_acc', 'plane_acc'):
            x, y = getattr(eo, q), getattr(eb, q)
            assert float((x - y).abs().max()) <= 1e-12 * max(float(y.abs().max()), 1e-300), q
    assert float(eb.box_acc.abs().min()) > 0 and (not window or float(eb.plane_acc.abs().max()) > 0)


@pytest.mark.gpu
def test_two_streams_side_by_side():
    """Two grids advanced from two threads on two streams end with the bits they have alone."""
    import threading
    import torch
    from lens_sensor_b200 import engine as E
    gs = [_grid('s', 1500, 431, False, 5), _grid('p', 1201, 431, True, 6)]
    alone = [_grid('s', 1500, 431, False, 5), _grid('p', 1201, 431, True, 6)]
    tab = E.StepTable(7, 400, gs[0].dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in gs]

    def go(g, s):
        for n in range(7, 407, 50):
            g.step(tab, n, 50, None, s)
    ts = [threading.Thread(target=go, args=v) for v in zip(gs, streams)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    torch.cuda.synchronize()
    for g, b in zip(gs, alone):
        g.check()
        b.step(tab, 7, 400)
        torch.cuda.synchronize()
        for q in FIELDS[g.pol]:
            assert torch.equal(getattr(g, q), getattr(b, q)), q


@pytest.mark.gpu
def test_capture_takes_the_steps():
    """On a capturing stream the call is a sequence of plain launches (the resident entry declines)."""
    import torch
    from lens_sensor_b200 import engine as E
    a, b = _grid('s', 140, 96, False, 5), _grid('s', 140, 96, False, 5)
    tab = E.StepTable(7, 20, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            a.step(tab, 7, 20)
        g.replay()
    torch.cuda.synchronize()
    b.step(tab, 7, 20)
    torch.cuda.synchronize()
    assert torch.equal(a.ez, b.ez)


@pytest.mark.gpu
def test_watchdog_ends_the_launch():
    import torch
    from lens_sensor_b200 import engine as E
    a = _grid('s', 140, 96, False, 5)
    tab = E.StepTable(7, 20, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    st = N.load().lens_te2d_resident_watchdog_test(ctypes.byref(a.s), ctypes.byref(tab.s), 7, 20, E._ptr(a.rs_scratch),
                                                   a.rs_scratch.numel(), E._ptr(a.rs_err), None)
    assert st == 0
    torch.cuda.synchronize()
    with pytest.raises(N.LensError):
        a.check()
    assert bool(torch.isnan(a.ez).any())
    a.rs_err.zero_()
    for t in a.state():
        t.zero_()
    a.step(tab, 7, 20)
    torch.cuda.synchronize()
    a.check()
    assert bool(torch.isfinite(a.ez).all())


WIDE = [  # from the size the wide passes start at
    ('s', 8200, 257, False, {}), ('s', 3001, 401, False, {}), ('s', 16001, 130, False, {}), ('p', 2701, 263, True, {}),
    ('p', 5501, 128, False, {}), ('p', 1030, 700, True, {}), ('s', 4100, 513, False, dict(full_x=True)),
    ('p', 2700, 301, True, dict(source=False)), ('s', 4101, 500, False, dict(pec=(0, 1, 0, 1))),
    ('p', 2703, 300, True, dict(pec=(1, 0, 1, 0)))]


@pytest.mark.gpu
@pytest.mark.parametrize('rows', [False, True])
@pytest.mark.parametrize('case', WIDE, ids=lambda c: f'{c[0]}-{c[1]}x{c[2]}')
def test_wide_passes_keep_the_bits(case, rows, monkeypatch):
    """The four-columns-a-thread passes against the one-cell-a-thread kernels (which a
    driven step of no rows runs), coefficient rows read once or each its own."""
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny, lossy, kw = case
    steps = 8
    a, b = (_grid(pol, nx, ny, lossy, 9, **kw) for _ in range(2))
    monkeypatch.setattr(E, 'RS_MIN_STEPS', 1 << 30)
    if rows:
        co = [a.ce_e, a.ce_h] if pol == 's' else [a.ca_x, a.ca_y] + ([a.da_x, a.da_y] if lossy else [])
        a.rowref = E.repeated_rows(co)
        ref = a.rowref.cpu().numpy()
        assert (ref <= np.arange(nx)).all() and len(set(ref.tolist())) < nx
        for c in co:
            assert torch.equal(c[a.rowref.long()], c)
    tab = E.StepTable(7, steps, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    ea, eb = _epi(a, steps, True), _epi(b, steps, True)
    a.step(tab, 7, steps, ea)
    none = N.Drive2D()
    fn = b.lib.lens_te2d_step_driven if pol == 's' else b.lib.lens_tm2d_step_driven
    assert fn(ctypes.byref(b.s), ctypes.byref(tab.s), ctypes.byref(eb.s), ctypes.byref(none), 7, steps, None) == 0
    torch.cuda.synchronize()
    for q in FIELDS[pol]:
        assert torch.equal(getattr(a, q), getattr(b, q)), q
    for q in b.psi:
        assert torch.equal(a.psi[q], b.psi[q]), q
    for q in SUMS:
        if getattr(eb, q) is not None:
            assert torch.equal(getattr(ea, q), getattr(eb, q)), q
    for q in ('box_acc', 'plane_acc'):
        x, y = getattr(ea, q), getattr(eb, q)
        assert float((x - y).abs().max()) <= 1e-12 * max(float(y.abs().max()), 1e-300), q


@pytest.mark.gpu
def test_coefficients_written_in_place():
    """A large grid whose coefficients change after it was made steps with the new ones."""
    import torch
    from lens_sensor_b200 import engine as E
    a, b = (_grid('s', 3001, 401, False, 9) for _ in range(2))
    assert a.rowref is not None
    for g in (a, b):
        g.ce_e[1400:1500].mul_(0.75)
    tab = E.StepTable(7, 8, a.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))
    a.step(tab, 7, 8)
    assert b.lib.lens_te2d_step(ctypes.byref(b.s), ctypes.byref(tab.s), None, 7, 8, None) == 0
    torch.cuda.synchronize()
    for q in FIELDS['s']:
        assert torch.equal(getattr(a, q), getattr(b, q)), q
