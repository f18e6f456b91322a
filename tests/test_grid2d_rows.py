"""The table of repeated coefficient rows that the wide 2D passes read (lens_te2d_row_table /
lens_tm2d_row_table): formed from the coefficients each span steps with, however they were
written, and the same bits as every row read for itself."""
import ctypes

import pytest

from lens_sensor_b200 import _native as N
from test_grid2d_resident import FIELDS, WIDE, _epi, _grid

SIZES = [('s', 9001, 513, False), ('s', 90001, 65, False), ('p', 7003, 449, True), ('p', 9100, 513, False), ('s', 40001, 100, False)]  # from the table's least size


def _coef(g):
    return [c for c in ((g.ce_e, g.ce_h) if g.pol == 's' else (g.ca_x, g.ca_y, g.da_x, g.da_y)) if c is not None]


def _one_cell(g, tab, n0, steps, epi=None):
    """The one-cell-a-thread kernels (a driven step of no rows)."""
    fn = g.lib.lens_te2d_step_driven if g.pol == 's' else g.lib.lens_tm2d_step_driven
    e = ctypes.byref(epi.s) if epi is not None else None
    assert fn(ctypes.byref(g.s), ctypes.byref(tab.s), e, ctypes.byref(N.Drive2D()), n0, steps, None) == 0


def _tab(g, steps):
    from lens_sensor_b200 import engine as E
    return E.StepTable(7, steps, g.dt, 2.2e15, 2.2e15, E.cw_envelope(3.5e14))


def _same(a, b):
    import torch
    for q in FIELDS[a.pol]:
        assert torch.equal(getattr(a, q), getattr(b, q)), q
    for q in b.psi:
        assert torch.equal(a.psi[q], b.psi[q]), q


@pytest.mark.gpu
@pytest.mark.parametrize('case', SIZES, ids=lambda c: f'{c[0]}-{c[1]}x{c[2]}')
def test_table_is_the_first_row_of_each_run(case):
    import torch
    from lens_sensor_b200 import engine as E
    pol, nx, ny, lossy = case
    g = _grid(pol, nx, ny, lossy, 9)
    co = _coef(g)
    co[0][10:13] = co[0][9]                    # a run that the other arrays break or not
    co[-1][11].view(torch.int32)[ny - 2] ^= 1  # one bit of one value
    ref = torch.full((nx,), -1, dtype=torch.int32, device='cuda')
    fn = g.lib.lens_te2d_row_table if pol == 's' else g.lib.lens_tm2d_row_table
    assert fn(ctypes.byref(g.s), None, 0, 1 << 20, E._ptr(ref), None) == 0
    want = E.repeated_rows(co)
    if pol == 'p':      # the last row has no Ex: Ey's coefficients alone decide
        want[nx - 1] = E.repeated_rows([c for c in co[1::2]])[nx - 1] if bool(
            all(torch.equal(c[nx - 1], c[nx - 2]) for c in co[1::2])) else nx - 1
    assert torch.equal(ref, want)
    assert ref[12] != ref[10] and int((ref == torch.arange(nx, device='cuda')).sum()) < nx
    assert fn(ctypes.byref(g.s), None, 0, 1, E._ptr(ref), None) == N.ERR_SIZE   # one step does not gain by it


@pytest.mark.gpu
@pytest.mark.parametrize('case', SIZES, ids=lambda c: f'{c[0]}-{c[1]}x{c[2]}')
def test_steps_with_the_table(case):
    import torch
    pol, nx, ny, lossy = case
    a, b = (_grid(pol, nx, ny, lossy, 9) for _ in range(2))
    tab = _tab(a, 8)
    a.step(tab, 7, 8)
    _one_cell(b, tab, 7, 8)
    torch.cuda.synchronize()
    _same(a, b)
    assert int((a.rowref == torch.arange(nx, device='cuda')).sum()) < nx   # formed, with rows that repeat


WRITES = {  # ways to write a coefficient array that no counter of the array sees, and one that it does
    'data': lambda c: c.data[1400:1500].mul_(0.75),
    'dlpack': lambda c: __import__('torch').from_dlpack(__import__('torch').utils.dlpack.to_dlpack(c))[1400:1500].mul_(0.75),
    'inplace': lambda c: c[1400:1500].mul_(0.75),
}


@pytest.mark.gpu
@pytest.mark.parametrize('how', WRITES)
@pytest.mark.parametrize('pol', 'sp')
def test_coefficients_written_in_any_way(pol, how):
    """Rows 1400-1499 change by a factor that repeats (1400: a row of their own before)."""
    import torch
    a, b = (_grid(pol, 9000, 520, True, 9) for _ in range(2))
    assert a.rowref is not None
    tab = _tab(a, 40)
    for g in (a, b):
        g.step(tab, 7, 16)
        WRITES[how](_coef(g)[0])
    a.step(tab, 23, 16)
    _one_cell(b, tab, 23, 16)
    torch.cuda.synchronize()
    _same(a, b)


@pytest.mark.gpu
def test_captured_span_reads_the_coefficients_of_its_replay():
    import torch
    a, b = (_grid('s', 9001, 513, False, 9) for _ in range(2))
    tab = _tab(a, 16)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            a.step(tab, 7, 16)
        for g in (a, b):
            g.ce_e.data[1400:1500].mul_(0.75)
        graph.replay()
    torch.cuda.synchronize()
    _one_cell(b, tab, 7, 16)
    torch.cuda.synchronize()
    _same(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize('case', WIDE, ids=lambda c: f'{c[0]}-{c[1]}x{c[2]}')
def test_wide_passes_without_a_table(case):
    """Every row read for itself (NULL rowref) against the one-cell-a-thread kernels."""
    import torch
    pol, nx, ny, lossy, kw = case
    a, b = (_grid(pol, nx, ny, lossy, 9, **kw) for _ in range(2))
    tab = _tab(a, 8)
    ea, eb = _epi(a, 8, True), _epi(b, 8, True)
    fn = a.lib.lens_te2d_step_rows if pol == 's' else a.lib.lens_tm2d_step_rows
    assert fn(ctypes.byref(a.s), None, ctypes.byref(tab.s), ctypes.byref(ea.s), 7, 8, None) == 0
    _one_cell(b, tab, 7, 8, eb)
    torch.cuda.synchronize()
    _same(a, b)
    for q in ('dft', 'prev', 'iavg'):
        assert torch.equal(getattr(ea, q), getattr(eb, q)), q


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny', [(10001, 130), (6901, 200), (3701, 399)])
def test_tm_windows_with_a_table(nx, ny):
    """Grids whose fields lie in the L2 and, with their sums, beyond it: a table and wide passes inside the windows."""
    import torch
    a, b = (_grid('p', nx, ny, True, 9) for _ in range(2))
    a.rs_scratch, a.rowref = None, torch.empty(nx, dtype=torch.int32, device='cuda')   # step by step
    tab = _tab(a, 16)
    ea, eb = _epi(a, 16, True), _epi(b, 16, True)
    was = a.launches
    a.step(tab, 7, 16, ea)
    assert a.launches - was == 2 + 3 * 16
    _one_cell(b, tab, 7, 16, eb)
    torch.cuda.synchronize()
    _same(a, b)
    for q in ('dft', 'dft_ex', 'prev', 'iavg'):
        assert torch.equal(getattr(ea, q), getattr(eb, q)), q
    far = N.Epi2D.from_buffer_copy(ea.s)      # the same arrays, their windows elsewhere: nothing to gain
    far.dft_n0, far.dft_n1, far.prev_n0, far.prev_n1, far.iavg_n0 = 90, 99, 90, 99, 90
    assert a.lib.lens_tm2d_row_table(ctypes.byref(a.s), ctypes.byref(far), 7, 16, a.rowref.data_ptr(), None) == N.ERR_SIZE


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny', [(6900, 101), (5000, 200), (3501, 399), (3499, 401)])
@pytest.mark.parametrize('lossy', [True, False])
def test_tm_spans_into_their_windows(nx, ny, lossy):
    """TM grids on either side of the size from which the wide passes run inside the windows too."""
    import torch
    a, b = (_grid('p', nx, ny, lossy, 9) for _ in range(2))
    tab = _tab(a, 9)
    ea, eb = _epi(a, 9, True), _epi(b, 9, True)
    assert a.lib.lens_tm2d_step_rows(ctypes.byref(a.s), None, ctypes.byref(tab.s), ctypes.byref(ea.s), 7, 9, None) == 0
    _one_cell(b, tab, 7, 9, eb)
    torch.cuda.synchronize()
    _same(a, b)
    for q in ('dft', 'dft_ex', 'prev', 'iavg'):
        assert torch.equal(getattr(ea, q), getattr(eb, q)), q


@pytest.mark.gpu
@pytest.mark.parametrize('pol,nx,ny', [('s', 20001, 60), ('s', 39063, 128), ('s', 8999, 129), ('s', 4297, 256), ('s', 5061, 257),
                                       ('s', 7039, 256), ('s', 80001, 64), ('p', 12001, 64), ('p', 25001, 129), ('p', 17001, 130),
                                       ('p', 3901, 385), ('p', 8601, 256)])
@pytest.mark.parametrize('small', [True, False])
def test_either_side_of_the_wide_sizes(pol, nx, ny, small):
    """Spans of a plain step, steps with boxes, and steps with sums, by grid and box size."""
    import torch
    from lens_sensor_b200 import engine as E
    out = []
    for k in range(2):
        g = _grid(pol, nx, ny, pol == 'p' and small, 9)
        tab = _tab(g, 6)
        ep = E.Epi2D(g, boxes=[(5, 12, 3, ny - 2)] if small else [(5, nx // 2, 0, ny)], dft=(10, 12), dft_ex=pol == 'p')
        for n, e in ((7, None), (8, ep)):
            m = 1 if e is None else 5
            if k:
                fn = g.lib.lens_te2d_step_driven if pol == 's' else g.lib.lens_tm2d_step_driven
                assert fn(ctypes.byref(g.s), ctypes.byref(tab.s), ctypes.byref(e.s) if e else None, ctypes.byref(N.Drive2D()),
                          n, m, None) == 0
            else:
                fn = g.lib.lens_te2d_step if pol == 's' else g.lib.lens_tm2d_step
                assert fn(ctypes.byref(g.s), ctypes.byref(tab.s), ctypes.byref(e.s) if e else None, n, m, None) == 0
        torch.cuda.synchronize()
        out.append((g, ep))
    (a, ea), (b, eb) = out
    _same(a, b)
    assert torch.equal(ea.dft, eb.dft)
    assert float((ea.box_acc - eb.box_acc).abs().max()) <= 1e-12 * float(eb.box_acc.abs().max())
