"""The batched TM node DFT on sums that start on 8 bytes: the bits of the same sums on 16."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('storage', ['f32', 'f16'])
@pytest.mark.parametrize('persistent', [False, True])
def test_tm_sums_on_eight_bytes(storage, persistent):
    import torch
    from lens_sensor_b200 import batch2d as B
    from lens_sensor_b200 import engine as E
    from lens_sensor_b200.workloads import sweep2d
    sp = next(s for s in sweep2d(count=4)[0] if s.pol == 'p')
    st, dtype = B.DTYPES[storage]
    dev = E._device(None)
    out = []
    for off in (0, 2):
        q = B.Instance(sp, 120, dtype, dev, window=(20, 120))
        buf = torch.zeros(q.dft.numel() + 4, dtype=torch.float32, device=dev)
        q.dft = buf[off:off + q.dft.numel()].view(q.dft.shape)
        q.s.dft = q.dft.data_ptr()
        assert q.s.dft % 16 == 4 * off
        g = B.Group([q], st, 4, dev)
        tab = E.StepTable(0, 120, sp.dt, q.omega, q.omega, E.cw_envelope(sp.f0))
        (g.step_persistent if persistent else g.step)(tab, 0, 120)
        torch.cuda.synchronize()
        g.check()
        out.append(q.dft.clone())
        assert not buf[:off].any() and not buf[off + q.dft.numel():].any()
    assert bool(out[0].any()) and torch.equal(out[0], out[1])
