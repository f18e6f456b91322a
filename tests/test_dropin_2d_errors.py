"""The 2D drivers look at what a grid's steps reported: a grid whose launches ran out of their
waits ends the call with an error, not with a result."""
import json
import os
import types

import pytest

import _oracle_engine
from lens_sensor_b200 import _native as N
from lens_sensor_b200 import fdtd2d_core as D2

HERE = os.path.dirname(__file__)


class _FailedGrid(_oracle_engine.Grid2D):
    def step(self, *a, **kw):
        pass

    def check(self):
        raise N.LensError('a wait between bands timed out')


@pytest.mark.parametrize('name,method', [('dropin_2d_stitch', 'te'), ('dropin_2d_stitch', 'tm'),
                                         ('dropin_2d_sliding', None), ('dropin_2d', None)])
def test_a_timed_out_launch_raises(name, method, tmp_path, monkeypatch):
    gold = json.load(open(os.path.join(HERE, 'golden', name + '.json')))
    case = gold[method or sorted(gold)[0]]
    monkeypatch.chdir(tmp_path)
    eng = types.SimpleNamespace(**{k: v for k, v in vars(_oracle_engine).items() if not k.startswith('__')})
    eng.Grid2D = _FailedGrid
    monkeypatch.setattr(D2, 'E', eng)
    kw = dict(case['kw'])
    if case.get('stack'):
        kw['stack'] = [dict(L, n=complex(*L['n'])) for L in case['stack']]
    with pytest.raises(N.LensError):
        D2.run_beads(**kw)
