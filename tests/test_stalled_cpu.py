"""
MMX_STATUS_STALLED, which a launch reports whose blocks did not run together, is an error of every entry point that reads
states: the fields are not valid, and an inactive right-hand side must not pass for a converged one.  On state arrays
made up here; nothing is launched.
"""
from types import SimpleNamespace

import numpy as np
import pytest

from macromax_b200 import _native as nat


def _state(status, batch=1):
    st = np.zeros(batch, dtype=nat.STATE_DTYPE)
    st['iteration'], st['prev_norm'], st['residue'] = 3, 1.0, 0.5
    st['status'][-1] = status
    return st


def _engine(monkeypatch, status, batch=2):
    """An IterationEngine without a device, whose launches do nothing and whose states are those of an ended solve."""
    from macromax_b200.engine import IterationEngine
    monkeypatch.setattr(nat, 'load', lambda *a: SimpleNamespace(mmx_plan_chunk_ends=lambda plan, kind: 1))
    eng = object.__new__(IterationEngine)
    eng.plan, eng.chi_kind, eng.batch = SimpleNamespace(handle=None), nat.MMX_CHI_SCALAR, batch
    eng.read_state = lambda: _state(status, batch)
    eng.write_state = lambda st: None
    eng.iterate = lambda n, **kw: None
    return eng


def _run(eng):
    eng.run(1e-3, 10.0)


def _solution(eng):
    from macromax_b200 import Solution
    sol = object.__new__(Solution)
    sol._engine, sol._snapshot = eng, None
    sol.solve(None, rtol=1e-3, maxiter=10)


def _batch(eng):
    from macromax_b200.batch import BatchSolution
    b = object.__new__(BatchSolution)
    b.engine = eng
    b.solve(rtol=1e-3, maxiter=10)


def _uneven(eng):
    from macromax_b200.batch import UnevenBatch
    u = object.__new__(UnevenBatch)
    u.members, u.iterate = [SimpleNamespace(engine=eng)], lambda n: None
    u.solve(rtol=1e-3, maxiter=10)


def _mixed_uneven(eng):
    from macromax_b200.mixed import MixedUnevenSolution
    u = object.__new__(MixedUnevenSolution)
    u.members = [SimpleNamespace(_done=np.zeros(2, dtype=bool), _start=lambda *a: None, inner=SimpleNamespace(engine=eng),
                                 _outer_begin=lambda rtol: False, _outer_end=lambda: None)]
    u._uneven = SimpleNamespace(iterate=lambda n: None)
    u.solve(max_outer=1)


def _hook(eng):
    from macromax_b200.refhook import _FusedRunner
    r = object.__new__(_FusedRunner)
    r.engine, r.ncomp, r.shape = SimpleNamespace(fields=np.zeros((2, 1, 4))), 1, (4,)
    r.sync_out(SimpleNamespace(), eng.read_state())


@pytest.mark.parametrize('entry', [_run, _solution, _batch, _uneven, _mixed_uneven, _hook])
def test_stalled_states_raise(monkeypatch, entry):
    with pytest.raises(nat.NativeError):
        entry(_engine(monkeypatch, nat.MMX_STATUS_STALLED))


@pytest.mark.parametrize('entry', [_run, _solution, _batch, _uneven, _mixed_uneven])
def test_ended_states_do_not(monkeypatch, entry):
    entry(_engine(monkeypatch, nat.MMX_STATUS_TIMEOUT))
