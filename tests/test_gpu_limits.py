"""
What the default variant does at the ends of its range, against the runtime-radix passes: an alpha that the divergence
guard has raised beyond the range of the data type, solves from the alpha that an earlier solve left, and waits between
the blocks of a launch that run out or cannot be made.
"""
import os

import numpy as np
import pytest

from test_gpu_any_length import _problem
from test_gpu_fast import _solution, rel

pytestmark = pytest.mark.gpu


def _variants():
    from macromax_b200 import _native as nat
    return {'passes': nat.MMX_VARIANT_PASSES, 'loop': nat.MMX_VARIANT_LOOP, 'generic': nat.MMX_VARIANT_GENERIC}


# one CTA of 1D grids, chunks in one launch, passes with the length at run time and compiled for it
@pytest.mark.parametrize('shape,components,launches', [((300,), 1, 'loop'), ((300,), 3, 'loop'), ((44, 60), 1, 'loop'),
                                                       ((18, 20, 22), 3, 'loop'), ((44, 60), 1, 'passes'),
                                                       ((18, 20, 22), 3, 'passes'), ((90, 70, 72), 1, 'passes'),
                                                       ((60, 70, 72), 3, 'passes')])
def test_updates_are_rejected_when_alpha_is_out_of_range(shape, components, launches):
    """alpha_i^2 beyond the range of float: no update is accepted, and the solve does not count as converged."""
    from macromax_b200 import autotune
    sols = [_solution(_problem(shape, components, 'scalar'), np.complex64) for _ in range(2)]
    for s, name in zip(sols, (launches, 'generic')):
        autotune.set_variant(s._engine, _variants()[name])
        st = s._engine.read_state()
        st['alpha_im'] = 2e19
        s._engine.write_state(st)
        s.solve(None, rtol=0, maxiter=5)
        assert (s.iteration, s.rejections) == (5, 5)
        assert s._engine.read_state()['prev_norm'][0] == np.inf
        assert not np.any(s.E)


@pytest.mark.parametrize('n', [200, 300, 420, 800])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_repeated_solves_of_a_longitudinal_field(n, dtype):
    """A 1D vector field along the axis converges to rounding level long before its 200 iterations end, and the rejections
    that follow leave alpha raised: each of three solves in a row gives the field of the runtime-radix passes."""
    from macromax_b200 import autotune
    fast, gen = [_solution(_problem((n,), 3, 'scalar'), dtype) for _ in range(2)]
    autotune.set_variant(gen._engine, _variants()['generic'])
    for _ in range(3):
        for s in (fast, gen):
            s.E = 0.0
            s.solve(None, rtol=0, maxiter=200)
        assert (fast.iteration, fast.rejections, fast.alpha) == (gen.iteration, gen.rejections, gen.alpha)
        assert np.array_equal(fast.E, gen.E)


@pytest.mark.parametrize('shape,components', [((300, 420), 1), ((36, 44, 39), 3)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_waits_that_run_out_are_reported(shape, components, dtype):
    """The CTAs of a chunk in one launch look at the grid barrier once and give up: every state is marked, the host raises,
    and the next launch of the plan starts from cleared counters."""
    from macromax_b200 import _native as nat, autotune
    wl = _problem(shape, components, 'scalar')
    os.environ['MMX_LOOP_POLL_LIMIT'] = '0'
    try:
        sol = _solution(wl, dtype)
    finally:
        del os.environ['MMX_LOOP_POLL_LIMIT']
    eng = sol._engine
    autotune.set_variant(eng, nat.MMX_VARIANT_LOOP)
    assert nat.load().mmx_plan_chunk_ends(eng.plan.handle, eng.chi_kind) == 1
    for _ in range(2):
        with pytest.raises(nat.NativeError):
            sol.solve(None, rtol=0, maxiter=10)
        st = eng.read_state()[0]
        assert int(st['status']) == nat.MMX_STATUS_STALLED
        assert (int(st['active']), int(st['iteration'])) == (0, 0)
    # the same plan in passes, and another one whose waits may take their time
    other = _solution(wl, dtype)
    autotune.set_variant(other._engine, nat.MMX_VARIANT_LOOP)
    autotune.set_variant(eng, nat.MMX_VARIANT_PASSES)
    for s in (sol, other):
        s.E = 0.0
        s.solve(None, rtol=0, maxiter=10)
        assert s.iteration == 10
    assert rel(sol.E, other.E) < (1e-5 if dtype == np.complex64 else 1e-12)


@pytest.mark.parametrize('shape,components,batch', [((640, 600), 1, 1), ((80, 78, 77), 1, 1), ((300, 420), 1, 4)])
def test_refused_launches_run_in_passes(shape, components, batch):
    """Where the blocks of a chunk in one launch cannot all run at once the launch is refused: the chunk runs in passes
    instead, also as a member of an uneven batch, and so do the plan's later ones."""
    from macromax_b200 import Bound, Grid, _native as nat, autotune
    from macromax_b200.batch import BatchSolution, UnevenBatch
    wl = _problem(shape, components, 'scalar')
    grid = Grid(shape=shape, step=wl['step'])

    def make():
        return BatchSolution(grid, np.stack([wl['source']] * batch), wl['epsilon'], vacuum_wavelength=wl['wavelength'],
                             bound=Bound(grid, thickness=wl['bound_thickness']))

    def one_launch(s):
        return nat.load().mmx_plan_chunk_ends(s.engine.plan.handle, s.engine.chi_kind)

    os.environ['MMX_LOOP_SMS'] = '4096'
    try:
        sols = [make() for _ in range(3)]
    finally:
        del os.environ['MMX_LOOP_SMS']
    ref = make()
    assert one_launch(ref) == 1
    autotune.set_variant(ref.engine, nat.MMX_VARIANT_PASSES)
    ref.solve(rtol=0, maxiter=10)
    assert all(one_launch(s) == 1 for s in sols)
    sols[0].solve(rtol=0, maxiter=10)
    for _ in range(10):
        sols[1].iterate(1)
    UnevenBatch(sols[2:]).solve(rtol=0, maxiter=10)
    for s in sols:
        assert one_launch(s) == 0
        assert np.all(s.iterations == 10) and np.all(s.state['status'] == 0)
        assert np.array_equal(s.E, ref.E)


@pytest.mark.parametrize('wide', ['0', '1'])
def test_tile_width_leaves_the_schedule_alone(wide):
    """MMX_WIDE_GREEN chooses the tiles of the vector axis-0 pass and nothing else: a grid whose chunks run in one launch
    keeps them, a grid with the fused epilogue has its bits; and the pass itself, reached with MMX_VARIANT_PASSES, gives the
    same bits with both tile widths."""
    from macromax_b200 import _native as nat, autotune, workloads as w
    ragged = _problem((128, 40, 45), 3, 'scalar')
    box = w.spheres_3d(n=128, nb_spheres=20)
    box = {**box, 'shape': (128, 64, 64), 'epsilon': box['epsilon'][:, :64, :64], 'source': box['source'][..., :64, :64]}
    sols = {}
    for name, env in (('set', wide), ('unset', None)):
        if env is not None:
            os.environ['MMX_WIDE_GREEN'] = env
        try:
            sols[name] = [_solution(x) for x in (ragged, box, box)]
        finally:
            os.environ.pop('MMX_WIDE_GREEN', None)
        autotune.set_variant(sols[name][2]._engine, nat.MMX_VARIANT_PASSES)
    for a, b in zip(sols['set'], sols['unset']):
        ends = [nat.load().mmx_plan_chunk_ends(s._engine.plan.handle, s._engine.chi_kind) for s in (a, b)]
        assert ends[0] == ends[1]
        for s in (a, b):
            s.solve(None, rtol=0, maxiter=12)
        assert np.array_equal(a.E, b.E)
    one = sols['unset'][0]._engine
    assert nat.load().mmx_plan_chunk_ends(one.plan.handle, one.chi_kind) == 1


@pytest.mark.parametrize('shape,components,launches', [((300,), 1, 'loop'), ((300,), 3, 'loop'), ((44, 60), 1, 'loop'),
                                                       ((18, 20, 22), 3, 'loop'), ((44, 60), 1, 'passes'), ((300,), 1, 'passes')])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_a_status_keeps_the_field(shape, components, launches, dtype):
    """An update after one of norm 0 ends a right-hand side with MMX_STATUS_ZERODIV: its field is that before the update,
    also when the last decision before had accepted one."""
    from macromax_b200 import _native as nat, autotune
    sol = _solution(_problem(shape, components, 'scalar'), dtype)
    eng = sol._engine
    autotune.set_variant(eng, _variants()[launches])
    sol.solve(None, rtol=0, maxiter=4)
    field = sol.E
    st = eng.read_state()
    assert st['accepted'][0] == 1
    st['prev_norm'], st['active'], st['maxiter'] = 0.0, 1, np.inf
    eng.write_state(st)
    eng.iterate(3)
    after = eng.read_state()
    assert (after['status'][0], after['active'][0], after['iteration'][0]) == (nat.MMX_STATUS_ZERODIV, 0, 5)
    assert after['cur'][0] == st['cur'][0]
    assert np.array_equal(sol.E, field)
