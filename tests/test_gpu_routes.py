"""
Which way the iterations of a plan go: the grids of these cases run their chunks in one launch, or in passes with a kernel of
their length on every axis, which is checked before the fields are.
"""
import numpy as np
import pytest

from test_gpu_any_length import _problem
from test_gpu_fast import _solution, rel

pytestmark = pytest.mark.gpu


def _compare(shape, components, medium, dtype, variant, one_launch, iterations):
    from macromax_b200 import _native as nat, autotune
    wl = _problem(shape, components, medium)
    fast, gen = _solution(wl, dtype), _solution(wl, dtype, generic=True)
    eng = fast._engine
    autotune.set_variant(eng, variant)
    assert nat.load().mmx_plan_chunk_ends(eng.plan.handle, eng.chi_kind) == one_launch
    for s in (fast, gen):
        s.solve(None, rtol=0, maxiter=iterations)
    assert fast.iteration == gen.iteration == iterations
    tol = 1e-5 if dtype == np.complex64 else 1e-12  # a few roundings per iteration of a contraction
    assert rel(fast.E, gen.E) < tol
    assert fast.residue == pytest.approx(gen.residue, rel=10 * tol)


# enough tiles for the kernels compiled for their length on every axis: the smallest and the largest, odd ones, radix 16
@pytest.mark.parametrize('shape,components,medium', [((35, 72, 80), 3, 'scalar'), ((143, 66, 75), 1, 'scalar'),
                                                     ((32, 182, 77), 3, 'symmetric'), ((192, 70, 72), 1, 'scalar'),
                                                     ((60, 110, 169), 3, 'scalar'), ((112, 108, 45), 3, 'symmetric'),
                                                     ((64, 96, 90), 3, 'general')])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_passes_of_own_lengths(shape, components, medium, dtype):
    from macromax_b200 import _native as nat
    _compare(shape, components, medium, dtype, nat.MMX_VARIANT_PASSES, 0, 6)


# several rows per tile and kept tile, more tiles than CTAs, every kind of chi; the largest grids keep most of an SM
@pytest.mark.parametrize('shape,components,medium', [((22, 26), 1, 'scalar'), ((512, 500), 1, 'scalar'),
                                                     ((150, 98), 3, 'scalar'), ((143, 30), 3, 'general'),
                                                     ((64, 40, 45), 3, 'scalar'), ((36, 44, 39), 3, 'symmetric'),
                                                     ((4, 225, 6), 3, 'general'), ((1100, 14), 1, 'scalar')])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_chunks_in_one_launch(shape, components, medium, dtype):
    from macromax_b200 import _native as nat
    _compare(shape, components, medium, dtype, nat.MMX_VARIANT_LOOP, 1, 10)
