"""
What the passes of the default variant do at the ends of their range, against the runtime-radix passes: an alpha that the
divergence guard has raised beyond the range of the data type.
"""
import numpy as np
import pytest

from test_gpu_any_length import _problem
from test_gpu_fast import _solution

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
