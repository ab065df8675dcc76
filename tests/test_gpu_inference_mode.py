"""
Solutions made under torch.inference_mode(): tensors made there count no versions.
"""
import numpy as np
import pytest

from test_gpu_any_length import _problem
from test_gpu_fast import _solution

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,components', [((300,), 1), ((44, 60), 1), ((20, 18, 26), 3)])
def test_iterations_with_a_callback(shape, components):
    """The callback sees the state of its iteration, also after the state has been written between two iterations."""
    import torch
    from macromax_b200 import autotune
    wl = _problem(shape, components, 'scalar')
    seen = {}

    def follow(name):
        def callback(s):
            seen.setdefault(name, []).append((s.iteration, s.residue, s.previous_update_norm, s.rejections))
            if s.iteration == 3:
                autotune.tune(s._engine, iters=2, use_cache=False, candidates=(0,))  # writes the states, and restores them
                assert s.iteration == 3
                s.iteration = 10
                assert s.iteration == 10
            return s.iteration < 14
        return callback

    plain = _solution(wl)
    plain.solve(follow('plain'))
    with torch.inference_mode():
        sol = _solution(wl)
        sol.solve(follow('inference'))
        sol.solve(None, rtol=0, maxiter=5)
        assert sol.iteration == 5
        field = sol.E
    plain.solve(None, rtol=0, maxiter=5)
    assert seen['plain'] == seen['inference']
    assert [s[0] for s in seen['plain']] == [1, 2, 3, 11, 12, 13, 14]
    assert np.array_equal(plain.E, field)
