"""
The projections of a 3-component spectrum in one kernel (mmx_project_ft), where the tensor expressions for other shapes and
tracked tensors say what they give: components without an axis that are not finite, and functions that torch records.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _backend(shape, dtype):
    from macromax_b200 import Grid
    from macromax_b200.backend import BackEndB200
    be = BackEndB200(3, Grid(shape=shape, step=125e-9), dtype)
    rng = np.random.default_rng(2)
    F = be.astype((rng.standard_normal((3, 1, *shape)) + 1j * rng.standard_normal((3, 1, *shape))).astype(dtype))
    return be, F


def _expressions(be, F, transversal):
    """The same by tensor expressions."""
    f = F.clone().requires_grad_(True)
    out = be.transversal_projection_ft(f) if transversal else be.longitudinal_projection_ft(f)
    assert out.requires_grad
    return out.detach()


@pytest.mark.parametrize('shape', [(7,), (130,), (13, 40), (64, 65)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
@pytest.mark.parametrize('transversal', [False, True])
def test_components_without_an_axis_stay_apart(shape, dtype, transversal):
    be, F = _backend(shape, dtype)
    last = (-1,) * len(shape)
    F[(2, 0, *last)] = complex(np.inf, 0)
    F[(2, 0, *(n // 2 for n in shape))] = complex(np.nan, np.nan)
    out = be.transversal_projection_ft(F) if transversal else be.longitudinal_projection_ft(F)
    got, ref = out.cpu().numpy(), _expressions(be, F, transversal).cpu().numpy()
    nd = len(shape)
    assert np.all(np.isfinite(got[:nd]))
    tol = 4 * np.finfo(dtype).eps  # a few roundings per sample
    assert np.linalg.norm(got[:nd] - ref[:nd]) <= tol * np.linalg.norm(F[:nd].cpu().numpy())
    assert np.array_equal(got[nd:], ref[nd:], equal_nan=True)


@pytest.mark.parametrize('transversal', [False, True])
def test_recorded_projections(transversal):
    """torch.jit.trace, make_fx and a dispatch mode see the operations, and what they recorded serves other tensors."""
    import torch
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode
    be, F = _backend((12, 10, 9), np.complex64)
    project = be.transversal_projection_ft if transversal else be.longitudinal_projection_ft
    other = torch.flip(F, (2, 3, 4)) * 0.5j
    ref = _expressions(be, other, transversal)
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Watch():
        watched = project(other)
    assert any('mul' in str(f) for f in seen)
    for out in (watched, torch.jit.trace(project, (F,), check_trace=False)(other), make_fx(lambda x: project(x))(F)(other)):
        assert torch.equal(out, ref)
