"""
The passes for axes of any length (complex64 lengths without a specialised kernel, and complex128), launched one by one
and as chunks of iterations in one launch, against the runtime-radix kernels and the numpy oracle: every radix up to 16,
two to four stages, ragged last tiles, scalar and vector fields, isotropic, symmetric and general 3x3 permittivities,
batches, rejected updates; and the transforms against numpy.
"""
import numpy as np
import pytest

from test_gpu_fast import _solution, rel

pytestmark = pytest.mark.gpu


def _problem(shape, components, medium, seed=3):
    rng = np.random.default_rng(seed)
    eps = 1.0 + 0.8 * rng.uniform(size=shape) + 0.05j
    if medium != 'scalar':
        full = np.zeros((3, 3, *shape), dtype=np.complex128)
        for i in range(3):
            full[i, i] = eps + 0.1 * i
            for j in range(i):
                full[i, j] = full[j, i] = 0.1 * rng.uniform(-1, 1, shape)
        if medium == 'general':
            full[0, 1] += 0.02j
        eps = full
    src = np.zeros((components, *shape), dtype=np.complex128)
    src[(0, *(n // 3 for n in shape))] = 1.0
    src[(components - 1, *(n // 2 for n in shape))] += 0.5j
    return dict(shape=shape, step=125e-9, wavelength=500e-9, epsilon=eps, source=src, bound_thickness=500e-9)


# 4 x 6 ... 4096: each radix 2..16 as first, middle or last of some axis; row and pencil counts that leave a partial tile
CASES = [((22, 26), 1, 'scalar'), ((300, 420), 1, 'scalar'), ((9, 1500), 1, 'scalar'), ((1100, 14), 1, 'scalar'),
         ((150, 98), 3, 'scalar'), ((143, 30), 3, 'general'), ((45, 33, 35), 1, 'scalar'), ((63, 50, 27), 3, 'scalar'),
         ((36, 44, 39), 3, 'symmetric'), ((25, 32, 21), 3, 'general'), ((4, 225, 6), 3, 'symmetric'),
         ((128, 40, 90), 3, 'scalar')]


@pytest.mark.parametrize('shape,components,medium', CASES)
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
@pytest.mark.parametrize('launches', ['passes', 'loop'])
def test_iteration_matches_generic_and_oracle(shape, components, medium, dtype, launches):
    from macromax_b200 import _native as nat, autotune
    from oracle import mmoracle as mo
    wl = _problem(shape, components, medium)
    fast, gen = _solution(wl, dtype), _solution(wl, dtype, generic=True)
    autotune.set_variant(fast._engine, nat.MMX_VARIANT_PASSES if launches == 'passes' else nat.MMX_VARIANT_LOOP)
    ref = mo.from_workload(wl, np.complex128)
    assert abs(fast.alpha - ref.alpha) <= 1e-9 * abs(ref.alpha)
    for s in (fast, gen):
        s.solve(None, rtol=0, maxiter=10)
    ref.solve(rtol=0, maxiter=10)
    assert fast.iteration == gen.iteration == 10
    # ten iterations of a contraction: a few roundings each
    tol = 1e-5 if dtype == np.complex64 else 1e-12
    assert rel(fast.E, gen.E) < tol
    assert rel(fast.E, ref.E) < max(tol, 1e-9 if medium != 'scalar' else 0)  # a 3x3 alpha: closed-form eigenvalues
    assert fast.residue == pytest.approx(gen.residue, rel=10 * tol)


# enough tiles for the kernels compiled for their length on every axis: the smallest and the largest, odd ones, radix 16
@pytest.mark.parametrize('shape,components,medium', [((35, 72, 80), 3, 'scalar'), ((143, 66, 75), 1, 'scalar'),
                                                     ((32, 182, 77), 3, 'symmetric'), ((192, 70, 72), 1, 'scalar'),
                                                     ((60, 110, 169), 3, 'scalar'), ((112, 108, 45), 3, 'symmetric'),
                                                     ((64, 96, 90), 3, 'general')])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_lengths_with_own_kernels_match_generic(shape, components, medium, dtype):
    wl = _problem(shape, components, medium)
    fast, gen = _solution(wl, dtype), _solution(wl, dtype, generic=True)
    for s in (fast, gen):
        s.solve(None, rtol=0, maxiter=6)
    tol = 1e-5 if dtype == np.complex64 else 1e-12
    assert rel(fast.E, gen.E) < tol
    assert fast.residue == pytest.approx(gen.residue, rel=10 * tol)


@pytest.mark.parametrize('shape,components', [((1000,), 1), ((77,), 3), ((4,), 1), ((2160,), 1), ((825,), 3)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_line_matches_generic_and_oracle(shape, components, dtype):
    from oracle import mmoracle as mo
    wl = _problem(shape, components, 'scalar')
    wl['bound_thickness'] = 0.0 if shape[0] < 8 else wl['bound_thickness']
    fast, gen = _solution(wl, dtype), _solution(wl, dtype, generic=True)
    ref = mo.from_workload(wl, np.complex128)
    for s in (fast, gen):
        s.solve(None, rtol=0, maxiter=20)
    ref.solve(rtol=0, maxiter=20)
    assert fast.iteration == gen.iteration == 20
    tol = 1e-5 if dtype == np.complex64 else 1e-12
    assert rel(fast.E, gen.E) < tol
    assert rel(fast.E, ref.E) < tol


@pytest.mark.parametrize('shape,components', [((300,), 1), ((44, 60), 1), ((18, 20, 22), 1), ((40, 36), 3)])
@pytest.mark.parametrize('launches', ['passes', 'loop'])
def test_rejected_updates_match_generic(shape, components, launches):
    """A medium with gain: the divergence guard rejects updates; alpha, the rejections and the field are the same."""
    from macromax_b200 import _native as nat, autotune
    wl = _problem(shape, components, 'scalar')
    rng = np.random.default_rng(9)
    wl['epsilon'] = wl['epsilon'] - 0.45j * rng.uniform(size=shape)
    wl['bound_thickness'] = 0.0
    fast, gen = _solution(wl, np.complex128), _solution(wl, np.complex128, generic=True)
    autotune.set_variant(fast._engine, nat.MMX_VARIANT_PASSES if launches == 'passes' else nat.MMX_VARIANT_LOOP)
    for s in (fast, gen):
        s.solve(None, rtol=0, maxiter=25)
    assert gen.rejections > 0
    assert (fast.rejections, fast.iteration) == (gen.rejections, gen.iteration)
    assert fast.alpha == pytest.approx(gen.alpha, rel=1e-14)
    assert rel(fast.E, gen.E) < 1e-9  # updates of a nearly diverging iteration


@pytest.mark.parametrize('shape,components,batch', [((60, 77), 1, 5), ((20, 18, 26), 3, 3), ((96, 10), 1, 40)])
def test_batch_members_match_single_solves(shape, components, batch):
    from macromax_b200 import Bound, Grid
    from macromax_b200.batch import BatchSolution
    wl = _problem(shape, components, 'scalar')
    rng = np.random.default_rng(5)
    src = wl['source'] * np.exp(2j * np.pi * rng.uniform(size=(batch,) + (1,) * (len(shape) + 1)))
    src[1::2] = np.roll(src[1::2], 3, axis=2)
    grid = Grid(shape=shape, step=wl['step'])
    bs = BatchSolution(grid, src, wl['epsilon'], bound=Bound(grid, thickness=wl['bound_thickness']),
                       vacuum_wavelength=wl['wavelength'])
    bs.solve(rtol=1e-3, maxiter=200)
    for b in (0, 1, batch - 1):
        one = _solution({**wl, 'source': src[b]})
        one.solve(None, rtol=1e-3, maxiter=200)
        assert one.iteration == bs.iterations[b]
        assert rel(bs.E[b], one.E) < 1e-5
    bs.close()


@pytest.mark.parametrize('shape', [(22, 26), (1500, 9), (4, 1100), (150, 128, 110), (39, 35, 143), (2048, 6), (13, 13),
                                   (60, 77, 96), (192, 100, 33)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_fftn_matches_numpy(shape, dtype):
    import torch
    from macromax_b200 import _native as nat
    rng = np.random.default_rng(1)
    x = (rng.standard_normal((2, *shape)) + 1j * rng.standard_normal((2, *shape))).astype(dtype)
    axes = tuple(range(1, 1 + len(shape)))
    ref = np.fft.fftn(x.astype(np.complex128), axes=axes)
    plan = nat.Plan(shape, 1, 1, nat.MMX_C64 if dtype == np.complex64 else nat.MMX_C128)
    xt = torch.from_numpy(x).cuda()
    yt = torch.empty_like(xt)
    stream = nat.ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or 0)
    tol = 2e-6 if dtype == np.complex64 else 1e-14
    nat.call('mmx_fftn', plan.handle, nat.device_ptr(xt), nat.device_ptr(yt), 2, 0, stream)
    assert np.linalg.norm(yt.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
    nat.call('mmx_fftn', plan.handle, nat.device_ptr(yt), nat.device_ptr(yt), 2, 1, stream)  # in place, inverse
    assert np.linalg.norm(yt.cpu().numpy() - x) <= tol * np.linalg.norm(x)
    plan.close()


@pytest.mark.parametrize('shape', [(7,), (300,), (13, 40), (64, 65), (5, 10, 20), (33, 4, 130)])
@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_projections_match_tensor_expressions(shape, dtype):
    import torch
    from macromax_b200 import Grid
    from macromax_b200.backend import BackEndB200
    be = BackEndB200(3, Grid(shape=shape, step=125e-9), dtype)
    rng = np.random.default_rng(2)
    F = be.astype((rng.standard_normal((3, 1, *shape)) + 1j * rng.standard_normal((3, 1, *shape))).astype(dtype))
    k = [np.asarray(x, dtype=np.float64) for x in be._grid.k]
    k2 = sum(x ** 2 for x in k) + np.zeros(shape)
    f = F.cpu().numpy().astype(np.complex128)[:, 0]
    k2.flat[0] = 1.0
    proj = sum(k[a] * f[a] for a in range(len(shape))) / k2
    ref = np.zeros_like(f)
    for a in range(len(shape)):
        ref[a] = k[a] * proj
        ref[a].flat[0] = f[a].flat[0]
    tol = 4 * np.finfo(dtype).eps  # a few roundings per sample
    conj = torch.conj(F)  # a lazily conjugated tensor
    assert np.linalg.norm(be.longitudinal_projection_ft(F).cpu().numpy()[:, 0] - ref) <= tol * np.linalg.norm(f)
    assert np.linalg.norm(be.transversal_projection_ft(F).cpu().numpy()[:, 0] - (f - ref)) <= tol * np.linalg.norm(f)
    assert np.linalg.norm(be.transversal_projection_ft(conj).cpu().numpy()[:, 0] - np.conj(f - ref)) <= tol * np.linalg.norm(f)


def test_chunks_in_one_launch_on_two_streams():
    """Two solves whose chunks are one launch each, queued on two streams without waiting: the fields of the solves alone."""
    import torch
    from macromax_b200 import Bound, Grid, _native as nat
    from macromax_b200.batch import BatchSolution

    def make(shape, dtype):
        wl = _problem(shape, 1, 'scalar')
        grid = Grid(shape=shape, step=wl['step'])
        return BatchSolution(grid, wl['source'][None], wl['epsilon'], bound=Bound(grid, thickness=wl['bound_thickness']),
                             vacuum_wavelength=wl['wavelength'], dtype=dtype)

    cases = [((300, 420), np.complex64), ((256, 256), np.complex128)]
    alone = [make(*c) for c in cases]
    both = [make(*c) for c in cases]
    for s in alone:
        assert nat.load().mmx_plan_chunk_ends(s.engine.plan.handle, s.engine.chi_kind) == 1
        for _ in range(4):
            s.engine.iterate(30)
            torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in both]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, stream in zip(both, streams):
            s.engine.iterate(30, stream=stream)
    torch.cuda.synchronize()
    for s, ref in zip(both, alone):
        nat.check_stalled(s.state)
        assert np.array_equal(s.iterations, ref.iterations)
        assert np.array_equal(s.E, ref.E)
