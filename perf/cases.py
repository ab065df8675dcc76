"""
The work that programs built on this package have it do: whole solves of a fixed number of iterations through
``Solution`` and ``BatchSolution``, a mixed-precision solve, one step of a material optimisation, and the transforms
of the back end, over the grids, data types and media that its tests, workloads and benchmark use.

A case says what is solved (``kind``), the grid, the field's components, the data type and the iterations of one pass:

- ``solve``: ``Solution``, from a zero field; ``callback`` true: with a Python callback after every iteration.
- ``batch``: ``BatchSolution``, ``batch`` sources in one material.
- ``mixed``: ``MixedSolution``, ``batch`` sources, complex64 iterations refined to an FP64 residue of 1e-12.
- ``gradient``: ``adjoint.solve`` and its backward pass: field and gradient with respect to the permittivity, the set-up
  for the new permittivity included, as in every step of an optimisation.
- ``transform``: ``BackEndB200.convolve``: a vector field to k-space, projected, and back.

``exact`` restates each in plain 64-bit torch.
"""
import math

import numpy as np
import torch

WAVELENGTH = 500e-9
STEP = WAVELENGTH / 4
K0 = 2 * math.pi / WAVELENGTH


def listed():
    return [
        # a layered 1D medium: the smallest solves, as in the plane-wave tests; one launch per iteration
        dict(name='line_c128', kind='solve', n0=1000, components=1, medium='scalar', dtype='complex128', iterations=200),
        # disks in 2D in the default data type (double precision input gives a complex128 solve)
        dict(name='disks_256_c128', kind='solve', n0=256, n1=256, components=1, medium='scalar', dtype='complex128',
             iterations=100),
        # a 2D grid fitted to its structure instead of to a power of two, with a callback that follows the residue, as
        # scripts that plot or log the progress do
        dict(name='disks_ragged_callback', kind='solve', n0=300, n1=420, components=1, medium='scalar', dtype='complex64',
             iterations=50, callback=True),
        # the headline: 3D vector Maxwell in an isotropic medium
        dict(name='spheres_128_c64', kind='solve', n0=128, n1=128, n2=128, components=3, medium='scalar',
             dtype='complex64', iterations=60),
        # the same on a box that is not a cube of powers of two
        dict(name='spheres_ragged_c64', kind='solve', n0=100, n1=126, n2=90, components=3, medium='scalar',
             dtype='complex64', iterations=60),
        # and in the default data type
        dict(name='spheres_ragged_c128', kind='solve', n0=72, n1=80, n2=75, components=3, medium='scalar',
             dtype='complex128', iterations=60),
        # the largest: an anisotropic polycrystal
        dict(name='grains_192_c64', kind='solve', n0=192, n1=192, n2=192, components=3, medium='matrix',
             dtype='complex64', iterations=30),
        dict(name='grains_ragged_c64', kind='solve', n0=84, n1=75, n2=66, components=3, medium='matrix',
             dtype='complex64', iterations=30),
        # many incident waves on one scattering slab, as the columns of a scattering matrix are solved
        dict(name='slab_512x64_c64', kind='batch', n0=512, n1=512, components=1, medium='scalar', dtype='complex64',
             iterations=30, batch=64),
        # the same to double-precision residues
        dict(name='slab_mixed_200x8', kind='mixed', n0=200, n1=180, components=1, medium='scalar', dtype='complex128',
             batch=8),
        # one step of an inverse design: forward and adjoint solves of a few sources
        dict(name='design_64x4', kind='gradient', n0=64, n1=64, n2=64, components=1, medium='scalar', dtype='complex64',
             iterations=120, batch=4),
        # the back end's own transforms, which set-up and post-processing of the reference package call
        dict(name='transform_ragged_c128', kind='transform', n0=150, n1=128, n2=110, components=3, dtype='complex128'),
    ]


def _axis(rng, lo, hi):
    """An axis length between lo and hi, spread over the logarithm: one that the transforms take (no prime above 13)."""
    n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    while True:
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return min(n, hi)
        n += 1


def draw(rng):
    kind = rng.choice(['solve'] * 6 + ['batch', 'mixed', 'gradient', 'transform'])
    if kind == 'solve':
        dims = rng.choice([1, 2, 2, 3, 3, 3])
        dtype = rng.choice(['complex64', 'complex128'])
        if dims == 1:
            components = rng.choice([1, 3])
            return dict(kind=kind, n0=_axis(rng, 200, 800 if components == 3 else 2400), components=components,
                        medium='scalar', dtype=dtype, iterations=200)
        if dims == 2:
            return dict(kind=kind, n0=_axis(rng, 48, 768), n1=_axis(rng, 48, 768), components=rng.choice([1, 1, 3]),
                        medium='scalar', dtype=dtype, iterations=rng.randint(50, 100), callback=rng.random() < 0.3)
        medium = rng.choice(['scalar', 'scalar', 'matrix'])
        top = 160 if dtype == 'complex64' else 120
        return dict(kind=kind, n0=_axis(rng, 32, top), n1=_axis(rng, 32, top), n2=_axis(rng, 32, top),
                    components=3 if medium == 'matrix' else rng.choice([1, 3]), medium=medium, dtype=dtype,
                    iterations=rng.randint(20, 40))
    if kind == 'batch':
        return dict(kind=kind, n0=_axis(rng, 96, 512), n1=_axis(rng, 96, 512), components=1, medium='scalar',
                    dtype='complex64', iterations=rng.randint(20, 40), batch=rng.randint(2, 64))
    if kind == 'mixed':
        return dict(kind=kind, n0=_axis(rng, 96, 256), n1=_axis(rng, 96, 256), components=1, medium='scalar',
                    dtype='complex128', batch=rng.randint(1, 16))
    if kind == 'gradient':
        return dict(kind=kind, n0=_axis(rng, 32, 96), n1=_axis(rng, 32, 96), n2=_axis(rng, 32, 96), components=1,
                    medium='scalar', dtype='complex64', iterations=rng.randint(60, 120), batch=rng.randint(1, 4))
    return dict(kind=kind, n0=_axis(rng, 48, 160), n1=_axis(rng, 48, 160), n2=_axis(rng, 48, 160), components=3,
                dtype=rng.choice(['complex64', 'complex128']))


def _shape(case):
    return tuple(case[a] for a in ('n0', 'n1', 'n2') if a in case)


def _ramp(shape, px):
    """Absorbing extinction: 0 .. 0.5 over the outer px samples of every axis, the largest of the axes' ramps."""
    res = np.zeros(shape)
    for a, n in enumerate(shape):
        i = np.arange(n)
        depth = np.clip(np.maximum((px - i) / px, (i - (n - 1 - px)) / px), 0, 1)
        res = np.maximum(res, 0.5 * depth.reshape([n if b == a else 1 for b in range(len(shape))]))
    return res


def _inputs(case, seed):
    """Permittivity [*shape] or [3, 3, *shape], sources [batch, components, *shape] (complex128) and the thickness of
    the absorbing layer."""
    rng = np.random.default_rng(seed)
    shape, c, batch = _shape(case), case['components'], case.get('batch', 1)
    nd = len(shape)
    px = max(4, min(shape) // 10)
    if case['medium'] == 'matrix':
        # grains of a uniaxial crystal, each turned at random
        grains = 64
        tensors = np.empty((grains, 3, 3), dtype=np.complex128)
        for g in range(grains):
            q, r = np.linalg.qr(rng.standard_normal((3, 3)))
            q = q * np.sign(np.diag(r))
            tensors[g] = (q * np.array([1.50 + 1e-3j, 1.50 + 1e-3j, 1.65 + 1e-3j]) ** 2) @ q.T
        centres = torch.as_tensor(rng.uniform(0, 1, (grains, 3)) * np.array(shape), device='cuda')
        axes = [torch.arange(n, device='cuda', dtype=torch.float64) for n in shape]
        best = label = None
        for g in range(grains):
            d = [(x - centres[g, a]) ** 2 for a, x in enumerate(axes)]
            d = d[0][:, None, None] + d[1][:, None] + d[2]
            if best is None:
                best, label = d, torch.zeros(shape, dtype=torch.int64, device='cuda')
            else:
                label[d < best] = g
                best = torch.minimum(best, d)
        eps = torch.empty((3, 3, *shape), dtype=torch.complex128, device='cuda')
        ten = torch.as_tensor(tensors, device='cuda')
        ramp = torch.as_tensor(_ramp(shape, px), device='cuda')
        for i in range(3):
            for j in range(3):
                eps[i, j] = ten[:, i, j][label]
            eps[i, i] += 1j * ramp
        eps = eps.cpu().numpy()
    else:
        eps = np.ones(shape, dtype=np.complex128)
        open_grid = np.ogrid[tuple(slice(n) for n in shape)]
        side = min(shape) / 128
        for _ in range({1: 12, 2: 30, 3: 120}[nd]):
            centre = rng.uniform(0, 1, nd) * shape
            radius = rng.uniform(3, 10) * max(side, 0.5)
            index = rng.uniform(1.3, 1.6)
            box = tuple(slice(max(0, int(x - radius)), min(n, int(x + radius) + 2)) for x, n in zip(centre, shape))
            d2 = sum((g[tuple(b if a == k else slice(None) for k, b in enumerate(box))] - centre[a]) ** 2
                     for a, g in enumerate(open_grid))
            eps[box][d2 <= radius ** 2] = index ** 2 + 0.005j
        if case['kind'] == 'gradient':
            mid = tuple(slice(n // 4, n // 4 + n // 2) for n in shape)
            eps[mid] = rng.uniform(1.0, 2.0, eps[mid].shape)
        eps = eps + 1j * _ramp(shape, px)
    # a beam from a sheet near the first boundary: a Gaussian profile with a tilt of its own for each source
    src = np.zeros((batch, c, *shape), dtype=np.complex128)
    at = min(px + 4, shape[-1] - 1)
    for b in range(batch):
        sheet = np.exp(1j * rng.uniform(0, 2 * np.pi))
        for a, n in enumerate(shape[:-1]):
            x = np.arange(n)
            wave = np.exp(-((x - n / 2) / (0.3 * n)) ** 2 + 1j * K0 * STEP * math.sin(rng.uniform(-1, 1)) * x)
            sheet = sheet * wave.reshape([n if k == a else 1 for k in range(nd - 1)])
        src[b, 0, ..., at] = sheet
    return eps, src, px * STEP


class _State:
    pass


def prepare(case, seed):
    from macromax_b200 import Bound, Grid, Solution
    s = _State()
    s.case = case
    dtype = np.dtype(case['dtype'])
    grid = Grid(shape=_shape(case), step=STEP)
    if case['kind'] == 'transform':
        from macromax_b200.backend import BackEndB200
        s.backend = BackEndB200(3, grid, dtype)
        s.field = s.backend.astype(_field(case, seed))
        return s
    eps, src, thickness = _inputs(case, seed)
    bound = Bound(grid, thickness=thickness)
    if case['kind'] == 'solve':
        s.solution = Solution(grid, vectorial=case['components'] == 3, vacuum_wavelength=WAVELENGTH, epsilon=eps,
                              source_distribution=src[0], bound=bound, dtype=dtype)
    elif case['kind'] == 'batch':
        from macromax_b200.batch import BatchSolution
        s.solution = BatchSolution(grid, src, eps, bound=bound, vacuum_wavelength=WAVELENGTH, dtype=dtype)
    elif case['kind'] == 'mixed':
        from macromax_b200.mixed import MixedSolution
        s.solution = MixedSolution(grid, src, eps, bound=bound, vacuum_wavelength=WAVELENGTH)
    else:
        s.grid, s.bound = grid, bound
        s.epsilon = torch.from_numpy(eps).cuda()
        s.sources = torch.from_numpy(src).to('cuda', torch.complex64)
        s.weight = torch.from_numpy(_detector(case)).cuda()
    return s


def _field(case, seed):
    rng = np.random.default_rng(seed)
    shape = (3, 1, *_shape(case))
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(case['dtype'])


def _detector(case):
    """Real weights of the design's loss: a patch behind the scatterer."""
    shape = _shape(case)
    w = np.zeros(shape, dtype=np.float32)
    w[tuple(slice(n // 2 - n // 8, n // 2 + n // 8) for n in shape[:-1]) + (shape[-1] - shape[-1] // 6,)] = 1.0
    return w


def run(state):
    case = state.case
    if case['kind'] == 'solve':
        sol = state.solution
        sol.E = 0.0
        if case.get('callback'):
            sol.solve(lambda s: s.iteration < case['iterations'] and s.residue > 1e-9)
            return sol.E
        sol.solve(None, rtol=0, maxiter=case['iterations'])
        return sol.E_device
    if case['kind'] == 'batch':
        state.solution.set_fields(0.0)
        state.solution.solve(rtol=0, maxiter=case['iterations'])
        return state.solution.E_device
    if case['kind'] == 'mixed':
        state.solution.x.zero_()
        state.solution.solve(rtol=1e-12)
        return state.solution.x
    if case['kind'] == 'gradient':
        from macromax_b200 import adjoint
        eps = state.epsilon.detach().clone().requires_grad_(True)
        E = adjoint.solve(eps, state.sources, state.grid, K0, bound=state.bound, rtol=0, maxiter=case['iterations'])
        scale = 1 / E.detach().abs().max()
        loss = (state.weight * (E * scale).abs() ** 2).sum()
        loss.backward()
        return {'field': E.detach() * K0 ** 2, 'gradient': eps.grad}
    return state.backend.convolve(state.backend.transversal_projection_ft, state.field)


def work(case):
    """A solve reads the field, the source and the material and writes the field once in every iteration; two transforms
    per component and iteration, and the products with the material."""
    shape, c = _shape(case), case['components']
    n, word = math.prod(shape), np.dtype(case['dtype']).itemsize
    batch = case.get('batch', 1)
    fft = 5 * n * math.log2(n)
    if case['kind'] == 'transform':
        return dict(bytes=2 * c * n * word, flops=2 * c * fft)
    if case['kind'] == 'mixed':  # the iterations depend on the medium: the sources and the material in, the field out
        return dict(bytes=(2 * batch + 1) * n * word, flops=2 * batch * fft)
    m = 6 if case['medium'] == 'matrix' else 1
    solves = 2 if case['kind'] == 'gradient' else 1
    k = case['iterations'] * solves
    return dict(bytes=k * word * n * (3 * c * batch + m), flops=k * batch * (2 * c * fft + n * (16 * c * c if m > 1 else 16 * c)))


# ----------------------------------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch.
# ----------------------------------------------------------------------------------------------------------------------
def _minimise(f):
    """Nelder-Mead along a line from the simplex {0, 1} (reflection 1, expansion 2, contraction 1/2, shrink 1/2), until
    the simplex and its values are within 0.01."""
    sim, val = [0.0, 1.0], [f(0.0), f(1.0)]
    calls, steps = 2, 1

    def order():
        if val[1] < val[0]:
            sim.reverse()
            val.reverse()

    order()
    while calls < 100 and steps < 100:
        if abs(sim[1] - sim[0]) <= 0.01 and abs(val[1] - val[0]) <= 0.01:
            break
        best, worst = sim
        r = 2 * best - worst
        fr = f(r)
        calls += 1
        if fr < val[0]:
            e = 3 * best - 2 * worst
            fe = f(e)
            calls += 1
            sim[1], val[1] = (e, fe) if fe < fr else (r, fr)
        else:  # in one dimension a reflected point is never between the best and the second worst
            c = 1.5 * best - 0.5 * worst if fr < val[1] else 0.5 * best + 0.5 * worst
            fc = f(c)
            calls += 1
            if (fc <= fr) if fr < val[1] else (fc < val[1]):
                sim[1], val[1] = c, fc
            else:
                sim[1] = best + 0.5 * (worst - best)
                val[1] = f(sim[1])
                calls += 1
        steps += 1
        order()
    return sim[0], val[0]


def _largest_singular(ab, eps):
    """The largest singular value of ab - eps over the grid; 3x3: from the characteristic cubic of its square."""
    if eps.dim() < 5:
        return float((ab - eps).abs().max())
    d = -eps.reshape(3, 3, -1)
    d[range(3), range(3)] += ab
    h = torch.einsum('kin,kjn->ijn', d.conj(), d)
    q = (h[0, 0] + h[1, 1] + h[2, 2]).real / 3
    a = [h[i, i].real - q for i in range(3)]
    off = h[0, 1].abs() ** 2 + h[0, 2].abs() ** 2 + h[1, 2].abs() ** 2
    p = ((a[0] ** 2 + a[1] ** 2 + a[2] ** 2 + 2 * off) / 6).sqrt()
    det = (a[0] * a[1] * a[2] + 2 * (h[0, 1] * h[1, 2] * h[0, 2].conj()).real - a[0] * h[1, 2].abs() ** 2
           - a[1] * h[0, 2].abs() ** 2 - a[2] * h[0, 1].abs() ** 2)
    r = torch.where(p > 0, det / (2 * p ** 3), torch.zeros_like(p)).clamp(-1, 1)
    return float((q + 2 * p * torch.cos(torch.acos(r) / 3)).max()) ** 0.5


class _Iteration:
    def __init__(self, eps, thickness, shape):
        self.eps, self.shape, self.nd = eps, shape, len(shape)
        real, imag = _minimise(lambda ab: _largest_singular(ab, eps))
        kappa = math.log(1e-3) / (-K0 * thickness)
        self.alpha = complex(real, max(imag + 0.05, 2 * max(0.0, real + kappa ** 2) ** 0.5 * kappa))
        self.k = [(2 * math.pi * torch.fft.fftfreq(n, STEP * K0, dtype=torch.float64, device=eps.device)).reshape(
            [n if b == a else 1 for b in range(self.nd)]) for a, n in enumerate(shape)]
        self.k2 = sum(k ** 2 for k in self.k).expand(shape)
        self.over = torch.where(self.k2 == 0, torch.zeros_like(self.k2), 1 / self.k2)

    def chi(self, alpha, x):
        """i (eps - alpha) / alpha_i applied to x [components, *shape]."""
        y = torch.einsum('ij...,j...->i...', self.eps, x) if self.eps.dim() == 5 else self.eps * x
        return (1j / alpha.imag) * (y - alpha * x)

    def green(self, alpha, x):
        axes = tuple(range(1, 1 + self.nd))
        F = torch.fft.fftn(x, dim=axes)
        g = -1j * alpha.imag / (self.k2 - alpha)
        if F.shape[0] == 1:
            return torch.fft.ifftn(g * F, dim=axes)
        proj = sum(self.k[a] * F[a] for a in range(self.nd)) * self.over
        for a in range(3):
            along = self.k[a] * proj if a < self.nd else torch.zeros_like(proj)
            if a < self.nd:
                along[(0,) * self.nd] = F[a][(0,) * self.nd]
            F[a] = g * (F[a] - along) + (1j * alpha.imag / alpha) * along
        return torch.fft.ifftn(F, dim=axes)

    def solve(self, source, iterations, residue=0.0):
        """The field (times k0^2) for a source, from zero."""
        alpha, E, before = self.alpha, torch.zeros_like(source), math.inf
        for _ in range(iterations):
            d = self.chi(alpha, self.green(alpha, self.chi(alpha, E) + (1j / alpha.imag) * source) - E)
            now = float(torch.linalg.vector_norm(d))
            if now / before < 1:
                E = E + d
                before = now
            else:
                alpha = complex(alpha.real, 1.5 * alpha.imag)
            if residue and before < residue * float(torch.linalg.vector_norm(E)):
                break
        return E


def exact(case, seed):
    if case['kind'] == 'transform':
        F = torch.fft.fftn(torch.from_numpy(_field(case, seed)).cuda().to(torch.complex128), dim=(2, 3, 4))
        k = [(2 * math.pi * torch.fft.fftfreq(n, STEP, dtype=torch.float64, device='cuda')).reshape(
            [n if b == a else 1 for b in range(3)]) for a, n in enumerate(_shape(case))]
        k2 = sum(x ** 2 for x in k)
        k2[0, 0, 0] = 1.0
        proj = sum(k[a] * F[a, 0] for a in range(3)) / k2
        for a in range(3):
            F[a, 0] -= k[a] * proj
            F[a, 0, 0, 0, 0] = 0.0
        return torch.fft.ifftn(F, dim=(2, 3, 4))
    eps, src, thickness = _inputs(case, seed)
    shape = _shape(case)
    it = _Iteration(torch.from_numpy(eps).cuda(), thickness, shape)
    sources = [torch.from_numpy(x).cuda() for x in src]
    flat = (len(sources), case['components'], math.prod(shape))
    if case['kind'] == 'solve':
        E = it.solve(sources[0], case['iterations'])
        return E.cpu().numpy() / K0 ** 2 if case.get('callback') else E
    if case['kind'] == 'batch':
        return torch.stack([it.solve(x, case['iterations']) for x in sources]).reshape(flat)
    if case['kind'] == 'mixed':
        return torch.stack([it.solve(x, 20000, 1e-14) for x in sources]).reshape(flat)
    fields = torch.stack([it.solve(x, case['iterations']) for x in sources])
    weight = torch.from_numpy(_detector(case)).cuda()
    physical = fields / K0 ** 2
    scale = 1 / physical.abs().max()
    nus = torch.stack([it.solve((2 * scale ** 2 * weight * x).conj(), case['iterations']) for x in physical])
    return {'field': fields, 'gradient': ((nus * fields).sum(dim=(0, 1)) / K0 ** 2).conj().resolve_conj()}
