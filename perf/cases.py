"""Performance cases: the solves a user of this package runs, from the smallest
particle to the largest dense sweep.

Every case goes through the public classes.  ``prepare`` builds what a program
keeps between calls (particle, solver with its refined tables, excitation, point
sets, H-matrices), ``run`` makes one pass, ``exact`` restates the same numbers in
64-bit torch from the face geometry alone.

Kinds:

* ``solve``: the drop-in wavelength loop ``sig, bem = bem.solve(exc.potential(p,
  enei))`` with extinction and scattering of every solution; new matrices at
  every wavelength.
* ``sweep``: ``bem.solve_spectrum(exc, eneis)``, FP64 or mixed precision.
* ``batch``: ``BatchedBEMRet.solve_spectrum`` over particles of uneven size.
* ``stat``: ``BEMStat.solve_spectrum``, quasistatic spectra.
* ``iter``: ``BEMRetIter`` with H-matrix compression and GMRES at one wavelength.
* ``hmat``: the four H-matrix products one GMRES step makes.
* ``near``: field map of a solution on a grid of points beside the particle.
"""

import math
import random

import numpy as np
import torch

from mnpbem_b200 import (BEMRet, BEMRetIter, BEMStat, ComParticle, ComPoint, CompGreenRet,
                         EpsConst, EpsDrude, PlaneWaveRet, PlaneWaveStat, Point, trirod,
                         trisphere)
from mnpbem_b200.batch import BatchedBEMRet
from mnpbem_b200.excitation import pinfty
from mnpbem_b200.hmatrix import hmat_matvec
from mnpbem_b200.shapes import random_particles

DRUDE = (10.0, 9.065, 0.0708)                 # gold, as in bench.py
EV2NM = 1.0 / 8.0655477e-4
SPHERE_FACES = {32: 60, 60: 116, 144: 284, 256: 508, 400: 796, 576: 1148, 784: 1564,
                1024: 2044, 1225: 2446, 1444: 2884}
SPHERE_DIAMETER = {32: 10.0, 60: 10.0, 1444: 40.0}     # packaged at one size only


def listed():
    return [
        # one small sphere, two wavelengths: what a quick look or a fit's inner call costs
        dict(name='solve_sphere60', kind='solve', shape='sphere', nv=32, diameter=10.0, eps=1.0,
             precision='fp64', nlam=2, npol=1),
        # the 284-face sphere of the plain spectrum, wavelength by wavelength
        dict(name='solve_sphere284', kind='solve', shape='sphere', nv=144, diameter=20.0,
             eps=1.0, precision='fp64', nlam=4, npol=1),
        # a mid-size rod (1365 flat quads and triangles, an odd count), three polarisations
        dict(name='solve_rod1365', kind='solve', shape='rod', diameter=17.3, length=61.0,
             nphi=36, ntheta=10, nz=22, eps=1.77, precision='fp64', nlam=2, npol=3),
        # the 2884-face sphere one wavelength at a time, the reference's arithmetic
        dict(name='solve_sphere2884', kind='solve', shape='sphere', nv=1444, diameter=40.0,
             eps=1.0, precision='fp64', nlam=2, npol=1),
        # the same in mixed precision
        dict(name='solve_mixed_sphere2884', kind='solve', shape='sphere', nv=1444,
             diameter=40.0, eps=1.0, precision='mixed', nlam=2, npol=1),
        # the plain 41-wavelength spectrum in one batch
        dict(name='sweep_sphere284', kind='sweep', shape='sphere', nv=144, diameter=20.0,
             eps=1.0, precision='fp64', nlam=41, npol=1, batch=41),
        # the headline sweep: 81 wavelengths of the 2884-face sphere, mixed precision
        dict(name='sweep_mixed_sphere2884', kind='sweep', shape='sphere', nv=1444,
             diameter=40.0, eps=1.0, precision='mixed', nlam=81, npol=1, batch=27),
        # six particles of uneven size in padded groups, three polarisations each
        dict(name='batch_uneven6', kind='batch', count=6, set=3, nlam=13, npol=3,
             pad_ratio=1.25),
        # quasistatic spectrum of the 1148-face sphere
        dict(name='stat_sphere1148', kind='stat', shape='sphere', nv=576, diameter=30.0,
             eps=1.0, nlam=41, npol=3, batch=41),
        # one wavelength of the 2400-face rod by H-matrix GMRES
        dict(name='iter_rod2400', kind='iter', shape='rod', diameter=20.0, length=80.0, nphi=31,
             ntheta=21, nz=41, eps=1.0, npol=1),
        # products with the four H-matrices of the 9600-face rod
        dict(name='hmat_rod9600', kind='hmat', shape='rod', diameter=20.0, length=80.0, nphi=61,
             ntheta=31, nz=101, eps=1.0, npol=1),
        # field map on a 64 x 48 grid beside the 1564-face sphere
        dict(name='near_sphere1564', kind='near', shape='sphere', nv=784, diameter=30.0, eps=1.0,
             npol=1, gx=64, gz=48),
    ]


def _rod_of(rng, lo, hi):
    """Rod grid with about lo..hi faces (log-uniform), odd counts among them."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nphi = max(6, int(round(math.sqrt(n / 1.5) * rng.uniform(0.8, 1.2))))
    rings = max(8, int(n / nphi))
    ntheta = max(3, int(rings * rng.uniform(0.2, 0.3)))
    d = round(rng.uniform(10.0, 30.0), 3)
    return dict(shape='rod', diameter=d, length=round(rng.uniform(max(30.0, d + 10.0), 120.0), 3),
                nphi=nphi + 1, ntheta=ntheta, nz=max(2, rings - 2 * (ntheta - 1) + 1))


def draw(rng):
    kind = rng.choice(['solve', 'solve', 'solve_mixed', 'sweep', 'sweep_mixed', 'batch', 'stat',
                       'iter', 'hmat', 'near'])
    eps = round(rng.uniform(1.0, 2.25), 3)
    npol = rng.choice([1, 1, 3])
    if kind == 'solve':
        return dict(kind='solve', eps=eps, precision='fp64', nlam=rng.choice([2, 3, 4]),
                    npol=npol, **_rod_of(rng, 60, 2884))
    if kind == 'solve_mixed':
        return dict(kind='solve', eps=eps, precision='mixed', nlam=2, npol=npol,
                    **_rod_of(rng, 700, 2884))
    if kind == 'sweep':
        geo = _rod_of(rng, 100, 1200)
        return dict(kind='sweep', eps=eps, precision='fp64', nlam=rng.randint(9, 41), npol=npol,
                    batch=rng.choice([16, 41]), **geo)
    if kind == 'sweep_mixed':
        geo = _rod_of(rng, 280, 2600)
        return dict(kind='sweep', eps=eps, precision='mixed', nlam=rng.randint(9, 41), npol=npol,
                    batch=rng.choice([16, 27]), **geo)
    if kind == 'batch':
        return dict(kind='batch', count=rng.randint(3, 6), set=rng.randint(4, 1000),
                    nlam=rng.randint(5, 13), npol=npol, pad_ratio=1.25)
    if kind == 'stat':
        return dict(kind='stat', eps=eps, nlam=rng.randint(9, 41), npol=npol, batch=32,
                    **_rod_of(rng, 100, 2000))
    if kind == 'iter':
        return dict(kind='iter', eps=1.0, npol=1, **_rod_of(rng, 1200, 3000))
    if kind == 'hmat':
        return dict(kind='hmat', eps=eps, npol=npol, **_rod_of(rng, 1500, 9000))
    return dict(kind='near', eps=eps, npol=npol, gx=rng.randint(9, 80), gz=rng.randint(9, 80),
                **_rod_of(rng, 200, 2600))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _particle(case):
    eps = [EpsConst(case['eps']), EpsDrude(*DRUDE)]
    if case['shape'] == 'sphere':
        p = trisphere(case['nv'], case['diameter'])
    else:
        p = trirod(case['diameter'], case['length'], (case['nphi'], case['ntheta'], case['nz']))
    return ComParticle(eps, [p], [[2, 1]], 1)


def _members(case):
    return [cp for cp, _ in random_particles(case['count'], seed=case['set'])]


def _nfaces(case):
    if case['shape'] == 'sphere':
        return SPHERE_FACES[case['nv']]
    return (case['nphi'] - 1) * (2 * (case['ntheta'] - 1) + case['nz'] - 1)


def _light(case, seed):
    """Wavelengths (jittered grid over the visible) and polarisations of one input."""
    rng = random.Random('%d/%s' % (seed, case['kind']))
    lo, hi, nlam = 400.0, 800.0, case.get('nlam', 1)
    step = (hi - lo) / nlam
    eneis = [lo + step * (i + rng.uniform(0.05, 0.95)) for i in range(nlam)]
    if case['npol'] == 1:
        a = rng.uniform(0.0, 2.0 * math.pi)
        return eneis, [[math.cos(a), math.sin(a), 0.0]], [[0.0, 0.0, 1.0]]
    return (eneis, [[1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]],
            [[0.0, 0.0, 1.0], [0.0, 0.0, 1.0], [1.0, 0.0, 0.0]])


def _grid(case):
    """Grid of points in a plane 2 nm beside the particle, in the host medium."""
    span = case['diameter']
    height = case.get('length', span)
    x = np.linspace(-span, span, case['gx'])
    z = np.linspace(-height, height, case['gz'])
    X, Z = np.meshgrid(x, z, indexing='ij')
    return np.stack([X.ravel(), np.full(X.size, 0.5 * span + 2.0), Z.ravel()], axis=1)


def _vectors(case, seed):
    """Two packed Krylov vectors (4 npol, n): smooth over the surface as the surface
    charges GMRES multiplies with are, complex128."""
    p = _particle(case)
    g = np.random.default_rng(seed)
    pos = np.asarray(p.pos) / case['length']
    out = []
    for _ in range(2):
        q = g.normal(size=(4 * case['npol'], 3)) * 6.0
        amp = g.normal(size=(4 * case['npol'], 2)) @ np.array([1.0, 1j])
        noise = g.normal(size=(4 * case['npol'], len(pos), 2)) @ np.array([1.0, 1j])
        out.append(amp[:, None] * np.exp(1j * (q @ pos.T)) + 0.1 * noise)
    return out


def prepare(case, seed):
    kind = case['kind']
    eneis, pol, dirs = _light(case, seed)
    if kind == 'batch':
        return dict(kind=kind, exc=PlaneWaveRet(pol, dirs), eneis=eneis,
                    bem=BatchedBEMRet(_members(case), refine_tol=1e-10, mem_bytes=24 << 30,
                                      tuner=None, pad_ratio=case['pad_ratio']))
    p = _particle(case)
    s = dict(kind=kind, p=p, eneis=eneis)
    if kind == 'solve':
        s.update(bem=BEMRet(p, precision=case['precision']), exc=PlaneWaveRet(pol, dirs))
    elif kind == 'sweep':
        s.update(bem=BEMRet(p, precision=case['precision']), exc=PlaneWaveRet(pol, dirs),
                 batch=case['batch'])
    elif kind == 'stat':
        s.update(bem=BEMStat(p), phip=PlaneWaveStat(pol).potential(p, eneis[0]).phip,
                 batch=case['batch'])
    elif kind == 'iter':
        s.update(bem=BEMRetIter(p, hmatrix=True, htol=1e-6, cleaf=64, tol=1e-6,
                                preconditioner='none'), exc=PlaneWaveRet(pol, dirs))
    elif kind == 'hmat':
        bem = BEMRetIter(p, hmatrix=True, htol=1e-6, cleaf=64, tol=1e-6, preconditioner='none')
        bem(eneis[0])
        bem._scratch = None                   # ACA work space: not needed by the products
        for h in (bem.G1, bem.G2, bem.H1, bem.H2):
            h.scratch = None
        v1, v2 = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in _vectors(case, seed)]
        s.update(mats=[bem.G1, bem.G2, bem.H1, bem.H2], xs=[v1, v2, v1, v2],
                 ys=[torch.empty_like(v1) for _ in range(4)], nc=v1.shape[0])
    elif kind == 'near':
        bem = BEMRet(p)
        exc = PlaneWaveRet(pol, dirs)
        s['sig'], _ = bem.solve(exc.potential(p, eneis[0]))
        s['green'] = CompGreenRet(ComPoint(p.eps, [Point(_grid(case))], [1]), p)
    return s


def _fields(sig):
    return dict(sig1=sig.sig1, sig2=sig.sig2, h1=sig.h1, h2=sig.h2)


def run(s):
    kind = s['kind']
    if kind == 'solve':
        out = []
        for enei in s['eneis']:
            sig, _ = s['bem'].solve(s['exc'].potential(s['p'], enei))
            out.append(dict(_fields(sig), ext=s['exc'].extinction(sig),
                            sca=s['exc'].scattering(sig)[0]))
        return out
    if kind == 'sweep':
        sigs = s['bem'].solve_spectrum(s['exc'], s['eneis'], batch=s['batch'])
        return {k: np.stack([getattr(g, k) for g in sigs]) for k in ('sig1', 'sig2', 'h1', 'h2')}
    if kind == 'batch':
        res = s['bem'].solve_spectrum(s['exc'], s['eneis'])
        return dict(ext=res['ext'], sca=res['sca'])
    if kind == 'stat':
        return s['bem'].solve_spectrum(s['phip'], s['eneis'], batch=s['batch'])
    if kind == 'iter':
        s['bem'].clear()                      # one pass = one new wavelength: operator and solve
        sig, _ = s['bem'].solve(s['exc'].potential(s['p'], s['eneis'][0]))
        return _fields(sig)
    if kind == 'hmat':
        return list(hmat_matvec(s['mats'], s['xs'], s['ys'], s['nc']))
    f = s['green'].field(s['sig'])
    return dict(e=f.e, h=f.h)


def work(case):
    """Bytes (inputs once, outputs once) and real operations of one pass: four LU
    factorisations (8/3 n^3 each), two right solves with n columns (8 n^3 each) and one
    inverse from its factors (16/3 n^3) per retarded wavelength."""
    kind, L, K = case['kind'], case.get('nlam', 1), case['npol']
    if kind == 'batch':
        sizes = [d['faces'] for _, d in random_particles(case['count'], seed=case['set'])]
        return dict(bytes=float(sum(104 * n + 16 * L * K for n in sizes)),
                    flops=float(sum(32.0 * n ** 3 * L for n in sizes)))
    n = _nfaces(case)
    geo = 104.0 * n
    if kind in ('solve', 'sweep'):
        return dict(bytes=geo + 128.0 * n * K * L, flops=32.0 * n ** 3 * L + 120.0 * n * n * L)
    if kind == 'stat':
        return dict(bytes=8.0 * n * n + 16.0 * n * K * (L + 1), flops=8.0 / 3.0 * n ** 3 * L)
    # about 290 stored complex64 entries per row and level of the cluster tree
    stored = 4 * 290.0 * n * math.log2(max(n, 256) / 64.0)
    if kind == 'iter':
        return dict(bytes=geo + 128.0 * n * K + 8.0 * stored * 100, flops=8.0 * stored * 4 * 100)
    if kind == 'hmat':
        return dict(bytes=8.0 * stored + 6 * 64.0 * n * K, flops=8.0 * stored * 4 * K)
    pts = case['gx'] * case['gz']
    return dict(bytes=geo + 64.0 * n * K + 120.0 * pts * K, flops=(100.0 + 110.0 * K) * pts * n)


# ---------------------------------------------------------------------------
# the same numbers in 64 bits: Green functions with the refined near and self
# elements, the BEM equations and the cross sections, from the face geometry
# ---------------------------------------------------------------------------
ORDER = 5
TINY = float(np.finfo(float).eps)


def _dev():
    return 'cuda' if torch.cuda.is_available() else 'cpu'


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


def _near_pairs(pos1, pos2, rad):
    """(rows, cols, is_self): pairs closer than three radii of the column face, in the
    expanded-square distance the refinement is defined by (mnpbem/greenfun/
    refine_utils.py:12-158); rad: per row."""
    d2 = np.sum(pos1 * pos1, axis=1)[:, None] + np.sum(pos2 * pos2, axis=1)[None, :] \
        - 2.0 * (pos1 @ pos2.T)
    d2[d2 < 1e-10] = 0.0
    d = np.sqrt(d2)
    near = ((d - rad['col'][None, :]) / rad['unit'] < 3.0) | (d == 0)
    rows, cols = np.nonzero(near)
    return rows, cols, d[rows, cols] == 0


def _points_of(q, n):
    """Quadrature points sorted by face, with offsets, from (pos, w, face)."""
    pos, w, face = q[0], q[1], q[2]
    if hasattr(w, 'tocoo'):
        w = w.tocoo()
        face = np.empty(w.shape[1], dtype=np.int64)
        face[w.col] = w.row
        val = np.empty(w.shape[1])
        val[w.col] = w.data
        w = val
    face = np.asarray(face)
    order = np.argsort(face, kind='stable')
    off = np.concatenate([[0], np.cumsum(np.bincount(face, minlength=n))])
    return np.asarray(pos)[order], np.asarray(w)[order], off


def _expand(cols, off):
    """Pair index and point index of every quadrature point of every pair's column face."""
    cnt = (off[1:] - off[:-1])[cols]
    pair = np.repeat(np.arange(len(cols)), cnt)
    start = np.concatenate([[0], np.cumsum(cnt)[:-1]])
    return pair, off[cols][pair] + np.arange(len(pair)) - start[pair]


def _near_taylor(src, centre, rows, cols, q):
    """Taylor coefficients g (P, 6), f (P, 3, 6) of near pairs: source points src[rows],
    quadrature of faces cols, expansion about the centroid distance."""
    P = len(rows)
    g = torch.zeros(P, ORDER + 1, dtype=torch.float64, device=_dev())
    f = torch.zeros(P, 3, ORDER + 1, dtype=torch.float64, device=_dev())
    qpos, qw, off = _t(q[0]), _t(q[1]), q[2]
    r0 = (_t(centre)[_t(cols)] - _t(src)[_t(rows)]).norm(dim=1)
    for s in range(0, P, 200000):
        sl = slice(s, min(P, s + 200000))
        pair, pt = [_t(a) for a in _expand(cols[sl], off)]
        v = _t(src)[_t(rows[sl])][pair] - qpos[pt]
        w = qw[pt]
        r = v.norm(dim=1).clamp_min(TINY)
        dl = r - r0[sl][pair]
        for m in range(ORDER + 1):
            g[sl, m].index_add_(0, pair, w * dl ** m / r / math.factorial(m))
            c = -dl ** m / (r ** 3 * math.factorial(m))
            if m:
                c = c + dl ** (m - 1) / (r ** 2 * math.factorial(m - 1))
            f[sl, :, m].index_add_(0, pair, v * (w * c)[:, None])
    return g, f


class _Surface(object):
    """Refined tables of a particle and its G, F matrices at any wavenumber."""

    def __init__(self, p):
        self.pos, self.nvec, self.area = _t(p.pos), _t(p.nvec), _t(p.area)
        n = self.n = len(p.pos)
        rad = np.asarray(p.bradius())
        pos = np.asarray(p.pos)
        rows, cols, own = _near_pairs(pos, pos, dict(col=rad, unit=rad[:, None]))
        self.rows, self.cols = _t(rows), _t(cols)
        g, f = _near_taylor(pos, pos, rows, cols, _points_of(p.quad(np.arange(n)), n))
        # self pairs: polar quadrature
        sel = np.nonzero(own)[0]
        ppos, pw, off = _points_of(p.quadpol(np.arange(n)), n)
        pair, pt = [_t(a) for a in _expand(cols[sel], off)]
        i = self.rows[_t(sel)]
        w = _t(pw)[pt]
        v = self.pos[i][pair] - _t(ppos)[pt]
        r = v.norm(dim=1).clamp_min(TINY)
        far = torch.zeros(len(sel), dtype=torch.float64, device=_dev()) \
            .scatter_reduce_(0, pair, r, 'amax')
        rr = torch.maximum(r, 1e-4 * far[pair])
        axes = [self.nvec, _t(p.tvec1), _t(p.tvec2)]
        dots = [(a[i][pair] * v).sum(1) for a in axes]
        add = lambda x: torch.zeros(len(sel), dtype=torch.float64,
                                    device=_dev()).index_add_(0, pair, x)
        for m in range(ORDER + 1):
            c = 1.0 / math.factorial(m)
            g[_t(sel), m] = add(w * r ** (m - 1)) * c
            parts = [add(w * (m - 1) * dots[0] * r ** (m - 3)) * c,
                     add(w * (m - 1) * dots[1] * r ** m / rr ** 3) * c,
                     add(w * (m - 1) * dots[2] * r ** m / rr ** 3) * c]
            f[_t(sel), :, m] = sum(a[i] * x[:, None] for a, x in zip(axes, parts))
        # quasistatic F and the closed-surface sums per particle
        x = self.pos[:, None, :] - self.pos[None, :, :]
        self.d = x.norm(dim=2).clamp_min(TINY)
        self.d.fill_diagonal_(TINY)
        self.ndx = (self.nvec[:, None, :] * x).sum(2)
        del x
        Fs = -self.ndx * self.area[None, :] / self.d ** 3
        stat = (self.nvec[self.rows] * f[:, :, 0]).sum(1)
        stat[_t(sel)] = -add(w * dots[0] / r ** 3)
        Fs[self.rows, self.cols] = stat
        corr = torch.zeros(n, dtype=torch.float64, device=_dev())
        lo = 0
        for q in p.p:
            hi = lo + len(q.pos)
            a = self.area[lo:hi]
            corr[lo:hi] = -2 * math.pi - (a[:, None] * Fs[lo:hi, lo:hi] / a[None, :]).sum(0)
            lo = hi
        Fs[range(n), range(n)] += corr
        self.Fstat = Fs
        f[_t(sel), :, 0] += corr[i][:, None] * self.nvec[i]
        self.g, self.fn = g, torch.einsum('pc,pcm->pm', self.nvec[self.rows], f)

    def matrices(self, k):
        k = complex(k)
        ik = torch.tensor([(1j * k) ** m for m in range(ORDER + 1)], dtype=torch.complex128,
                          device=_dev())
        G = (self.area[None, :] / self.d).to(torch.complex128)
        F = (1j * k - 1.0 / self.d) / self.d ** 2 * (self.ndx * self.area[None, :])
        G[self.rows, self.cols] = self.g.to(torch.complex128) @ ik
        F[self.rows, self.cols] = self.fn.to(torch.complex128) @ ik
        ph = torch.exp(1j * k * self.d)
        return G * ph, F * ph

    def operators(self, eps_host, enei):
        """G1, H1 inside the metal, G2, H2 in the host, and both dielectric constants."""
        w = EV2NM / enei
        e1 = DRUDE[0] - DRUDE[1] ** 2 / (w * (w + 1j * DRUDE[2]))
        e2 = complex(eps_host)
        k0 = 2 * math.pi / enei
        G1, H1 = self.matrices(k0 * np.sqrt(e1))
        G2, H2 = self.matrices(k0 * np.sqrt(e2))
        H1.diagonal().add_(2 * math.pi)
        H2.diagonal().sub_(2 * math.pi)
        return G1, G2, H1, H2, e1, e2, k0


def _solution(surf, eps_host, enei, pol, dirs):
    """sig1, h1, sig2, h2 as (n, K), (n, 3, K) of the plane waves, all entering from the
    outside (Garcia de Abajo & Howie, PRB 65, 115418, Eqs. 10-22)."""
    G1, G2, H1, H2, e1, e2, k0 = surf.operators(eps_host, enei)
    n, K = surf.n, len(pol)
    k = k0 * np.sqrt(e2)
    pol, dirs = _t(np.asarray(pol, float)), _t(np.asarray(dirs, float))
    phase = torch.exp(1j * complex(k) * (surf.pos @ dirs.T)) / (1j * k0)       # (n, K)
    a = phase[:, None, :] * pol.T[None]                                        # (n, 3, K)
    alpha = (1j * complex(k) * (surf.nvec @ dirs.T))[:, None, :] * a
    nv = surf.nvec.to(torch.complex128)
    De = -1j * k0 * e2 * torch.einsum('nc,nck->nk', nv, a)
    S1 = torch.linalg.solve(G1, H1, left=False)
    S2 = torch.linalg.solve(G2, H2, left=False)
    Di = torch.linalg.inv(S1 - S2)
    L = e1 - e2
    Sig = e1 * S1 - e2 * S2 + (k0 * L) ** 2 * Di * (surf.nvec @ surf.nvec.T)
    del S2
    mm = lambda M, x: (M @ x.reshape(n, -1)).reshape(x.shape)
    alpha = alpha - mm(S1, a)
    De = De + 1j * k0 * e1 * torch.einsum('nc,nck->nk', nv, a)
    inner = L * torch.einsum('nc,nck->nk', nv, mm(Di, alpha))
    s2 = torch.linalg.solve(Sig, De + 1j * k0 * inner)
    h2 = mm(Di, 1j * k0 * L * nv[:, :, None] * s2[:, None, :] + alpha)
    both = lambda s, h: torch.cat([s[:, None, :], h], dim=1).reshape(n, -1)
    x1 = torch.linalg.solve(G1, both(s2, h2 + a)).reshape(n, 4, K)
    x2 = torch.linalg.solve(G2, both(s2, h2)).reshape(n, 4, K)
    return x1[:, 0], x1[:, 1:], x2[:, 0], x2[:, 1:]


def _cross_sections(surf, eps_host, enei, sol, pol, dirs):
    """Extinction (optical theorem) and scattering (power over the far-field sphere)."""
    _, _, s2, h2 = sol
    k0 = 2 * math.pi / enei
    k = k0 * math.sqrt(eps_host)

    def far(u):
        ph = torch.exp(-1j * k * (u @ surf.pos.T)) * surf.area
        P = torch.einsum('dn,nck->dck', ph, h2)
        e = 1j * k0 * P - 1j * k * u[:, :, None] * (ph @ s2)[:, None, :]
        uu = u[:, :, None].to(P.dtype).expand_as(P)
        return e, 1j * k * torch.linalg.cross(uu, P, dim=1)

    e, _ = far(_t(np.asarray(dirs, float)))
    ext = [4 * math.pi / k * float((_t(np.asarray(pol[i], float)) * e[i, :, i]).sum().imag)
           for i in range(len(pol))]
    u, area = pinfty()
    e, h = far(_t(u))
    flux = 0.5 * (torch.linalg.cross(e, h.conj(), dim=1).real * _t(u)[:, :, None]).sum(1)
    sca = (_t(area) @ flux) / (0.5 * math.sqrt(eps_host))
    return np.array(ext), sca.cpu().numpy()


def _as_fields(sol, K):
    s1, h1, s2, h2 = [x.cpu().numpy() for x in sol]
    if K == 1:
        s1, h1, s2, h2 = [x[..., 0] for x in (s1, h1, s2, h2)]
    return dict(sig1=s1, sig2=s2, h1=h1, h2=h2)


def exact(case, seed):
    kind, K = case['kind'], case['npol']
    eneis, pol, dirs = _light(case, seed)
    if kind == 'iter':
        # what GMRES approaches is the solution for the compressed operator, which has
        # no closed form: it differs from the dense one by the compression's error
        return None
    if kind == 'batch':
        parts = _members(case)
        ext = np.zeros((len(parts), len(eneis), K))
        sca = np.zeros_like(ext)
        for i, p in enumerate(parts):
            surf = _Surface(p)
            for j, enei in enumerate(eneis):
                sol = _solution(surf, 1.77, enei, pol, dirs)
                ext[i, j], sca[i, j] = _cross_sections(surf, 1.77, enei, sol, pol, dirs)
        return dict(ext=ext, sca=sca)
    p = _particle(case)
    surf = _Surface(p)
    if kind in ('solve', 'sweep'):
        out = []
        for enei in eneis:
            sol = _solution(surf, case['eps'], enei, pol, dirs)
            f = _as_fields(sol, K)
            if kind == 'solve':
                ext, sca = _cross_sections(surf, case['eps'], enei, sol, pol, dirs)
                f.update(ext=float(ext[0]) if K == 1 else ext,
                         sca=float(sca[0]) if K == 1 else sca)
            out.append(f)
        return out if kind == 'solve' else {k: np.stack([f[k] for f in out]) for k in out[0]}
    if kind == 'stat':
        phip = -surf.nvec @ _t(np.asarray(pol, float)).T
        out = []
        for enei in eneis:
            w = EV2NM / enei
            e1 = DRUDE[0] - DRUDE[1] ** 2 / (w * (w + 1j * DRUDE[2]))
            M = -surf.Fstat.to(torch.complex128)
            M.diagonal().sub_(2 * math.pi * (e1 + case['eps']) / (e1 - case['eps']))
            out.append(torch.linalg.solve(M, phip.to(torch.complex128)).cpu().numpy())
        return np.stack(out)
    if kind == 'hmat':
        ops = surf.operators(case['eps'], eneis[0])[:4]
        x1, x2 = [_t(v) for v in _vectors(case, seed)]
        return [(A @ x.T).T.contiguous() for A, x in zip(ops, (x1, x2, x1, x2))]
    # near: fields of the outside charges at the points
    sol = _solution(surf, case['eps'], eneis[0], pol, dirs)
    pts = _grid(case)
    k0 = 2 * math.pi / eneis[0]
    k = k0 * math.sqrt(case['eps'])
    rad = np.asarray(p.bradius())
    rows, cols, _ = _near_pairs(pts, np.asarray(p.pos), dict(col=rad, unit=rad[None, :]))
    x = _t(pts)[:, None, :] - surf.pos[None]
    d = x.norm(dim=2)
    G = (surf.area / d).to(torch.complex128)
    Gp = ((1j * k - 1.0 / d) / d ** 2 * surf.area)[:, :, None] * x
    if len(rows):
        g, f = _near_taylor(pts, np.asarray(p.pos), rows, cols,
                            _points_of(p.quad(np.arange(surf.n)), surf.n))
        ik = torch.tensor([(1j * k) ** m for m in range(ORDER + 1)], dtype=torch.complex128,
                          device=_dev())
        G[_t(rows), _t(cols)] = g.to(torch.complex128) @ ik
        Gp[_t(rows), _t(cols)] = f.to(torch.complex128) @ ik
    ph = torch.exp(1j * k * d)
    G, Gp = G * ph, Gp * ph[:, :, None]
    _, _, s2, h2 = sol
    e = 1j * k0 * torch.einsum('pn,nck->pck', G, h2) - torch.einsum('pnc,nk->pck', Gp, s2)
    h = torch.stack([torch.einsum('pn,nk->pk', Gp[:, :, (c + 1) % 3], h2[:, (c + 2) % 3]) -
                     torch.einsum('pn,nk->pk', Gp[:, :, (c + 2) % 3], h2[:, (c + 1) % 3])
                     for c in range(3)], dim=1)
    e, h = e.cpu().numpy(), h.cpu().numpy()
    return dict(e=e[..., 0], h=h[..., 0]) if K == 1 else dict(e=e, h=h)
