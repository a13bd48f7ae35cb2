"""Fields and potentials at points over the numbers of columns: one kernel instance
each for 1, 2, 3 and 4 columns, chunks of four beyond; columns of the points' own
(``diag``); media with and without loss; refined pairs, none, and all of them; and
more faces than the bits of the refined pairs have room for.  Against the sums
over the entries in FP64 torch."""
import numpy as np
import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _inputs(npt, n, B, K, pairs, seed):
    g = np.random.default_rng(seed)
    d = dict(pt=g.normal(size=(npt, 3)) * 3.0, pos=g.normal(size=(n, 3)),
             area=g.uniform(0.5, 1.5, n) / n, face_med=np.tile([2, 1], (n, 1)).astype(np.int32),
             pt_med=(1 + np.arange(npt) % 2).astype(np.int32),
             k=g.uniform(0.5, 2.0, (B, 2)) + 1j * np.array([0.0, 0.3]),   # medium 2 absorbs
             k0=g.uniform(0.5, 1.0, B),
             sol=g.normal(size=(B, 8, K, n)) + 1j * g.normal(size=(B, 8, K, n)))
    d['face_med'][::7] = [1, 2]
    d['face_med'][3::11] = [1, 1]                       # both sides in the host
    d['pt_med'][npt // 2] = 0                           # a point in no medium: zeros
    cols = {'none': [np.zeros(0, int)] * npt, 'all': [np.arange(n)] * npt}.get(pairs)
    if cols is None:
        cols = [np.sort(g.choice(n, size=min(n, 1 + 5 * i), replace=False)) for i in range(npt)]
        cols[0] = np.unique([0, n - 1])                 # a pair is listed once
    d['rptr'] = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    d['cols'] = np.concatenate(cols + [np.zeros(1, int)]).astype(np.int32)
    d['g'] = g.normal(size=(len(d['cols']), 6)) / n
    d['f'] = g.normal(size=(len(d['cols']), 3, 6)) / n
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in d.items()}


def _expected(t, mode, diag):
    """(outputs, sums of the terms' magnitudes), each a pair."""
    npt, n = len(t['pt']), len(t['pos'])
    B, _, K, _ = t['sol'].shape
    KC = diag or K
    kw = dict(dtype=torch.complex128, device='cuda')
    o1 = torch.zeros((B, npt, 3, KC) if mode == 0 else (B, npt, KC), **kw)
    o2 = torch.zeros((B, npt, 3, KC), **kw)
    s1, s2 = torch.zeros_like(o1), torch.zeros_like(o2)
    for b in range(B):
        for i in range(npt):
            med = int(t['pt_med'][i])
            if med == 0:
                continue
            k = t['k'][b, med - 1]
            x = t['pt'][i] - t['pos']
            d = x.norm(dim=1)
            G = (t['area'] / d).to(torch.complex128)
            Gp = ((1j * k - 1 / d) / d ** 2 * t['area'])[:, None] * x
            lo, hi = int(t['rptr'][i]), int(t['rptr'][i + 1])
            c = t['cols'][lo:hi].long()
            ik = torch.stack([(1j * k) ** m for m in range(6)])
            G[c] = t['g'][lo:hi].to(torch.complex128) @ ik
            Gp[c] = t['f'][lo:hi].to(torch.complex128) @ ik
            ph = torch.exp(1j * k * d)
            G, Gp = G * ph, Gp * ph[:, None]
            cs = slice(i * diag, (i + 1) * diag) if diag else slice(0, K)
            for s in range(2):
                on = (t['face_med'][:, s] == med).to(torch.complex128)
                sg = t['sol'][b, 4 * s, cs] * on                        # (KC, n)
                h = t['sol'][b, 4 * s + 1:4 * s + 4, cs] * on           # (3, KC, n)
                for f, a1, a2 in ((lambda v: v, o1, o2), (torch.abs, s1, s2)):
                    g_, gp, sg_, h_ = f(G) + 0j, f(Gp) + 0j, f(sg) + 0j, f(h) + 0j
                    sign = -1.0 if a1 is o1 else 1.0
                    if mode == 1:
                        a1[b, i] += sg_ @ g_
                        a2[b, i] += torch.einsum('ckn,n->ck', h_, g_)
                        continue
                    ikh = (1j if a1 is o1 else 1.0) * t['k0'][b]
                    a1[b, i] += ikh * torch.einsum('ckn,n->ck', h_, g_) \
                        + sign * torch.einsum('kn,nc->ck', sg_, gp)
                    for e in range(3):
                        p, q = (e + 1) % 3, (e + 2) % 3
                        a2[b, i, e] += h_[q] @ gp[:, p] + sign * (h_[p] @ gp[:, q])
    return (o1, o2), (s1, s2)


def _check(npt, n, B, K, diag, mode, pairs, seed):
    t = _inputs(npt, n, B, K, pairs, seed)
    KC = diag or K
    kw = dict(dtype=torch.complex128, device='cuda')
    o1 = torch.full((B, npt, 3, KC) if mode == 0 else (B, npt, KC), complex('nan'), **kw)
    o2 = torch.full((B, npt, 3, KC), complex('nan'), **kw)
    call('mnpb_point_green', _lib.stream_handle(), npt, ptr(t['pt']), ptr(t['pt_med']), n,
         ptr(t['pos']), ptr(t['area']), ptr(t['face_med']), 2, ptr(t['k']), ptr(t['rptr']),
         ptr(t['cols']), ptr(t['g']), ptr(t['f']), mode, B, K, diag, ptr(t['k0']), ptr(t['sol']),
         ptr(o1), ptr(o2))
    want, size = _expected(t, mode, diag)
    for got, w, s in zip((o1, o2), want, size):
        # a term is good to some 40 rounding errors (phase k d of up to about 20,
        # distance, powers), and the sums to n of them
        assert bool(((got - w).abs() <= (40 + n) * EPS * s.abs().real + 1e-300).all())


@pytest.mark.parametrize('K', [1, 2, 3, 4, 5, 8, 11])
@pytest.mark.parametrize('mode', [0, 1])
def test_columns(gpu_ok, K, mode):
    _check(5, 301, 2, K, 0, mode, 'some', seed=K)


@pytest.mark.parametrize('diag', [1, 2, 3, 6])
@pytest.mark.parametrize('mode', [0, 1])
def test_columns_of_each_point(gpu_ok, diag, mode):
    _check(4, 130, 1, 4 * diag, diag, mode, 'some', seed=diag)


@pytest.mark.parametrize('n', [1, 31, 32, 33, 128, 129])
@pytest.mark.parametrize('pairs', ['none', 'all', 'some'])
def test_refined_pairs(gpu_ok, n, pairs):
    _check(3, n, 1, 2, 0, 0, pairs, seed=n)


@pytest.mark.parametrize('n', [262144, 262145])
def test_bits_up_to_their_room(gpu_ok, n):
    # 32 KB of bits; one face more searches the list for every face
    _check(3, n, 1, 1, 0, 0, 'some', seed=n)
