"""The FP64 LU and solves on two streams: ordered with the caller's stream on both sides,
from more threads at once than there are second streams, and under the caller's
own capture, where it stays on one stream."""
import threading

import numpy as np
import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


class _LU:
    """One factorisation of random matrices; the buffers belong to the
    stream that is current here."""

    def __init__(self, n, batch, seed):
        g = torch.Generator(device='cuda').manual_seed(seed)
        self.n, self.batch = n, batch
        self.A = torch.randn(batch, n, n, dtype=torch.complex128, device='cuda', generator=g)
        self.LU = torch.empty_like(self.A)
        self.piv = torch.zeros((batch, n), dtype=torch.int32, device='cuda')
        self.info = torch.zeros(batch, dtype=torch.int32, device='cuda')

    def run(self):
        n = self.n
        self.LU.copy_(self.A)                    # queued before, on the same stream
        call('mnpb_getrf_f64', _lib.stream_handle(), n, self.batch, ptr(self.LU), n, n * n,
             ptr(self.piv), n, ptr(self.info))
        self.out = self.LU.clone()               # queued after
        self.LU.fill_(float('nan'))

    def check(self):
        """|P A - L U| <= 4 n eps |L| |U| in the largest entry."""
        torch.cuda.synchronize()
        assert not self.info.any()
        n = self.n
        for b in range(self.batch):
            A, M = self.A[b].T, self.out[b].T
            L = torch.tril(M, -1) + torch.eye(n, device='cuda')
            U = torch.triu(M)
            perm = np.arange(n)
            for i, r in enumerate(self.piv[b].cpu().numpy()):
                perm[[i, r]] = perm[[r, i]]
            err = (A[torch.from_numpy(perm).cuda()] - L @ U).abs().max()
            bound = 4 * n * np.finfo(np.float64).eps * (L.abs() @ U.abs()).max()
            assert float(err) <= float(bound)


@pytest.mark.parametrize('n,batch', [(257, 5), (384, 4), (513, 3), (900, 4), (1281, 1)])
def test_ordered_with_the_callers_stream(gpu_ok, n, batch):
    with torch.cuda.stream(torch.cuda.Stream()):
        f = _LU(n, batch, n)
        for _ in range(3):
            f.run()
        f.check()


def test_threads_at_once(gpu_ok):
    fs, errors = [None] * 12, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                fs[i] = _LU(640 + 60 * i, 2, i)
                for _ in range(4):
                    fs[i].run()
                torch.cuda.current_stream().synchronize()
        except Exception as e:                   # noqa: BLE001 (reported below)
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(12)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    for f in fs:
        f.check()


def test_captured_by_the_caller(gpu_ok):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        f = _LU(700, 2, 7)
        f.run()
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f.run()
    f.out.zero_()
    g.replay()
    g.replay()
    f.check()


def test_solves_in_halves_repeat(gpu_ok):
    """The factorisation of a wavelength's matrices (solves split over two
    streams) from eight threads at once: bitwise what one thread alone gets."""
    n, B = 700, 2
    L = _lib.lib()
    g = torch.Generator(device='cuda').manual_seed(3)
    kw = dict(dtype=torch.complex128, device='cuda', generator=g)
    G0 = torch.randn(2, B, n, n, **kw) + 10 * torch.eye(n, device='cuda')
    H0 = torch.randn(2, B, n, n, **kw)
    eps = torch.tensor([1.77, 0.0, -4.0, 0.9] * B, dtype=torch.float64, device='cuda')
    kv = torch.full((B,), 0.0125, dtype=torch.float64, device='cuda')
    nv = torch.randn(n, 3, dtype=torch.float64, device='cuda', generator=g)
    torch.cuda.synchronize()

    def init():
        G, H, D = G0.clone(), H0.clone(), torch.empty(B, n, n, dtype=torch.complex128,
                                                      device='cuda')
        piv = torch.zeros(3, B, n, dtype=torch.int32, device='cuda')
        info = torch.zeros(2, B, dtype=torch.int32, device='cuda')
        work = torch.empty(int(L.mnpb_bemret_workspace_f64(n, B)), dtype=torch.uint8,
                           device='cuda')
        call('mnpb_bemret_init_f64', _lib.stream_handle(), n, B, ptr(G[0]), ptr(G[1]), ptr(H[0]),
             ptr(H[1]), ptr(D), n, n * n, ptr(eps), ptr(kv), ptr(nv), 0, ptr(piv), ptr(info),
             ptr(work), work.numel())
        torch.cuda.current_stream().synchronize()
        return G, H, D

    want = init()
    assert all(bool(torch.isfinite(torch.view_as_real(x)).all()) for x in want)
    got, ts = [None] * 8, []

    def work_(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = init()

    for i in range(8):
        ts.append(threading.Thread(target=work_, args=(i,)))
        ts[-1].start()
    for t in ts:
        t.join()
    for r in got:
        assert r is not None and all(torch.equal(a, b) for a, b in zip(r, want))
