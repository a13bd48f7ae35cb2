"""The FP64 factorisations give the same bits whether or not a second stream was to
be had: alone, under the caller's own capture (one stream), and from more threads
at once than there are second streams.  Sizes whose last block has 1 to 16 columns,
which go to the products' few-column kernels, and one that has none such."""
import threading

import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


def _rand(*shape, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device='cuda', generator=g)


class _LU:
    def __init__(self, n, batch):
        self.n, self.batch = n, batch
        self.A = _rand(batch, n, n, seed=n)
        self.out = torch.empty_like(self.A)
        self.piv = torch.zeros((batch, n), dtype=torch.int32, device='cuda')
        self.info = torch.zeros(batch, dtype=torch.int32, device='cuda')

    def run(self):
        n = self.n
        self.out.copy_(self.A)
        call('mnpb_getrf_f64', _lib.stream_handle(), n, self.batch, ptr(self.out), n, n * n,
             ptr(self.piv), n, ptr(self.info))

    def result(self):
        return [self.out.clone(), self.piv.clone()]


class _Init:
    """LUs, two right solves and an inverse of a wavelength's matrices."""

    def __init__(self, n, batch):
        self.n, self.batch = n, batch
        self.G0 = _rand(2, batch, n, n, seed=n) + 10 * torch.eye(n, device='cuda')
        self.H0 = _rand(2, batch, n, n, seed=n + 1)
        self.G, self.H = torch.empty_like(self.G0), torch.empty_like(self.H0)
        self.D = torch.empty(batch, n, n, dtype=torch.complex128, device='cuda')
        self.eps = torch.tensor([1.77, 0.0, -4.0, 0.9] * batch, dtype=torch.float64, device='cuda')
        self.kv = torch.full((batch,), 0.0125, dtype=torch.float64, device='cuda')
        self.nv = torch.ones(n, 3, dtype=torch.float64, device='cuda')
        self.piv = torch.zeros(3, batch, n, dtype=torch.int32, device='cuda')
        self.info = torch.zeros(2, batch, dtype=torch.int32, device='cuda')
        self.work = torch.empty(int(_lib.lib().mnpb_bemret_workspace_f64(n, batch)),
                                dtype=torch.uint8, device='cuda')

    def run(self):
        n = self.n
        self.G.copy_(self.G0)
        self.H.copy_(self.H0)
        call('mnpb_bemret_init_f64', _lib.stream_handle(), n, self.batch, ptr(self.G[0]),
             ptr(self.G[1]), ptr(self.H[0]), ptr(self.H[1]), ptr(self.D), n, n * n,
             ptr(self.eps), ptr(self.kv), ptr(self.nv), 0, ptr(self.piv), ptr(self.info),
             ptr(self.work), self.work.numel())

    def result(self):
        return [x.clone() for x in (self.G, self.H, self.D, self.piv)]


CASES = [(_LU, 1290, 1), (_LU, 652, 2), (_LU, 700, 2), (_Init, 650, 2), (_Init, 1290, 1)]


def _same(got, want):
    return all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize('kind,n,batch', CASES)
def test_same_bits_under_capture(gpu_ok, kind, n, batch):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        f = kind(n, batch)
        f.run()
        want = f.result()
    s.synchronize()
    assert bool(torch.isfinite(torch.view_as_real(want[0])).all())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f.run()
    g.replay()
    torch.cuda.synchronize()
    assert _same(f.result(), want)


@pytest.mark.parametrize('kind,n,batch', CASES)
def test_same_bits_from_many_threads(gpu_ok, kind, n, batch):
    f = kind(n, batch)
    f.run()
    want = f.result()
    torch.cuda.synchronize()
    count = 20                                   # the pool holds eight second streams
    start, got, errors = threading.Barrier(count), [None] * count, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                h = kind(n, batch)
                torch.cuda.current_stream().synchronize()
                start.wait()
                h.run()
                got[i] = h.result()
                torch.cuda.current_stream().synchronize()
        except Exception as e:                   # noqa: BLE001 (reported below)
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(count)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    assert all(_same(r, want) for r in got)
