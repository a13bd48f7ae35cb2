"""Row interchanges of ``mnpb_getrs_f64`` that no LU of this package makes: targets
above the step's own row, also such that step and target chase each other (two
rows exchanged twice, rings of rows).  They are carried out in their order, as
LAPACK's laswp does, on every route: few right-hand sides, many, and more rows
than the interchanges are composed for."""
import numpy as np
import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


def _targets(n, kind):
    i = np.arange(n)
    if kind == 'pairs':                      # 0 <-> 1, 1 <-> 0, 2 <-> 3, ...
        return np.minimum(i ^ 1, n - 1)
    if kind == 'ring':                       # every step targets the row before
        return (i - 1) % n
    if kind == 'first':
        return np.zeros(n, dtype=int)
    return np.random.default_rng(n).integers(0, n, n)


@pytest.mark.parametrize('kind', ['pairs', 'ring', 'first', 'random'])
@pytest.mark.parametrize('n,nrhs,batch', [(2, 1, 1), (65, 3, 2), (300, 1, 2), (300, 16, 1),
                                          (300, 20, 2), (1100, 40, 1), (4500, 1, 1)])
def test_any_targets_in_order(gpu_ok, kind, n, nrhs, batch):
    A = torch.eye(n, dtype=torch.complex128, device='cuda').repeat(batch, 1, 1)
    p = np.stack([np.roll(_targets(n, kind), b) for b in range(batch)])
    piv = torch.from_numpy(p.astype(np.int32)).cuda()
    X = torch.arange(n, dtype=torch.float64, device='cuda').to(torch.complex128) \
        .repeat(batch, nrhs, 1)
    call('mnpb_getrs_f64', _lib.stream_handle(), n, batch, nrhs, ptr(A), n, n * n, ptr(piv), n,
         ptr(X), n, n * nrhs)
    for b in range(batch):
        want = np.arange(n)
        for c, r in enumerate(p[b]):
            want[[c, r]] = want[[r, c]]
        assert np.array_equal(X[b].real.cpu().numpy(), np.tile(want, (nrhs, 1)))
