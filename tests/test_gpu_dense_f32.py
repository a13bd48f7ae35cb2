"""FP32 (TF32-stored) LU panels at the sizes where the kernel changes: one or
two rows per thread of a cluster, the shared-memory slab of large batches."""
import numpy as np
import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

TF32 = 2.0 ** -11


def _planar(batch, n, ld, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn((batch, 2, n, ld), generator=g, dtype=torch.float32).cuda()


def _matrix(P, n):
    return torch.complex(P[:, 0, :, :n].double(), P[:, 1, :, :n].double()).transpose(1, 2)


def _getrf(A, n):
    B, _, _, ld = A.shape
    LU = A.clone()
    piv = torch.zeros((B, n), dtype=torch.int32, device='cuda')
    info = torch.zeros(B, dtype=torch.int32, device='cuda')
    wb = int(_lib.lib().mnpb_f32_workspace(n, B))
    work = torch.empty(wb, dtype=torch.uint8, device='cuda')
    call('mnpb_getrf_c32p', _lib.stream_handle(), n, B, ptr(LU), ld, ld * n, 2 * ld * n, ptr(piv),
         n, ptr(info), ptr(work), wb)
    return LU, piv, info


@pytest.mark.parametrize('n,batch', [(1, 2), (9, 3), (32, 1), (33, 2), (100, 149), (100, 148),
                                     (384, 2), (385, 2), (400, 80), (769, 1), (1537, 50),
                                     (3100, 1), (6200, 1)])
def test_lu_planar(gpu_ok, n, batch):
    """|P A - L U| <= 8 2^-11 |L| |U| in the largest entry: L, U and the block
    inverses the updates multiply with are stored as TF32."""
    ld = (n + 3) // 4 * 4
    A = _planar(batch, n, ld, seed=n)
    LU, piv, info = _getrf(A, n)
    assert not info.any()
    for b in sorted({0, batch // 2, batch - 1}):
        M = _matrix(LU[b:b + 1], n)[0]
        L = torch.tril(M, -1)
        L.diagonal().fill_(1.0)
        U = torch.triu(M)
        perm = np.arange(n)
        for c, r in enumerate(piv[b].cpu().numpy()):
            assert c <= r < n
            perm[[c, r]] = perm[[r, c]]
        a = _matrix(A[b:b + 1], n)[0][torch.from_numpy(perm).cuda()]
        assert float((a - L @ U).abs().max()) <= 8 * TF32 * float((L.abs() @ U.abs()).max())
        # partial pivoting on |re| + |im|: no multiplier above sqrt(2) by more than rounding
        assert float(torch.tril(M, -1).abs().max() if n > 1 else 0.0) <= 2 ** 0.5 * (1 + 4 * TF32)


def test_lu_planar_zero_column(gpu_ok):
    n = 70
    A = torch.zeros((2, 2, n, 72), device='cuda')
    for b in range(2):
        A[b, 0, torch.arange(n), torch.arange(n)] = 1.5
    A[1, 0, 40, 40] = 0.0
    LU, piv, info = _getrf(A, n)
    assert torch.equal(LU, A)
    assert info.cpu().tolist() == [0, 41]
    assert np.array_equal(piv.cpu().numpy(), np.tile(np.arange(n), (2, 1)))
