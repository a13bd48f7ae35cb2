"""FP64 dense building blocks at the sizes where their kernels change: LU
panels (rows per CTA, CTAs per cluster, columns per leaf, remainders) and
matrix products (tile edges, depth remainders, strides), solves (few and many
right-hand sides, interchange chains)."""
import numpy as np
import pytest
import scipy.linalg as sla
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _rand(*shape, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(shape + (2,), generator=g, dtype=torch.float64)
    return torch.view_as_complex(x).cuda()


def _getrf(A):
    """LU of A (batch, n, n), stored column by column: factors, pivots, info."""
    B, n, _ = A.shape
    LU = A.clone()
    piv = torch.zeros((B, n), dtype=torch.int32, device='cuda')
    info = torch.zeros(B, dtype=torch.int32, device='cuda')
    call('mnpb_getrf_f64', _lib.stream_handle(), n, B, ptr(LU), n, n * n, ptr(piv), n, ptr(info))
    torch.cuda.synchronize()
    return LU, piv, info


def _check_lu(A, LU, piv):
    """|P A - L U| <= 4 n eps |L| |U|, entrywise bounded by its maximum (the
    standard backward error bound of LU, complex arithmetic)."""
    n = A.shape[-1]
    for a, f, p in zip(A, LU, piv.cpu().numpy()):
        M = f.transpose(0, 1)
        L = torch.tril(M, -1)
        L.diagonal().fill_(1.0)
        U = torch.triu(M)
        perm = np.arange(n)
        for c, r in enumerate(p):
            perm[[c, r]] = perm[[r, c]]
        err = (a.transpose(0, 1)[torch.from_numpy(perm).cuda()] - L @ U).abs().max()
        bound = 4 * n * EPS * (L.abs() @ U.abs()).max()
        assert float(err) <= float(bound)


@pytest.mark.parametrize('n,batch', [(1, 3), (7, 2), (31, 1), (32, 2), (33, 5), (65, 150),
                                     (384, 2), (385, 2), (417, 1), (800, 3), (1200, 1)])
def test_lu_matches_lapack_pivots(gpu_ok, n, batch):
    A = _rand(batch, n, n, seed=n)
    LU, piv, info = _getrf(A)
    assert not info.any()
    _check_lu(A, LU, piv)
    for a, p in zip(A[:3].cpu().numpy(), piv[:3].cpu().numpy()):
        assert np.array_equal(sla.lu_factor(a.T)[1], p)


@pytest.mark.parametrize('n', [3073, 3105, 6150])
def test_lu_narrow_leaves(gpu_ok, n):
    # more rows than 8 CTAs hold 32 (16) columns of: 16- (8-) column leaves
    A = _rand(1, n, n, seed=n)
    LU, piv, info = _getrf(A)
    assert not info.any()
    _check_lu(A, LU, piv)


@pytest.mark.parametrize('n', [5, 40, 500])
def test_lu_ties_and_zero_columns(gpu_ok, n):
    # equal magnitudes: the first row wins; a zero column leaves its diagonal
    # in place and is reported once, by its first index
    A = torch.ones((2, n, n), dtype=torch.complex128, device='cuda')
    A[0] = torch.tril(A[0])                      # upper triangular matrix of ones
    A[1].zero_()
    A[1].diagonal().fill_(1.0 + 1.0j)
    A[1, n // 2] = 0.0                           # column n // 2
    LU, piv, info = _getrf(A)
    want = np.arange(n)
    assert np.array_equal(piv.cpu().numpy(), np.stack([want, want]))
    assert info.cpu().tolist() == [0, n // 2 + 1]
    assert torch.equal(LU[1], A[1])


@pytest.mark.parametrize('m,n,k,batch', [(1, 1, 1, 1), (33, 31, 7, 2), (32, 32, 8, 1),
                                         (64, 4, 33, 3), (65, 65, 25, 1), (700, 33, 40, 5),
                                         (63, 1, 200, 2), (129, 5, 513, 1), (64, 12, 64, 400),
                                         (1000, 16, 2900, 1), (2500, 13, 130, 3),
                                         (640, 70, 9, 40), (1300, 1290, 64, 1), (50, 40, 0, 2)])
@pytest.mark.parametrize('alpha,beta', [(-1.0, 1.0), (0.5 - 2.0j, 0.0), (1.0j, -0.25 + 1.0j)])
def test_zgemm_tiles(gpu_ok, m, n, k, batch, alpha, beta):
    # leading dimensions and strides larger than the matrices
    lda, ldb, ldc = m + 3, k + 2, m + 1
    A = _rand(batch, k + 1, lda, seed=1)
    B = _rand(batch, n + 2, ldb, seed=2)
    C0 = _rand(batch, n + 1, ldc, seed=3)
    C = C0.clone()
    al, be = complex(alpha), complex(beta)
    call('mnpb_zgemm', _lib.stream_handle(), m, n, k, batch, al.real, al.imag, ptr(A), lda,
         (k + 1) * lda, ptr(B), ldb, (n + 2) * ldb, be.real, be.imag, ptr(C), ldc, (n + 1) * ldc)
    a, b = A[:, :k, :m].transpose(1, 2), B[:, :n, :k].transpose(1, 2)
    c = C0[:, :n, :m].transpose(1, 2)
    ref = al * (a @ b) + be * c
    bound = 4 * (k + 3) * EPS * (abs(al) * (a.abs() @ b.abs()) + abs(be) * c.abs())
    got = C[:, :n, :m].transpose(1, 2)
    assert bool(((got - ref).abs() <= bound).all())
    assert torch.equal(C[:, n:], C0[:, n:]) and torch.equal(C[:, :, m:], C0[:, :, m:])


@pytest.mark.parametrize('n,nrhs,batch', [(1, 1, 2), (5, 2, 1), (63, 4, 1), (64, 1, 3),
                                          (65, 5, 2), (130, 16, 1), (300, 3, 80), (700, 1, 1),
                                          (700, 7, 1), (129, 17, 2), (200, 33, 1),
                                          (385, 385, 2), (1100, 100, 1), (4500, 2, 1),
                                          (5100, 1, 1)])
def test_getrs_few_and_many(gpu_ok, n, nrhs, batch):
    """|A x - b| <= 12 n eps |L| |U| |x| + |b| eps (backward error of the LU solve)."""
    A = _rand(batch, n, n, seed=n + 1)
    LU, piv, _ = _getrf(A)
    ldb = n + 2
    B0 = _rand(batch, nrhs + 1, ldb, seed=2)
    X = B0.clone()
    call('mnpb_getrs_f64', _lib.stream_handle(), n, batch, nrhs, ptr(LU), n, n * n, ptr(piv), n,
         ptr(X), ldb, (nrhs + 1) * ldb)
    assert torch.equal(X[:, nrhs:], B0[:, nrhs:]) and torch.equal(X[:, :, n:], B0[:, :, n:])
    x, b = X[:, :nrhs, :n].transpose(1, 2), B0[:, :nrhs, :n].transpose(1, 2)
    F = LU.transpose(1, 2)
    L = torch.tril(F, -1).abs()
    L.diagonal(dim1=1, dim2=2).fill_(1.0)
    mag = L @ (torch.triu(F).abs() @ x.abs())
    # row interchanges permute the bound's rows: compare with each column's largest
    res = (A.transpose(1, 2) @ x - b).abs().amax(1)
    assert bool((res <= 12 * n * EPS * mag.amax(1) + 4 * EPS * b.abs().amax(1)).all())


def test_getrs_interchange_chains(gpu_ok):
    # pivots whose targets repeat and chain: every step targets the last row, or
    # the row after next, or itself
    n = 300
    A = torch.eye(n, dtype=torch.complex128, device='cuda')
    for p in (np.full(n, n - 1), np.minimum(np.arange(n) + 2, n - 1), np.arange(n),
              np.where(np.arange(n) % 3 == 0, n - 1, np.minimum(np.arange(n) + 5, n - 1))):
        piv = torch.from_numpy(p.astype(np.int32)).cuda()[None]
        for nrhs in (1, 20):
            X = torch.arange(n, dtype=torch.float64, device='cuda').to(torch.complex128) \
                .repeat(nrhs, 1)
            call('mnpb_getrs_f64', _lib.stream_handle(), n, 1, nrhs, ptr(A), n, n * n, ptr(piv),
                 n, ptr(X), n, n * nrhs)
            want = np.arange(n)
            for c, r in enumerate(p):
                want[[c, r]] = want[[r, c]]
            assert np.array_equal(X.real.cpu().numpy(), np.tile(want, (nrhs, 1)))


@pytest.mark.parametrize('n,batch', [(5, 2), (33, 1), (128, 2), (129, 1), (300, 3), (1000, 1),
                                     (4300, 1)])
def test_right_solve_and_inverse(gpu_ok, n, batch):
    """Sigma1 = H1 G1^-1 and Delta^-1 of ``mnpb_bemret_init_f64`` on random
    matrices: |Sigma1 G1 - H1| <= 8 n eps |Sigma1| |G1| growth and
    |Delta Delta^-1 - I| <= 8 n eps |Delta| |Delta^-1| growth in the largest
    entry, with a growth factor of 30 for the factorisations."""
    G1, G2, H1, H2 = [_rand(batch, n, n, seed=s) for s in (1, 2, 3, 4)]
    GG, HH = torch.stack([G1, G2]), torch.stack([H1, H2])
    D = torch.empty_like(G1)
    eps = torch.tensor([[-10.0, 1.0, 1.0, 0.0]], dtype=torch.float64, device='cuda') \
        .repeat(batch, 1)
    kvac = torch.full((batch,), 0.01, dtype=torch.float64, device='cuda')
    nvec = torch.zeros((n, 3), dtype=torch.float64, device='cuda')
    piv = torch.empty((3, batch, n), dtype=torch.int32, device='cuda')
    info = torch.zeros((2, batch), dtype=torch.int32, device='cuda')
    wb = int(_lib.lib().mnpb_bemret_workspace_f64(n, batch))
    work = torch.empty(wb, dtype=torch.uint8, device='cuda')
    call('mnpb_bemret_init_f64', _lib.stream_handle(), n, batch, ptr(GG[0]), ptr(GG[1]),
         ptr(HH[0]), ptr(HH[1]), ptr(D), n, n * n, ptr(eps), ptr(kvac), ptr(nvec), 0, ptr(piv),
         ptr(info), ptr(work), wb)
    assert not info.any()
    T = lambda x: x.transpose(1, 2)
    S1, g1 = T(HH[0]), T(G1)
    scale = 30 * 8 * n * EPS
    res = (S1 @ g1 - T(H1)).abs().amax()
    assert float(res) <= scale * float((S1.abs() @ g1.abs()).amax())
    S2 = torch.linalg.solve(T(G2), T(H2), left=False)
    delta, inv = S1 - S2, T(D)
    eye = torch.eye(n, dtype=delta.dtype, device='cuda')
    # Sigma2 of the reference differs from the solver's by a relative error of
    # the same kind, which the inverse multiplies
    bound = scale * float((delta.abs() @ inv.abs()).amax() +
                          ((S2.abs() @ T(G2).abs()) @ torch.linalg.inv(T(G2)).abs()
                           @ inv.abs()).amax())
    assert float((delta @ inv - eye).abs().amax()) <= bound
