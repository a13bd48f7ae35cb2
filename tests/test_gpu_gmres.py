"""GMRES building blocks: one Arnoldi step over vector lengths around the
kernels' pieces (64 elements of the projection, 2048 of a chunk, 32 chunks),
rotations and the back substitution around its 256 threads."""
import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('L,j', [(1, 0), (63, 0), (64, 3), (65, 5), (2049, 4), (5000, 33),
                                 (70000, 9)])
def test_arnoldi_step(gpu_ok, L, j):
    """One Arnoldi step against a basis of j + 1 orthonormal vectors: h = V^H w,
    the new vector orthonormal to them (CGS2: to c L eps)."""
    g = torch.Generator().manual_seed(L + j)
    j = min(j, L - 1)
    X = torch.view_as_complex(torch.randn((L, j + 2, 2), generator=g, dtype=torch.float64))
    Q = torch.linalg.qr(X[:, :j + 1])[0]
    V = torch.zeros((j + 2, L), dtype=torch.complex128, device='cuda')
    V[:j + 1] = Q.T.cuda()
    w0 = X[:, j + 1].contiguous().cuda()
    w = w0.clone()
    H = torch.zeros(j + 2, dtype=torch.complex128, device='cuda')
    nrm = torch.zeros(1, dtype=torch.float64, device='cuda')
    wb = int(_lib.lib().mnpb_gmres_workspace(L, j))
    work = torch.empty(wb, dtype=torch.uint8, device='cuda')
    call('mnpb_gmres_arnoldi', _lib.stream_handle(), L, j, ptr(V), L, ptr(w), ptr(H), ptr(nrm),
         ptr(work), wb)
    tol = 16 * (L ** 0.5 + j) * 2.0 ** -52
    h = V[:j + 1].conj() @ w0
    assert float((H[:j + 1] - h).abs().max()) <= tol * float(w0.norm())
    r = w0 - V[:j + 1].T @ h
    r = r - V[:j + 1].T @ (V[:j + 1].conj() @ r)
    # a residual of rounding size (L = j + 1) has no direction to compare
    if float(r.norm()) > 1e-8 * float(w0.norm()):
        assert abs(float(nrm) - float(r.norm())) <= tol * float(w0.norm())
        assert abs(float(H[j + 1].real) - float(nrm)) == 0.0
        got = V.conj() @ V.T
        eye = torch.eye(j + 2, dtype=got.dtype, device='cuda')
        assert float((got - eye).abs().max()) <= tol * float(w0.norm() / r.norm())


@pytest.mark.parametrize('m', [1, 2, 37, 256, 257, 700])
def test_givens_and_back_substitution(gpu_ok, m):
    """Rotating a random Hessenberg matrix column by column and solving gives the
    least-squares solution: |H^H (beta e1 - H y)| <= 64 m^2 eps |H| |y|-sized."""
    g = torch.Generator().manual_seed(m)
    Hm = torch.view_as_complex(torch.randn((m + 1, m, 2), generator=g, dtype=torch.float64))
    Hm = torch.triu(Hm, -1) / m ** 0.5 + 2.0 * torch.eye(m + 1, m, dtype=torch.float64)
    ldh = m + 1
    H = Hm.T.contiguous().cuda()                      # column-major
    cs = torch.zeros(m, dtype=torch.float64, device='cuda')
    sn = torch.zeros(m, dtype=torch.complex128, device='cuda')
    gv = torch.zeros(m + 1, dtype=torch.complex128, device='cuda')
    gv[0] = 3.0
    res = torch.zeros(1, dtype=torch.float64, device='cuda')
    for j in range(m):
        call('mnpb_gmres_givens', _lib.stream_handle(), j, ptr(H), ldh, ptr(cs), ptr(sn), ptr(gv),
             ptr(res))
    y = torch.zeros(m, dtype=torch.complex128, device='cuda')
    z = torch.zeros(m, dtype=torch.complex128, device='cuda')
    eye = torch.eye(m, dtype=torch.complex128, device='cuda')
    call('mnpb_gmres_update', _lib.stream_handle(), m, m, ptr(H), ldh, ptr(gv), ptr(eye), m,
         ptr(y), ptr(z))
    assert torch.equal(y, z)
    e1 = torch.zeros(m + 1, dtype=torch.complex128)
    e1[0] = 3.0
    r = e1 - Hm @ y.cpu()
    tol = 64 * m * 2.0 ** -52
    size = float(torch.linalg.matrix_norm(Hm)) * (3.0 + float(torch.linalg.matrix_norm(Hm)) *
                                                  float(y.cpu().norm()))
    assert float((Hm.conj().T @ r).norm()) <= tol * size
    assert abs(float(res) - float(r.norm())) <= tol * size
