"""FP32 (TF32-stored) LU panels at the sizes where the kernel changes: one or
two rows per thread of a cluster, the shared-memory slab of large batches; and
the mixed solve over the widths of its few-column kernels."""
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


@pytest.mark.parametrize('n,batch,K,shift', [(40, 2, 1, 0), (64, 1, 2, 0), (65, 3, 4, 0),
                                             (97, 1, 3, 1), (200, 5, 1, 1), (331, 40, 3, 0),
                                             (700, 1, 2, 0), (700, 1, 4, 3), (1500, 2, 1, 0)])
def test_mixed_solve_matches_fp64(gpu_ok, n, batch, K, shift):
    """The mixed factorisation's solve, refined to 1e-12 of the solution, against
    the FP64 solve of the same random systems: 1, 2, 3, 4 excitations use the
    1-, 4-, 8- and 12-column solves and products.  Both converge to the solution
    of the FP64 operator (``shift`` moves the factors off 16-byte alignment after
    the factorisation); their difference is bounded by the refinement's last
    correction and the FP64 solve's own error n eps kappa, kappa < 1e4 for
    these diagonally shifted matrices."""
    rng = torch.Generator().manual_seed(n)
    ld = (n + 3) // 4 * 4

    def mat(scale, shift):
        x = torch.randn((batch, n, n, 2), generator=rng, dtype=torch.float64) * scale / n ** 0.5
        x[..., 0] += shift * torch.eye(n, dtype=torch.float64)
        return torch.view_as_complex(x).cuda()

    G1, G2, H1, H2 = mat(0.2, 1.0), mat(0.2, 1.3), mat(0.2, 2.0), mat(0.2, -2.0)
    eps = torch.tensor([[-8.0, 1.0, 1.0, 0.0]], dtype=torch.float64, device='cuda') \
        .repeat(batch, 1)
    kvac = torch.full((batch,), 0.05, dtype=torch.float64, device='cuda')
    nv = torch.randn((n, 3), generator=rng, dtype=torch.float64)
    nv = (nv / nv.norm(dim=1, keepdim=True)).cuda()
    b = torch.view_as_complex(torch.randn((batch, 8, K, n, 2), generator=rng,
                                          dtype=torch.float64)).cuda()
    L, sh = _lib.lib(), _lib.stream_handle()
    # FP64
    GG, HH = torch.stack([G1, G2]), torch.stack([H1, H2])
    D = torch.empty_like(G1)
    piv = torch.empty((3, batch, n), dtype=torch.int32, device='cuda')
    info = torch.zeros((2, batch), dtype=torch.int32, device='cuda')
    work = torch.empty(int(L.mnpb_bemret_workspace_f64(n, batch)), dtype=torch.uint8,
                       device='cuda')
    call('mnpb_bemret_init_f64', sh, n, batch, ptr(GG[0]), ptr(GG[1]), ptr(HH[0]), ptr(HH[1]),
         ptr(D), n, n * n, ptr(eps), ptr(kvac), ptr(nv), 0, ptr(piv), ptr(info), ptr(work),
         work.numel())
    x64 = torch.empty_like(b)
    wb = batch * n * 15 * K * 16
    w64 = torch.empty(wb, dtype=torch.uint8, device='cuda')
    call('mnpb_bemret_solve_f64', sh, n, batch, K, ptr(GG[0]), ptr(GG[1]), ptr(HH[0]),
         ptr(HH[1]), ptr(D), n, n * n, ptr(piv), ptr(eps), ptr(kvac), ptr(nv), 0, ptr(b),
         ptr(x64), ptr(w64), wb)
    # mixed: padded FP64 operator and planar copies
    pad = lambda A: torch.nn.functional.pad(torch.view_as_real(A), (0, 0, 0, ld - n))
    ops = [torch.view_as_complex(pad(A).contiguous()) for A in (G1, G2, H1, H2)]
    pl = [pad(A).permute(0, 3, 1, 2).float().contiguous() for A in (G1, G2, H1, H2)]
    GGp, HHp = torch.stack(pl[:2]), torch.stack(pl[2:])
    Dp = torch.empty_like(pl[0])
    dinv = torch.empty(int(L.mnpb_bemret_dinv_floats(n, batch)), device='cuda')
    wm = torch.empty(int(L.mnpb_bemret_workspace_mixed(n, batch)), dtype=torch.uint8,
                     device='cuda')
    call('mnpb_bemret_init_mixed', sh, n, batch, ptr(GGp[0]), ptr(GGp[1]), ptr(HHp[0]),
         ptr(HHp[1]), ptr(Dp), ld, ptr(eps), ptr(kvac), ptr(nv), 0, ptr(piv), ptr(info),
         ptr(dinv), ptr(wm), wm.numel())
    assert not info.any()
    if shift:
        def moved(t):
            buf = torch.empty(t.numel() + 4, device='cuda')
            out = buf[shift:shift + t.numel()].view(t.shape)
            return out.copy_(t)

        GGp, HHp, Dp = moved(GGp), moved(HHp), moved(Dp)
    x = torch.empty_like(b)
    wr = torch.empty(int(L.mnpb_bemret_refine_workspace(n, batch, K)), dtype=torch.uint8,
                     device='cuda')
    iters, rel = np.zeros(batch, dtype=np.int32), np.zeros(batch)
    call('mnpb_bemret_solve_refine', sh, n, batch, K, ptr(GGp[0]), ptr(GGp[1]), ptr(HHp[0]),
         ptr(HHp[1]), ptr(Dp), ld, ptr(piv), ptr(dinv), ptr(ops[0]), ptr(ops[1]), ptr(ops[2]),
         ptr(ops[3]), ptr(eps), ptr(kvac), ptr(nv), 0, ptr(b), ptr(x), 30, 1e-12, ptr(iters),
         ptr(rel), ptr(wr), wr.numel())
    err = (x - x64).flatten(1).norm(dim=1) / x64.flatten(1).norm(dim=1)
    assert float(err.max()) <= 1e-11 + 1e4 * n * 2.0 ** -52
