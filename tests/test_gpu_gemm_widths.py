"""TF32 tensor-core GEMM over its tile widths: 32, 64 and 128 columns are chosen
by how many tiles a product has, so each width is met here with full tiles and
remainders, with A read in place and packed, and with C in A's place."""

import pytest
import torch

from mnpbem_b200 import _lib
from mnpbem_b200._lib import call, ptr

pytestmark = pytest.mark.gpu
A_TF32, ROUND_C = 1, 2


def _planar(batch, cols, ld, seed):
    """Random planar matrices of TF32 values (exact operands of the tensor cores)."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    x = torch.randn(batch, 2, cols, ld, device='cuda', generator=g)
    return (x.view(torch.int32) & -8192).view(torch.float32)


def _complex(x, rows, cols):
    return torch.complex(x[:, 0, :cols, :rows].double(), x[:, 1, :cols, :rows].double()) \
        .transpose(1, 2)


@pytest.mark.parametrize('m,n,k,batch', [(1, 33, 4, 1), (128, 128, 128, 1), (129, 97, 32, 2),
                                         (300, 130, 36, 3), (128, 1190, 128, 4),
                                         (2700, 96, 32, 2), (2000, 200, 68, 2),
                                         (1000, 1000, 100, 1), (1000, 1000, 100, 3),
                                         (260, 65, 1000, 27), (384, 384, 40, 40)])
@pytest.mark.parametrize('flags', [0, A_TF32, A_TF32 | ROUND_C])
def test_widths(gpu_ok, m, n, k, batch, flags):
    """|C - ref| <= 4 (k + 4) 2^-23 |A||B| + 2^-22 |beta C0| (exact products, FP32
    sums that may truncate), plus 2^-11 |C| where C is stored as TF32."""
    lda, ldb = (m + 3) // 4 * 4 + 4, (k + 3) // 4 * 4
    A, B, C = _planar(batch, k, lda, 1), _planar(batch, n, ldb, 2), _planar(batch, n + 1, lda, 3)
    C0 = C.clone()
    work = torch.empty(int(_lib.lib().mnpb_cgemm_tf32_workspace(m, k, batch)),
                       dtype=torch.uint8, device='cuda')
    call('mnpb_cgemm_tf32_ex', _lib.stream_handle(), m, n, k, batch, -1.0, ptr(A), lda, k * lda,
         2 * k * lda, ptr(B), ldb, n * ldb, 2 * n * ldb, 0.5, ptr(C), lda, (n + 1) * lda,
         2 * (n + 1) * lda, ptr(work), work.numel(), flags)
    a, b = _complex(A, m, k), _complex(B, k, n)
    c0, got = _complex(C0, m, n), _complex(C, m, n)
    ref = 0.5 * c0 - a @ b
    bound = 4 * (k + 4) * 2.0 ** -23 * (a.abs() @ b.abs()) + 2.0 ** -22 * c0.abs()
    if flags & ROUND_C:
        bound = bound + 2.0 ** -11 * 2 ** 0.5 * ref.abs()
    assert bool(((got - ref).abs() <= bound).all())
    assert torch.equal(C[:, :, n:], C0[:, :, n:]) and torch.equal(C[..., m:], C0[..., m:])


@pytest.mark.parametrize('m,n,batch', [(700, 128, 1), (300, 100, 2), (2884, 128, 1), (500, 33, 3)])
def test_c_in_place_of_a(gpu_ok, m, n, batch):
    """C = A B with C in A's place, as the leaves of the right solves call it."""
    lda, ldb = (m + 3) // 4 * 4, (n + 3) // 4 * 4
    A, B = _planar(batch, n, lda, 4), _planar(batch, n, ldb, 5)
    a, b = _complex(A, m, n), _complex(B, n, n)
    call('mnpb_cgemm_tf32_ex', _lib.stream_handle(), m, n, n, batch, 1.0, ptr(A), lda, n * lda,
         2 * n * lda, ptr(B), ldb, n * ldb, 2 * n * ldb, 0.0, ptr(A), lda, n * lda, 2 * n * lda,
         0, 0, A_TF32)
    bound = 4 * (n + 4) * 2.0 ** -23 * (a.abs() @ b.abs())
    assert bool(((_complex(A, m, n) - a @ b).abs() <= bound).all())
