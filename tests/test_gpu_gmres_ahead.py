"""GMRES issues the next operator product before it knows a step's residual: every
product that runs is counted, also one that convergence makes useless, and the
solution is that of the steps that count, over restarts too."""
import math

import pytest
import torch

from mnpbem_b200.bem_iter import _Counter, gmres

pytestmark = pytest.mark.gpu


def _rand(*shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.view_as_complex(torch.randn(shape + (2,), generator=g,
                                             dtype=torch.float64)).cuda()


def _solve(mul, b, **kw):
    calls, cnt = [0], _Counter()

    def apply_A(v):
        calls[0] += 1
        return mul(v)

    x, flag, relres, it = gmres(apply_A, b, counter=cnt, **kw)
    assert cnt.matvecs == calls[0]
    return x, flag, relres, it, calls[0]


@pytest.mark.parametrize('steps', [1, 2, 3, 5, 8, 13])
def test_sudden_convergence_drops_a_counted_product(gpu_ok, steps):
    """Eigenvalues at the roots of unity: the residual stands still for steps - 1
    steps and vanishes with the last, whose successor's product is under way from
    the third step on."""
    n = 40 * steps
    d = torch.polar(torch.ones(n, dtype=torch.float64),
                    2 * math.pi * (torch.arange(n) % steps).double() / steps).cuda()
    b = torch.ones(n, dtype=torch.complex128, device='cuda')
    x, flag, relres, it, calls = _solve(lambda v: d * v, b, tol=1e-10, maxit=50)
    assert flag == 0 and it == [1, steps]
    # the steps, the true residual at the end, and the dropped product
    assert calls == steps + 1 + (1 if steps >= 3 else 0)
    assert float((d * x - b).norm()) <= 1e-10 * float(b.norm())


@pytest.mark.parametrize('restart', [1, 3, 4, 7, 40])
def test_restarts(gpu_ok, restart):
    n = 300
    A = torch.eye(n, device='cuda') + 0.25 * _rand(n, n, seed=1) / n ** 0.5
    b = _rand(n, seed=2)
    x, flag, relres, it, calls = _solve(lambda v: A @ v, b, tol=1e-9, maxit=60, restart=restart)
    assert flag == 0 and relres <= 1e-9
    assert float((A @ x - b).norm()) <= 1.01e-9 * float(b.norm())
    # one product per step and one per cycle's true residual, and at most one dropped
    # per cycle
    assert it[1] + it[0] <= calls <= it[1] + 2 * it[0]
