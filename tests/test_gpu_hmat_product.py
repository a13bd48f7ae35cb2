"""H-matrix products against the stored blocks and factors themselves, over the
numbers of columns (chunks of four and remainders), ranks on both sides of 16
and row pieces of every length the leaves give."""
import numpy as np
import pytest
import torch

from mnpbem_b200.clustertree import BlockPartition, ClusterTree, make_kaware_fadmiss
from mnpbem_b200.hmatrix import HMatrixGPU, HTopology, hmat_matvec

pytestmark = pytest.mark.gpu


def _case(n, cleaf, kmax, seed):
    g = np.random.default_rng(seed)
    pos = g.normal(size=(n, 3)) * np.array([4.0, 1.0, 1.0])
    tree = ClusterTree(pos, cleaf=cleaf)
    part = BlockPartition(tree, make_kaware_fadmiss(1e-3, eta0=2.5))
    topo = HTopology(part, kmax, torch.device('cuda'))
    d = np.linalg.norm(pos[:, None] - pos[None], axis=2) + 0.3
    mats = [np.exp(1j * k * d) / d for k in (0.5, 3.0)]
    return topo, [HMatrixGPU(topo, torch.from_numpy(np.ascontiguousarray(m.T)).cuda(), n, 1e-6)
                  for m in mats]


def _stored(topo, h, n):
    """The compressed matrix as stored, in face order."""
    A = np.zeros((n, n), dtype=complex)
    D = h.D.double().cpu().numpy().view(complex)
    for b, (r0, m, c0, k) in enumerate(topo.part.dense):
        o = topo.offD_h[b]
        A[r0:r0 + m, c0:c0 + k] = D[o:o + m * k].reshape(k, m).T
    for b, (r0, m, c0, k) in enumerate(topo.part.lowrank):
        U, V = h.factors(b)
        A[r0:r0 + m, c0:c0 + k] = U @ V.T
    c2p = topo.c2p.cpu().numpy()
    out = np.zeros_like(A)
    out[np.ix_(c2p, c2p)] = A
    return out


@pytest.mark.parametrize('n,cleaf,kmax', [(40, 64, 20), (333, 16, 12), (700, 33, 60),
                                          (1500, 64, 100)])
def test_product_of_stored_factors(gpu_ok, n, cleaf, kmax):
    topo, hs = _case(n, cleaf, kmax, seed=n)
    ref = [_stored(topo, h, n) for h in hs]
    g = np.random.default_rng(1)
    for nc in (1, 2, 3, 4, 5, 8, 11):
        xs = [g.normal(size=(nc, n)) + 1j * g.normal(size=(nc, n)) for _ in hs]
        dx = [torch.from_numpy(x).cuda() for x in xs]
        ys = hmat_matvec(hs, dx, [torch.empty_like(x) for x in dx], nc)
        for A, x, y in zip(ref, xs, ys):
            # FP64 sums of up to 2 n products in another order (the factors' sizes
            # bound the terms of the low-rank blocks)
            err = np.abs(y.cpu().numpy() - x @ A.T).max()
            size = (np.abs(x) @ np.abs(A).T).max()
            assert err <= 64 * n * 2.0 ** -52 * size
