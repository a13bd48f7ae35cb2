"""Row-sum items of the H-matrix products: the contribution lists are cut into 2 to 6
entries by how many there are.  The cut covers every list once, in order (no GPU),
and products with each length match the stored factors."""
import numpy as np
import pytest
import torch

from mnpbem_b200.clustertree import BlockPartition, ClusterTree, make_kaware_fadmiss
from mnpbem_b200.hmatrix import HMatrixGPU, HTopology, hmat_matvec
from test_gpu_hmat_product import _stored

# points, points per leaf, entries per item
CUTS = [(300, 32, 2), (800, 16, 3), (1000, 16, 4), (1200, 16, 5), (1500, 16, 6)]


def _topology(n, cleaf, device):
    pos = np.random.default_rng(n).normal(size=(n, 3)) * np.array([4.0, 1.0, 1.0])
    part = BlockPartition(ClusterTree(pos, cleaf=cleaf), make_kaware_fadmiss(1e-3, eta0=2.5))
    return pos, HTopology(part, 60, torch.device(device))


@pytest.mark.parametrize('n,cleaf,seg', CUTS)
def test_items_cover_every_list_once(n, cleaf, seg):
    _, topo = _topology(n, cleaf, 'cpu')
    items, cptr = topo.items.numpy(), topo.cptr.numpy()
    chunks, leaf_rows = topo.chunks.numpy(), topo.leaf_rows.numpy()
    assert (items[:, 2] - items[:, 1]).max() == seg
    ends = np.searchsorted(topo.lent_leaf, np.arange(topo.nleaf + 1))
    assert cptr[0] == 0 and cptr[-1] == len(items)
    for k, (leaf, r0) in enumerate(chunks):
        mine = items[cptr[k]:cptr[k + 1]]
        assert mine[0, 1] == ends[leaf] and mine[-1, 2] == ends[leaf + 1]
        assert np.array_equal(mine[1:, 1], mine[:-1, 2])
        assert (mine[:, 0] == k).all()
        assert (mine[:, 3] == (r0 << 6 | min(32, leaf_rows[leaf][1] - r0))).all()


@pytest.mark.gpu
@pytest.mark.parametrize('n,cleaf,seg', CUTS)
def test_products_with_each_length(gpu_ok, n, cleaf, seg):
    pos, topo = _topology(n, cleaf, 'cuda')
    d = np.linalg.norm(pos[:, None] - pos[None], axis=2) + 0.3
    h = HMatrixGPU(topo, torch.from_numpy(np.ascontiguousarray((np.exp(0.7j * d) / d).T)).cuda(),
                   n, 1e-6)
    A = _stored(topo, h, n)
    g = np.random.default_rng(1)
    for nc in (1, 4, 6):
        x = g.normal(size=(nc, n)) + 1j * g.normal(size=(nc, n))
        dx = torch.from_numpy(x).cuda()
        y, = hmat_matvec([h], [dx], [torch.empty_like(dx)], nc)
        # FP64 sums of up to 2 n products in another order
        err = np.abs(y.cpu().numpy() - x @ A.T).max()
        assert err <= 64 * n * 2.0 ** -52 * (np.abs(x) @ np.abs(A).T).max()
