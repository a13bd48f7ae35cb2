"""The batched solver's arena: batches of different face counts carved from one
allocation give what separate solvers give, pass after pass."""
import numpy as np
import pytest

from mnpbem_b200.batch import BatchedBEMRet
from mnpbem_b200.excitation import PlaneWaveRet
from mnpbem_b200.geometry import ComParticle, trirod, trisphere
from mnpbem_b200.materials import EpsConst, EpsDrude

pytestmark = pytest.mark.gpu


def _particles():
    eps = [EpsConst(1.77), EpsDrude(10.0, 9.065, 0.0708)]
    return [ComParticle(eps, [p], [[2, 1]], 1)
            for p in (trisphere(144, 20.0), trirod(12.0, 40.0, (11, 6, 9)), trisphere(60, 10.0))]


def test_arena_batches_match_single_particles(gpu_ok):
    exc = PlaneWaveRet([[1, 0, 0], [0, 1, 0]], [[0, 0, 1], [0, 0, 1]])
    parts = _particles()
    kw = dict(refine_tol=1e-11, tuner=None, max_batch=4)
    many = BatchedBEMRet(parts, **kw)
    one = [BatchedBEMRet([p], **kw) for p in parts]
    for eneis in ([500.0, 560.0, 610.0], [450.0, 700.0], [500.0, 560.0, 610.0, 650.0, 690.0]):
        res = many.solve_spectrum(exc, eneis)
        for i, b in enumerate(one):
            ref = b.solve_spectrum(exc, eneis)
            # both refined to 1e-11 of the solution
            assert np.abs(res['ext'][i] / ref['ext'][0] - 1).max() < 1e-9
            assert np.abs(res['sca'][i] / ref['sca'][0] - 1).max() < 1e-9
