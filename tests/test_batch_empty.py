"""A batched solver without particles: empty results, as a loop over none gives.
Needs no GPU."""
from mnpbem_b200.batch import BatchedBEMRet
from mnpbem_b200.excitation import PlaneWaveRet


def test_no_particles_give_empty_spectra():
    exc = PlaneWaveRet([[1, 0, 0], [0, 1, 0]], [[0, 0, 1], [0, 0, 1]])
    bem = BatchedBEMRet([], mem_bytes=1 << 20, tuner=None)
    for pad in (False, True):
        res = bem.solve_spectrum(exc, [500.0, 600.0, 700.0], keep_solutions=pad)
        assert res['ext'].shape == res['sca'].shape == (0, 3, 2)
        assert res['iters'].shape == (0, 3)
        assert bem.stats == []
    assert res['solutions'] == []
