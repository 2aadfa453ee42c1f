"""The in-place plane stage at the sizes where its passes change: odd y and z
sizes (two rows per complex line, a lone last row), primes (a pass of radix
1), sizes that need three passes per axis, the smallest planes, a flat plane.

Tolerance: FP32 transforms of at most 256 points per axis after the FP32 x
stage; the parity bar of the correlation grids, 1e-4 of the largest value.
"""
import numpy as np
import pytest

from oracle import fftdock_oracle as O

pytestmark = pytest.mark.gpu

DIMS = [(10, 8, 8), (9, 9, 9), (12, 11, 13), (14, 13, 22), (20, 15, 25), (16, 21, 33), (8, 125, 10), (8, 10, 125),
        (9, 26, 250), (11, 242, 26), (12, 16, 256), (8, 147, 27), (13, 64, 49), (10, 143, 30), (8, 256, 18)]


def _case(dims, n_rec=40, n_lig=5):
    rng = np.random.default_rng(sum(dims))
    half = 0.5 * 1.2 * np.array(dims)
    rec = rng.uniform(-0.9, 0.9, (n_rec, 3)) * half
    lig = rng.uniform(-0.35, 0.35, (n_lig, 3)) * half.min()
    return rec, lig, rng.integers(0, 18, n_rec).astype(np.int32), rng.integers(0, 18, n_lig).astype(np.int32), rng


@pytest.mark.parametrize("mode", ["fft", "tensor"])
@pytest.mark.parametrize("dims", DIMS)
def test_correlation_grid_and_peaks(dims, mode):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rec, lig, rt, lt, rng = _case(dims)
    ace = synth.ace_matrix(18, 5)
    rots = synth.quaternion_rotations(3, 7)
    geom = O.Geometry.centred(1.2, dims)
    tp = O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=ace)
    rg = O.receptor_terms(geom, rec, rt, tp)
    w = O.ligand_term_weights(lt, tp)
    rs = O.receptor_spectra(rg)
    with FFTScan(ScanConfig(grid_dims=dims, grid_step=1.2, term_set="shape_ace", peaks_per_rot=4, ace_matrix=ace,
                            pencil_mode=mode)) as s:
        s.set_receptor(rec, rt)
        s.set_ligand(lig, lt)
        res = s.scan(rots)
        for i, rot in enumerate(rots):
            ref = O.scan_rotation(geom, rg, rs, lig, w, rot, 4)
            cells, ok = O.bin_ligand(geom, rot, lig)
            assert ok
            corr = O.correlate(rs, O.ligand_grids(geom, cells, w))
            got = s.correlation_grid(rot)
            assert np.abs(got - corr).max() <= 1e-4 * np.abs(corr).max()
            _, _, score = res.rotation(i)
            assert np.all(np.abs(score - ref.scores) <= 1e-4 * np.maximum(np.abs(ref.scores), 1.0))


@pytest.mark.parametrize("dims", [(12, 24, 20), (9, 21, 25)])
def test_flat_plane_keeps_the_lowest_offsets(dims):
    """No receptor: every cell is zero, far more ties than the candidate list
    holds; the lowest offsets win."""
    from proddl2_gb300 import FFTScan, ScanConfig
    _, lig, _, _, _ = _case(dims)
    with FFTScan(ScanConfig(grid_dims=dims, grid_step=1.2, term_set="shape", peaks_per_rot=4)) as s:
        s.set_receptor(np.zeros((0, 3)))
        s.set_ligand(lig)
        cell, _, score = s.scan(np.eye(3)[None]).rotation(0)
    assert np.array_equal(cell, [[0, 0, k] for k in range(4)])
    assert np.all(score == 0.0)
