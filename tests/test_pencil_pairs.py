"""The tensor pencil stage over pencil pairs at its edges: windows of one to
five chunks, six (which runs one pencil at a time), x extents that are not a
multiple of 8 or 4, an odd y extent (one pencil at a time), z phase tables in
8 and 16 copies, accumulator groups of 1 to 18 terms, a partial second group of
128 rotations.

Tolerance: the parity bar of the correlation grids, 1e-4 of a grid's largest
value; the 16 smallest values of two forms within the bar differ by at most
twice that.
"""
import numpy as np
import pytest

from oracle import fftdock_oracle as O

pytestmark = pytest.mark.gpu

# dims, ligand diameter in cells, terms per sum
CASES = [((24, 24, 24), 4, 2), ((32, 32, 32), 12, 1), ((48, 48, 48), 20, 7), ((64, 64, 64), 30, 5),
         ((80, 80, 80), 37, 2), ((80, 80, 80), 45, 2), ((96, 96, 96), 36, 18), ((128, 128, 128), 37, 2),
         ((50, 24, 36), 14, 2), ((33, 20, 45), 9, 3), ((66, 27, 40), 22, 2), ((90, 16, 128), 13, 2),
         ((126, 120, 112), 37, 2), ((112, 128, 128), 37, 1), ((21, 40, 10), 5, 2)]


@pytest.mark.parametrize("dims,span,tg", CASES)
def test_pairs_match_the_oracle_and_the_fft_form(dims, span, tg):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rng = np.random.default_rng(sum(dims) + span)
    half = 0.5 * 1.2 * np.array(dims)
    rec = rng.uniform(-0.9, 0.9, (120, 3)) * half
    rt = rng.integers(0, 18, len(rec)).astype(np.int32)
    lig = rng.normal(size=(90, 3))
    lig *= (0.5 * 1.2 * (span - 1) * rng.uniform(0, 1, (90, 1)) ** (1 / 3)) / np.linalg.norm(lig, axis=1)[:, None]
    lt = rng.integers(0, 14, len(lig)).astype(np.int32)
    ace = rng.normal(size=(18, 18))
    ace = 0.5 * (ace + ace.T)
    rots = synth.quaternion_rotations(130, 7)
    geom = O.Geometry.centred(1.2, dims)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    cand, grids = {}, {}
    for mode in ("fft", "tensor"):
        with FFTScan(ScanConfig(grid_step=1.2, term_set="shape_ace", ace_matrix=ace, peaks_per_rot=4, rot_batch=256,
                                tc_terms_per_sum=tg, pencil_mode=mode, **kw)) as s:
            s.set_receptor(rec, rt)
            s.set_ligand(lig, lt)
            assert s.info()["pencil_path"] == mode
            cand[mode] = np.sort(s.candidates(rots)[0], axis=1)
            grids[mode] = [s.correlation_grid(r) for r in rots[[0, 127, 128]]]
    rg = O.receptor_terms(geom, rec, rt, O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=ace))
    w = O.ligand_term_weights(lt, O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=ace))
    rs = O.receptor_spectra(rg)
    scale = 0.0
    for i, rot in enumerate(rots[[0, 127, 128]]):
        cells, ok = O.bin_ligand(geom, rot, lig)
        assert ok
        corr = O.correlate(rs, O.ligand_grids(geom, cells, w))
        top = np.abs(corr).max()
        scale = max(scale, top)
        for mode in ("fft", "tensor"):
            assert np.abs(grids[mode][i] - corr).max() <= 1e-4 * top
    assert np.abs(cand["fft"] - cand["tensor"]).max() <= 2e-4 * scale
