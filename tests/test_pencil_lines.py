"""The FFT form of the pencil stage for one term and for ljComp at its edges:
odd y sizes (one class), x sizes with a padded, an uneven and a three-pass
plan, tiles that span several ky and a partial last tile, a ligand too large
to stage in shared memory, many terms on a box grid, BF16 spectra.

Tolerance: FP32 sums and transforms of at most 256 points per axis; the parity
bar of the correlation grids, 1e-4 of the largest value (BF16-stored spectra:
2^-8 relative per spectrum value, so 8e-3).
"""
import numpy as np
import pytest

from oracle import fftdock_oracle as O

pytestmark = pytest.mark.gpu


def _inputs(dims, n_rec, n_lig, seed):
    rng = np.random.default_rng(seed)
    half = 0.5 * 1.2 * np.array(dims)
    rec = rng.uniform(-0.9, 0.9, (n_rec, 3)) * half
    lig = rng.uniform(-0.33, 0.33, (n_lig, 3)) * half.min()
    return rec, lig, rng


def _check(s, geom, rg, w, lig, tol, n=2):
    from proddl2_gb300 import synth
    rs = O.receptor_spectra(rg)
    rots = synth.quaternion_rotations(n, 11)
    res = s.scan(rots)
    for i, rot in enumerate(rots):
        cells, ok = O.bin_ligand(geom, rot, lig)
        assert ok
        corr = O.correlate(rs, O.ligand_grids(geom, cells, w))
        got = s.correlation_grid(rot)
        assert np.abs(got - corr).max() <= tol * np.abs(corr).max()
        cell, _, score = res.rotation(i)
        for c, sc in zip(cell, score):
            e = O.direct_score(rg, cells, w, c)
            assert abs(e - sc) <= 1e-9 * max(1.0, abs(e))


GRIDS = [(11, 15, 20), (13, 9, 25), (16, 16, 16), (24, 24, 24), (48, 48, 48), (64, 64, 64), (80, 80, 80), (96, 96, 96),
         (125, 20, 14), (98, 26, 30), (121, 10, 12), (90, 24, 66), (256, 12, 256), (250, 14, 9)]


@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("terms", ["shape", "lj_comp", "lj_avg"])
def test_one_term_and_paired(dims, terms):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rec, lig, rng = _inputs(dims, 60, 21, sum(dims))
    geom = O.Geometry.centred(1.2, dims)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    with FFTScan(ScanConfig(grid_step=1.2, term_set=terms, peaks_per_rot=4, lj_cut=7.0, **kw)) as s:
        if terms == "shape":
            rg = O.receptor_terms(geom, rec, None, O.TermParams(term_set=O.TERMS_SHAPE))
            w = np.ones((len(lig), 1))
            s.set_receptor(rec)
            s.set_ligand(lig)
        else:
            sr, er, ar = synth.lj_params(len(rec), 3)
            sl, el, _ = synth.lj_params(len(lig), 4)
            ts = O.TERMS_LJ_COMP if terms == "lj_comp" else O.TERMS_LJ_AVG
            lj = O.LjParams(sr, er, ar, sl, el, mix=1, cut=7.0)
            rg, w = O.lj_receptor_terms(geom, rec, lj, ts), O.lj_ligand_weights(lj, ts)
            s.set_pair_lj(rec, sr, er, ar, lig, sl, el)
        _check(s, geom, rg, w, lig, 1e-4)


@pytest.mark.parametrize("dims,terms,n_lig", [((48, 48, 48), "shape", 32768), ((128, 128, 128), "lj_comp", 9000),
                                              ((90, 66, 70), "lj_comp", 9000)])
def test_entries_beyond_shared_memory(dims, terms, n_lig):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rec, lig, rng = _inputs(dims, 60, n_lig, 5)
    geom = O.Geometry.centred(1.2, dims)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    with FFTScan(ScanConfig(grid_step=1.2, term_set=terms, peaks_per_rot=2, lj_cut=7.0, **kw)) as s:
        if terms == "shape":
            rg = O.receptor_terms(geom, rec, None, O.TermParams(term_set=O.TERMS_SHAPE))
            w = np.ones((len(lig), 1))
            s.set_receptor(rec)
            s.set_ligand(lig)
        else:
            sr, er, ar = synth.lj_params(len(rec), 3)
            sl, el, _ = synth.lj_params(len(lig), 4)
            lj = O.LjParams(sr, er, ar, sl, el, mix=1, cut=7.0)
            rg, w = O.lj_receptor_terms(geom, rec, lj, O.TERMS_LJ_COMP), O.lj_ligand_weights(lj, O.TERMS_LJ_COMP)
            s.set_pair_lj(rec, sr, er, ar, lig, sl, el)
        _check(s, geom, rg, w, lig, 1e-4, n=1)


@pytest.mark.parametrize("dims,k", [((33, 26, 21), 2), ((125, 12, 10), 5)])
def test_many_terms_on_a_box(dims, k):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rec, lig, rng = _inputs(dims, 60, 21, 9)
    rt, lt = rng.integers(0, k, len(rec)).astype(np.int32), rng.integers(0, k, len(lig)).astype(np.int32)
    ace = synth.ace_matrix(k, 2)
    geom = O.Geometry.centred(1.2, dims)
    tp = O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=ace, n_types=k)
    rg, w = O.receptor_terms(geom, rec, rt, tp), O.ligand_term_weights(lt, tp)
    with FFTScan(ScanConfig(grid_dims=dims, grid_step=1.2, term_set="shape_ace", n_types=k, ace_matrix=ace,
                            pencil_mode="fft")) as s:
        s.set_receptor(rec, rt)
        s.set_ligand(lig, lt)
        _check(s, geom, rg, w, lig, 1e-4)


@pytest.mark.parametrize("n", [32, 80])
def test_bf16_spectra(n):
    from proddl2_gb300 import FFTScan, ScanConfig
    rec, lig, rng = _inputs((n, n, n), 80, 30, n)
    geom = O.Geometry.centred(1.2, n)
    rg = O.receptor_terms(geom, rec, None, O.TermParams(term_set=O.TERMS_SHAPE))
    with FFTScan(ScanConfig(grid_n=n, grid_step=1.2, term_set="shape", precision="bf16")) as s:
        s.set_receptor(rec)
        s.set_ligand(lig)
        _check(s, geom, rg, np.ones((len(lig), 1)), lig, 8e-3)
