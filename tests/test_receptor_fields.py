"""The receptor set-up where its warps' runs and lists can go wrong: rows
shorter and longer than 32 cells, cutoffs from below a cell to beyond the grid,
crowded atoms (many listed per run), atoms outside the grid, 1 and 32 types, a
context reused for receptors of different sizes.

Tolerance: FP64 sums in the oracle's order up to the order of the bins: 1e-12
relative to the largest value (the fields' own parity bar).
"""
import numpy as np
import pytest

from oracle import fftdock_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,step,cut,n_rec,types", [
    ((12, 10, 9), 1.2, 6.0, 40, 18), ((16, 9, 33), 1.2, 6.0, 200, 18), ((9, 11, 100), 1.2, 0.7, 300, 3),
    ((10, 12, 64), 0.5, 12.0, 60, 18), ((24, 24, 24), 1.2, 6.0, 3000, 32), ((14, 13, 50), 2.5, 3.0, 1, 1)])
def test_desolvation_terms(dims, step, cut, n_rec, types):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rng = np.random.default_rng(sum(dims))
    ace = synth.ace_matrix(types, 3)
    geom = O.Geometry.centred(step, dims)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    tp = O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=ace, n_types=types, ace_cut=cut)
    with FFTScan(ScanConfig(grid_step=step, term_set="shape_ace", n_types=types, ace_matrix=ace, ace_cut=cut,
                            **kw)) as s:
        for n in (n_rec, max(1, n_rec // 3), n_rec + 17):  # the kept work memory grows and is reused
            rec = rng.uniform(-1.2, 1.2, (n, 3)) * 0.5 * step * np.array(dims)
            rt = rng.integers(0, types, n).astype(np.int32)
            s.set_receptor(rec, rt)
            rg = O.receptor_terms(geom, rec, rt, tp)
            for t in range(0, types, max(1, types // 4)):
                assert np.abs(s.receptor_grid(t) - rg[t]).max() <= 1e-12 * max(1.0, np.abs(rg[t]).max())


@pytest.mark.parametrize("terms", ["lj_comp", "lj_avg"])
@pytest.mark.parametrize("dims,cut,n_rec", [((12, 10, 9), 9.0, 60), ((10, 9, 66), 30.0, 40), ((24, 24, 24), 9.0, 900)])
def test_lj_fields(terms, dims, cut, n_rec):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rng = np.random.default_rng(n_rec)
    half = 0.6 * np.array(dims)
    rec, lig = rng.uniform(-1.1, 1.1, (n_rec, 3)) * half, rng.uniform(-0.3, 0.3, (5, 3)) * half.min()
    geom = O.Geometry.centred(1.2, dims)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    ts = O.TERMS_LJ_COMP if terms == "lj_comp" else O.TERMS_LJ_AVG
    sr, er, ar = synth.lj_params(n_rec, 3)
    sl, el, _ = synth.lj_params(len(lig), 4)
    rg = O.lj_receptor_terms(geom, rec, O.LjParams(sr, er, ar, sl, el, mix=1, cut=cut), ts)
    with FFTScan(ScanConfig(grid_step=1.2, term_set=terms, lj_cut=cut, **kw)) as s:
        s.set_pair_lj(rec, sr, er, ar, lig, sl, el)
        for t in range(len(rg)):
            assert np.abs(s.receptor_grid(t) - rg[t]).max() <= 1e-12 * max(1.0, np.abs(rg[t]).max())
