"""Rounding of the FP32 transforms: the error of the correlation grids against
FP64 stays that of transforms whose scaled butterfly terms enter the last
additions as fused multiply-adds."""
import numpy as np
import pytest

from oracle import fftdock_oracle as O

pytestmark = pytest.mark.gpu

# rms errors with every such term contracted (FFT form, 18 terms, four rotations
# of these pairs); a product rounded on its own gives 1.05 times their mean
CONTRACTED = {(48, 160, 60): 1.150e-5, (64, 300, 200): 3.116e-5}


def test_rms_error_of_the_fft_form():
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    ratio = []
    for (n, n_rec, n_lig), expected in CONTRACTED.items():
        pair = synth.make_pair(n_rec, n_lig, 6, seed=5)
        geom = O.Geometry.centred(1.2, (n, n, n))
        rec = pair.receptor.xyz * min(1.0, 0.54 * n / np.abs(pair.receptor.xyz).max())
        lig = pair.ligand.xyz * min(1.0, 0.18 * n / np.linalg.norm(pair.ligand.xyz, axis=1).max())
        tp = O.TermParams(term_set=O.TERMS_SHAPE_ACE, ace_matrix=pair.ace)
        rs = O.receptor_spectra(O.receptor_terms(geom, rec, pair.receptor.ace_type, tp))
        w = O.ligand_term_weights(pair.ligand.ace_type, tp)
        err = []
        with FFTScan(ScanConfig(grid_n=n, term_set="shape_ace", ace_matrix=pair.ace, pencil_mode="fft")) as s:
            s.set_receptor(rec, pair.receptor.ace_type)
            s.set_ligand(lig, pair.ligand.ace_type)
            for rot in pair.rotations[:4]:
                cells, ok = O.bin_ligand(geom, rot, lig)
                assert ok
                err.append(s.correlation_grid(rot) - O.correlate(rs, O.ligand_grids(geom, cells, w)))
        ratio.append(np.sqrt(np.mean(np.square(err))) / expected)
    assert np.prod(ratio) ** (1 / len(ratio)) <= 1.03, ratio
