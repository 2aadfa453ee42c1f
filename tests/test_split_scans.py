"""A rotation's peaks do not depend on the call it is scanned in: the parts of a
rotation set (ranges of ranks and tasks, which may run another pencil form than
the whole set) give the peaks of one scan of it, scores to the last bit, and so
does the pair list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(dims, seed):
    rng = np.random.default_rng([seed, *dims])
    half = 0.6 * min(dims)
    rec, rt = rng.uniform(-0.9 * half, 0.9 * half, (120, 3)), rng.integers(0, 18, 120).astype(np.int32)
    lig, lt = rng.uniform(-0.25 * half, 0.25 * half, (70, 3)), rng.integers(0, 18, 70).astype(np.int32)
    ace = rng.normal(size=(18, 18))
    return rec, rt, lig, lt, ace + ace.T


@pytest.mark.parametrize("dims", [(32, 32, 32), (80, 80, 80), (112, 112, 112), (40, 36, 30), (77, 50, 44), (44, 35, 50)])
@pytest.mark.parametrize("part", [1, 15, 32, 100])
def test_parts_of_a_rotation_set(dims, part):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rec, rt, lig, lt, ace = _pair(dims, 6)
    n = 205
    rots = synth.quaternion_rotations(n, 8)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    with FFTScan(ScanConfig(term_set="shape_ace", ace_matrix=ace, peaks_per_rot=4, **kw)) as s:
        s.set_receptor(rec, rt)
        s.set_ligand(lig, lt)
        whole = s.scan(rots)
        for a in range(0, n, part):
            r = s.scan(rots[a:a + part], first_rot_id=a)
            assert np.array_equal(r.n_peaks, whole.n_peaks[a:a + part])
            assert np.array_equal(r.peaks, whole.peaks[a:a + part]), a


# (grid edge, atoms, seed, rotations whose 16th FP32 candidate is a near tie that
# the two pencil forms settle differently)
NEAR_TIES = [(48, 700, 150, 2, [8269, 8881, 12454, 17719, 18861, 19352]),
             (80, 1500, 400, 2, [2212, 2873, 4580, 5960]),
             (128, 4000, 1500, 13, [726, 981, 986, 1433, 1913, 2290, 2467, 2703])]


@pytest.mark.parametrize("edge,n_rec,n_lig,seed,ties", NEAR_TIES)
@pytest.mark.parametrize("peaks", [8, 9, 16])
def test_parts_with_many_peaks(edge, n_rec, n_lig, seed, ties, peaks):
    # up to all 16 candidates of a rotation are kept: above 8 peaks the parts run
    # the whole set's form
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    pair = synth.make_pair(n_rec, n_lig, 20000 if edge == 48 else 9000 if edge == 80 else 4000, seed=seed)
    rots = np.asarray(pair.rotations).reshape(-1, 9)
    rots = np.concatenate([rots[ties], rots[:256 - len(ties)]])
    with FFTScan(ScanConfig(grid_n=edge, term_set="shape_ace", ace_matrix=pair.ace, peaks_per_rot=peaks)) as s:
        s.set_receptor(pair.receptor.xyz, pair.receptor.ace_type)
        s.set_ligand(pair.ligand.xyz, pair.ligand.ace_type)
        whole = s.scan(rots)
        for a in range(0, len(rots), 16):
            r = s.scan(rots[a:a + 16], first_rot_id=a)
            assert np.array_equal(r.n_peaks, whole.n_peaks[a:a + 16])
            assert np.array_equal(r.peaks, whole.peaks[a:a + 16]), a


def test_pair_list_against_single_scans():
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    from proddl2_gb300.pairs import PairInput, scan_pairs
    rots = synth.quaternion_rotations(144, 3)   # a tail of 16 after a whole group
    edges = [48, 80, 96, 112]
    mols = [_pair((n, n, n), 7) for n in edges]
    ace = mols[0][4]
    cfg = ScanConfig(term_set="shape_ace", ace_matrix=ace, peaks_per_rot=4)
    res, _ = scan_pairs(cfg, [PairInput(m[0], m[2], rots, m[1], m[3], grid_n=n) for m, n in zip(mols, edges)],
                        tune=False)
    for m, n, r in zip(mols, edges, res):
        with FFTScan(ScanConfig(grid_n=n, term_set="shape_ace", ace_matrix=ace, peaks_per_rot=4)) as s:
            s.set_receptor(m[0], m[1])
            s.set_ligand(m[2], m[3])
            one = s.scan(rots)
        assert np.array_equal(r.n_peaks, one.n_peaks) and np.array_equal(r.peaks, one.peaks), n
