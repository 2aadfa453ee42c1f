"""The plane stage's CTA sizes: planes on both sides of the box grids' line
between 64 and 256 threads, the smallest ones and the single-warp cubic edge.
The 16 kept cells are exactly the smallest of the grid the stage returns, ties by
offset, ordinary planes and flat ones (far more ties than the candidate list
holds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(8, 8, 8), (9, 8, 9), (16, 16, 16), (8, 20, 36), (8, 22, 36), (10, 20, 39), (9, 21, 39), (8, 72, 72), (8, 78, 70),
        (10, 75, 70), (9, 75, 77), (24, 24, 24)]


@pytest.mark.parametrize("mode", ["fft", "tensor"])
@pytest.mark.parametrize("dims", DIMS)
def test_candidates_are_the_grid_s_smallest(dims, mode):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    rng = np.random.default_rng(sum(dims))
    half = 0.6 * min(dims)
    ace = synth.ace_matrix(18, 5)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 and dims[0] != 8 else dict(grid_dims=dims)
    rots = synth.quaternion_rotations(5, 7)
    with FFTScan(ScanConfig(term_set="shape_ace", ace_matrix=ace, peaks_per_rot=16, pencil_mode=mode, **kw)) as s:
        lig = rng.uniform(-0.3 * half, 0.3 * half, (12, 3)), rng.integers(0, 18, 12).astype(np.int32)
        for n_rec in (60, 0):  # no receptor: flat planes
            rec = rng.uniform(-half, half, (n_rec, 3)), rng.integers(0, 18, n_rec).astype(np.int32)
            s.set_receptor(*rec)
            s.set_ligand(*lig)
            value, offset = s.candidates(rots)
            for r, v, o in zip(rots, value, offset):
                grid = s.correlation_grid(r).reshape(-1)
                best = np.argsort(grid, kind="stable")[:16]
                assert np.array_equal(o, best) and np.array_equal(v, grid[best])
