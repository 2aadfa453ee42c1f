"""AUTO with the tensor form selected: a call's last few rotations after whole
groups of 128 run the FFT form, the others the tensor form.  Each part is then
bit for bit what a context of that form gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,few", [((48, 48, 48), 32), ((112, 112, 112), 16), ((40, 36, 30), 16)])
@pytest.mark.parametrize("n", [1, 16, 17, 32, 33, 127, 128, 129, 144, 160, 161, 1024 + 7])
def test_parts_equal_the_two_forms(dims, few, n):
    from proddl2_gb300 import FFTScan, ScanConfig, synth
    if dims[0] > 48 and n > 161:
        pytest.skip("the group boundary is covered by the small grids")
    rng = np.random.default_rng(sum(dims))
    half = 0.6 * np.array(dims)
    rec, rt = rng.uniform(-0.9, 0.9, (100, 3)) * half, rng.integers(0, 18, 100).astype(np.int32)
    lig, lt = rng.uniform(-0.25, 0.25, (40, 3)) * half.min(), rng.integers(0, 18, 40).astype(np.int32)
    ace = rng.normal(size=(18, 18))
    rots = synth.quaternion_rotations(n, 5)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    tail = n % 128
    cut = n - tail if n > 128 and 0 < tail <= few else (0 if n <= few else n)
    got = {}
    for mode in ("auto", "tensor", "fft"):
        with FFTScan(ScanConfig(grid_step=1.2, term_set="shape_ace", ace_matrix=ace + ace.T, peaks_per_rot=4,
                                rot_batch=128, pencil_mode=mode, **kw)) as s:
            s.set_receptor(rec, rt)
            s.set_ligand(lig, lt)
            assert s.info()["pencil_path"] == ("fft" if mode == "fft" else "tensor")
            p = s.scan(rots).peaks
            got[mode] = (p["cell"], p["score"], p["rot_id"])
    for a, t, f in zip(got["auto"], got["tensor"], got["fft"]):
        assert np.array_equal(a[:cut], t[:cut])
        assert np.array_equal(a[cut:], f[cut:])
