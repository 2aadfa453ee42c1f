"""Contexts of different grids in different threads: separate contexts are
independent, so set-up and scans of one go on beside those of another whose
kernels need more or less shared memory (the limit a kernel may ask for belongs
to the function, not to the context)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (dims, term set, pencil form) of the two contexts
PAIRS = [
    (((8, 8, 8), "shape", "auto"), ((16, 12, 144), "shape", "auto")),
    (((8, 8, 8), "shape_ace", "tensor"), ((12, 16, 144), "shape_ace", "tensor")),
    (((8, 8, 8), "lj_comp", "auto"), ((144, 12, 16), "lj_comp", "auto")),
    (((16, 16, 16), "shape_ace", "fft"), ((64, 64, 64), "shape_ace", "fft")),
]


def _context(dims, terms, mode):
    from proddl2_gb300 import FFTScan, ScanConfig
    rng = np.random.default_rng(sum(dims))
    ace = rng.normal(size=(18, 18))
    half = 0.6 * min(dims)
    rec, lig = rng.uniform(-half, half, (40, 3)), rng.uniform(-0.4 * half, 0.4 * half, (12, 3))
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    s = FFTScan(ScanConfig(grid_step=1.2, term_set=terms, ace_matrix=ace + ace.T, peaks_per_rot=2, rot_batch=16,
                           pencil_mode=mode, **kw))
    rt, lt = rng.integers(0, 18, 40).astype(np.int32), rng.integers(0, 18, 12).astype(np.int32)

    def set_pair():
        if terms == "lj_comp":
            s.set_pair_lj(rec, np.full(40, 3.4), np.full(40, 0.2), np.full(40, 0.4), lig, np.full(12, 3.3),
                          np.full(12, 0.3))
        else:
            s.set_receptor(rec, rt)
            s.set_ligand(lig, lt)
    return s, set_pair


@pytest.mark.parametrize("pair", PAIRS, ids=lambda p: "%s-%s" % (p[0][1], p[0][2]))
def test_two_grids_in_four_threads(pair):
    from proddl2_gb300 import synth
    rots = synth.quaternion_rotations(3, 4)
    runs, failures = [], []
    for spec in pair + pair:
        s, set_pair = _context(*spec)
        set_pair()
        runs.append((s, set_pair, s.scan(rots, raise_out_of_grid=False)))

    def work(s, set_pair, alone):
        try:
            for i in range(2000):
                set_pair()
                if i % 50 == 0:
                    r = s.scan(rots, raise_out_of_grid=False)
                    assert np.array_equal(r.n_peaks, alone.n_peaks) and np.array_equal(r.peaks, alone.peaks)
        except Exception as e:  # noqa: BLE001 (reported below)
            failures.append(repr(e))
    threads = [threading.Thread(target=work, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, _, _ in runs:
        s.close()
    assert not failures, failures
