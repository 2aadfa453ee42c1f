"""Box grids whose plane stage takes just under 48 KB of dynamic shared memory
beside its static arrays, as a process's first scan (the opt-in is kept per
function, so an earlier larger grid would hide a missing one)."""
import json
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import json, sys
import numpy as np
from proddl2_gb300 import FFTScan, ScanConfig, synth
dims, n = json.loads(sys.argv[1]), int(sys.argv[2])
rng = np.random.default_rng(1)
rec, lig = rng.uniform(-20, 20, (50, 3)), rng.uniform(-6, 6, (20, 3))
ace = rng.normal(size=(18, 18))
with FFTScan(ScanConfig(grid_dims=tuple(dims), term_set="shape_ace", ace_matrix=ace + ace.T, peaks_per_rot=4)) as s:
    s.set_receptor(rec, rng.integers(0, 18, 50).astype(np.int32))
    s.set_ligand(lig, rng.integers(0, 18, 20).astype(np.int32))
    print(json.dumps(s.scan(synth.quaternion_rotations(n, 2)).n_peaks.tolist()))
"""


@pytest.mark.parametrize("dims", [(40, 54, 208), (40, 55, 196), (36, 42, 256), (40, 100, 112)])
@pytest.mark.parametrize("n_rot", [3, 40])
def test_first_scan_of_a_process(dims, n_rot):
    out = subprocess.run([sys.executable, "-c", CODE, json.dumps(dims), str(n_rot)], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    assert json.loads(out.stdout.splitlines()[-1]) == [4] * n_rot
