"""Receptor set-up keeps at most 512 MiB of half spectra per context: larger
term sets are transformed a chunk of terms at a time, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(dims, n_types, **kw):
    from proddl2_gb300 import FFTScan, ScanConfig
    rng = np.random.default_rng(sum(dims) + n_types)
    ace = rng.normal(size=(n_types, n_types))
    half = 0.6 * min(dims)
    grid = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    s = FFTScan(ScanConfig(term_set="shape_ace", n_types=n_types, ace_matrix=ace + ace.T, peaks_per_rot=16, **grid, **kw))
    rec = (rng.uniform(-0.6 * half, 0.6 * half, (800, 3)), rng.integers(0, n_types, 800).astype(np.int32))
    lig = (rng.uniform(-0.2 * half, 0.2 * half, (150, 3)), rng.integers(0, n_types, 150).astype(np.int32))
    return s, rec, lig


def test_work_memory_is_bounded():
    import torch
    s, rec, lig = _context((144, 144, 144), 32, rot_batch=4)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s.set_receptor(*rec)
    used = free - torch.cuda.mem_get_info()[0]
    s.close()
    # half spectra, the shape flags (4 bytes a cell) and the atoms
    assert used <= (512 << 20) + 4 * 144 ** 3 + (32 << 20), used


# terms in one chunk, just over one, two with a shorter last one
@pytest.mark.parametrize("dims,n_types,mode", [
    ((128, 128, 128), 31, "tensor"), ((128, 128, 128), 32, "tensor"), ((144, 144, 144), 23, "fft"),
    ((144, 144, 144), 32, "fft"), ((128, 120, 250), 19, "tensor"), ((128, 120, 250), 19, "fft")])
def test_chunks_of_terms(dims, n_types, mode):
    from proddl2_gb300 import synth
    s, rec, lig = _context(dims, n_types, pencil_mode=mode, rot_batch=8)
    s.set_receptor(*rec)
    s.set_ligand(*lig)
    rots = synth.quaternion_rotations(4, 9)
    value, offset = s.candidates(rots)      # FP32, from the spectra of all terms
    peaks = s.scan(rots).peaks              # FP64, from the term grids
    s.close()
    for v, o, p in zip(value, offset, peaks):
        exact = {(c[0] * dims[1] + c[1]) * dims[2] + c[2]: e for c, e in zip(p["cell"].astype(int), p["score"])}
        got = dict(zip(o.tolist(), v.tolist()))
        assert exact.keys() == got.keys()
        # FP32 values lie within 2e-4 of FP64 (relative to the largest); a wrong
        # term moves them by far more
        big = max(abs(e) for e in exact.values())
        assert all(abs(got[k] - exact[k]) <= 1e-3 * big for k in exact)
