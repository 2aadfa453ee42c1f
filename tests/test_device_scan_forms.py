"""Device scans of whole groups of 128 rotations and a tail (both pencil forms
under AUTO) on a caller's stream: the host scan's peaks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 32, 32), (50, 44, 36)])
@pytest.mark.parametrize("n", [128, 134, 300])
def test_device_scan_equals_host_scan(dims, n):
    import torch
    from proddl2_gb300 import FFTScan, ScanConfig, _lib, synth
    rng = np.random.default_rng(n)
    half = 0.6 * min(dims)
    ace = synth.ace_matrix(18, 5)
    rots = synth.quaternion_rotations(n, 9)
    kw = dict(grid_n=dims[0]) if len(set(dims)) == 1 else dict(grid_dims=dims)
    with FFTScan(ScanConfig(term_set="shape_ace", ace_matrix=ace, peaks_per_rot=4, **kw)) as s:
        s.set_receptor(rng.uniform(-0.9 * half, 0.9 * half, (90, 3)), rng.integers(0, 18, 90).astype(np.int32))
        s.set_ligand(rng.uniform(-0.3 * half, 0.3 * half, (25, 3)), rng.integers(0, 18, 25).astype(np.int32))
        assert s.info()["pencil_path"] == "tensor"
        host = s.scan(rots, first_rot_id=3)
        d_rot = torch.tensor(np.asarray(rots).reshape(n, 9), dtype=torch.float64, device="cuda")
        d_peaks = torch.zeros(n * 4 * _lib.peak_dtype().itemsize, dtype=torch.uint8, device="cuda")
        d_np = torch.zeros(n, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        s.scan_device(d_rot.data_ptr(), n, d_peaks.data_ptr(), d_np.data_ptr(), first_rot_id=3,
                      stream_ptr=stream.cuda_stream)
        stream.synchronize()
        assert np.array_equal(d_np.cpu().numpy(), host.n_peaks)
        assert np.array_equal(d_peaks.cpu().numpy().view(_lib.peak_dtype()).reshape(n, 4), host.peaks)
