"""The proposal's GEMM tiles and gathers: a sample's prediction does not depend,
bit for bit, on how many are predicted with it (each output sums its products in
the same order under every tile), and gradients of batch sizes beside the tile
edges equal the sum of the single samples' gradients up to the roundings to BF16
(2e-3 relative per tensor, the bar of the gradient test; f2 6e-3)."""
import numpy as np
import pytest

from oracle import proposal_oracle as PO
from test_proposal import TENSORS, _rand_rot, _tensor_slices, _toy_samples

pytestmark = pytest.mark.gpu


def test_predictions_do_not_depend_on_the_batch():
    from proddl2_gb300.proposal import Proposal
    pairs, _, _, _, _ = _toy_samples(8, n_pairs=1, per_pair=1)
    rots = _rand_rot(np.random.default_rng(3), 4200)
    with Proposal(seed=4) as p:
        pid = p.add_pair(pairs[0][0], desc=pairs[0][2])
        full = p.predict(pid, rots)
        for n in (1, 2, 7, 31, 33, 63, 65, 129, 300, 1000, 2433, 4096, 4097):
            assert np.array_equal(p.predict(pid, rots[:n]), full[:n]), n
            assert np.array_equal(p.predict(pid, rots[-n:]), full[-n:]), n


@pytest.mark.parametrize("n", [1, 5, 31, 33, 65, 130])
def test_gradients_beside_tile_edges(n):
    from proddl2_gb300.proposal import Proposal
    pairs, samples, targets, ids, rots = _toy_samples(9, n_pairs=1, per_pair=n)
    with Proposal(seed=12) as p:
        pid = p.add_pair(pairs[0][0], desc=pairs[0][2])
        params = p.params.astype(np.float64)
        g, loss = p.gradients(np.full(n, pid), rots, targets)
    ref_loss, ref_g, _ = PO.forward_backward(params, samples, targets, bf=True)
    assert abs(loss - ref_loss) <= 2e-3 * max(1.0, ref_loss)
    for name, sl in _tensor_slices().items():
        r = np.linalg.norm(g[sl] - ref_g[sl]) / np.linalg.norm(ref_g[sl])
        assert r <= (6e-3 if name == "f2" else 2e-3), (name, r)


def test_cells_on_and_beside_the_boundaries():
    """Atoms on cell boundaries, within an FP32 rounding of them and outside the
    cube land in the oracle's FP64 cells."""
    from proddl2_gb300.proposal import Proposal
    base = np.array([[-1.0, -0.5, 0.25], [1.0, 0.125, -0.375], [0.0, 0.75, -1.0], [0.5, -0.25, 0.875]]) * 16.0
    eps = np.array([0.0, 1e-15, -1e-15, 1e-9, -1e-9, 1e-6, -1e-6, 1e-5, -1e-5])
    lig = (base[None] * (1 + eps[:, None, None])).reshape(-1, 3)
    R = [np.eye(3), np.array([[0.0, -1, 0], [1, 0, 0], [0, 0, 1]]), *_rand_rot(np.random.default_rng(1), 4)]
    desc = np.zeros(PO.DESC if hasattr(PO, "DESC") else 128, dtype=np.float32)
    with Proposal(seed=6) as p:
        pid = p.add_pair(lig, desc=desc)
        params = p.params.astype(np.float64)
        got = p.predict(pid, np.array(R))
    samples = [(lig, PO.half_width(lig), r, desc) for r in R]
    _, _, ref = PO.forward_backward(params, samples, np.zeros(len(R)), bf=True)
    assert np.allclose(got, ref, rtol=2e-3, atol=2e-3 * np.abs(ref).max())
