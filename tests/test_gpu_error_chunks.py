"""fc3dgpu_compute_error_device at the edges of its chunks (64 contacts, three
threads a row; rows loaded four blocks at a time) and without a velocity
output, against the oracle."""
import numpy as np
import pytest

from test_zz_no_alloc import _call, _reaction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 2, 63, 64, 65, 127, 130, 3000])
def test_chunk_edges(built_lib, nc):
    torch = pytest.importorskip("torch")
    import oracle as O
    g = np.random.default_rng(nc)
    # banded rows of 1 to 9 blocks, the diagonal dominant
    cols = [np.unique(np.clip(i + g.integers(-6, 7, g.integers(0, 9)), 0, nc - 1).tolist() + [i]) for i in range(nc)]
    rowptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    colidx = np.concatenate(cols).astype(np.int64)
    blocks = 0.1 * g.standard_normal((len(colidx), 9))
    blocks[colidx == np.repeat(np.arange(nc), np.diff(rowptr))] += np.eye(3).reshape(-1)
    q, mu, r = g.standard_normal(3 * nc), g.uniform(0.1, 0.9, nc), _reaction(nc, 5)
    norm_q = float(np.linalg.norm(q))
    err, u = O.compute_error_port(O.Problem(nc, rowptr, colidx, blocks, q, mu), r)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in
           dict(rowptr=rowptr, colidx=colidx, blocks=blocks.reshape(-1), q=q, mu=mu, r=r).items()}
    vel = torch.full((3 * nc,), float("nan"), dtype=torch.float64, device="cuda")
    out = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    for velocity in (vel, None):
        assert _call(built_lib, nc, len(colidx), dev, norm_q, velocity, out,
                     torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        # FP64 sums of at most 30 terms a row and nc rows in another order
        assert abs(float(out) - err) <= 1e-12 * err
    scale = max(1.0, float(np.abs(u).max()))
    np.testing.assert_allclose(vel.cpu().numpy(), u, rtol=0, atol=1e-13 * scale)
