"""fc3dgpu_compute_error_device on a column index out of range: the error is NaN
and the velocity that of the other blocks."""
import numpy as np
import pytest

from test_zz_no_alloc import _call, _reaction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-1, 70, 1 << 40])
@pytest.mark.parametrize("at", [0, 3, 4, 6])
def test_block_left_out(built_lib, bad, at):
    torch = pytest.importorskip("torch")
    nc, width = 70, 7  # rows of seven blocks: one round of four and a part of one
    g = np.random.default_rng(at)
    rowptr = width * np.arange(nc + 1, dtype=np.int64)
    colidx = np.stack([(i + np.arange(width)) % nc for i in range(nc)]).astype(np.int64)
    blocks = g.standard_normal((nc, width, 9))
    q, mu, r = g.standard_normal(3 * nc), np.full(nc, 0.5), _reaction(nc, 2)
    r[:3] = [1e6, -2e6, 3e6]  # contact 0's, which no bad column may stand for
    without = blocks.copy()
    without[40, at] = 0.0
    want = q.reshape(nc, 3) + np.einsum("iwcr,iwc->ir", without.reshape(nc, width, 3, 3), r.reshape(nc, 3)[colidx])
    colidx[40, at] = bad
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in
           dict(rowptr=rowptr, colidx=colidx.reshape(-1), blocks=blocks.reshape(-1), q=q, mu=mu, r=r).items()}
    vel = torch.zeros(3 * nc, dtype=torch.float64, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    assert _call(built_lib, nc, nc * width, dev, 1.0, vel, out, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert np.isnan(float(out))
    # rows of 21 products in two orders
    np.testing.assert_allclose(vel.cpu().numpy(), want.reshape(-1), rtol=0, atol=1e-14 * np.abs(want).max())
