"""The rolling solver's FP64 sweeps run six contacts a warp, five lanes each:
copies of the 21-contact rockfall problem whose colours fill one warp, one
block, several small blocks, and leave remainders of a warp, bit for bit the
oracle's sweeps in colour order."""
import numpy as np
import pytest

from test_gpu_rfc3d import _ctx, _order, sn  # noqa: F401
from test_rfc3d_oracle import load_rfc3d, tiled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 2, 3, 25, 61])
def test_bit_exact(sn, copies):  # noqa: F811
    import oracle as O
    P, _ = load_rfc3d("rfc3d_rockfall_21_54029")
    T = tiled(P, copies, 7)
    ctx = _ctx(sn, T)
    _, colour = ctx.colours()
    res = ctx.solve(0.0, 12)
    r, u = ctx.get_r_u()
    ctx.close()
    ref = O.rfc3d_nsgs_port(T, tol=0.0, maxiter=12, order=_order(colour))
    np.testing.assert_array_equal(r, ref.r)
    np.testing.assert_array_equal(u, ref.u)
    assert res["error"] == pytest.approx(ref.error, rel=1e-12, abs=0)
