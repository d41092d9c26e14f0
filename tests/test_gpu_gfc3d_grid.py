"""Global solver: r, u and v bit for bit with the oracle from one block to a
block on every SM and more slabs than blocks, after even and odd iteration
counts (the iterate's two buffers), and the error of the iterate kept."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_RTOL = 1e-12  # sums of squares of FP64 terms in another order


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 2, 1), (3, 3, 2), (6, 6, 4), (10, 9, 9), (10, 10, 9), (18, 17, 16)])
@pytest.mark.parametrize("sweeps", [1, 4, 7])
def test_blocks_and_buffers(gpu, dims, sweeps):
    import oracle as O
    import siconos_gb300.numerics as sn
    P = O.lattice_global(*dims, seed=5)
    ref = O.gfc3d_nsgs_port(P, tol=0.0, maxiter=sweeps, trace_cap=sweeps)
    more = O.gfc3d_nsgs_port(P, r0=ref.r, v0=ref.v, tol=0.0, maxiter=3)
    c = sn.Gfc3dContext.from_problem(P)
    try:
        res = c.solve(0.0, sweeps)
        r, u, v = c.get()
        tr = c.trace(sweeps)
        err = c.compute_error()
        kept = c.get()
        res2 = c.solve(0.0, 3)
        r2, u2, v2 = c.get()
    finally:
        c.close()
    assert res["iterations"] == ref.iterations and res2["iterations"] == more.iterations
    for got, want in ((r, ref.r), (u, ref.u), (v, ref.v), (kept[0], ref.r), (kept[1], ref.u), (kept[2], ref.v),
                      (r2, more.r), (u2, more.u), (v2, more.v)):
        assert np.array_equal(got, want)
    np.testing.assert_allclose(tr, ref.trace, rtol=ERR_RTOL)
    np.testing.assert_allclose([res["error"], err, res2["error"]], [ref.error, ref.error, more.error], rtol=ERR_RTOL)
