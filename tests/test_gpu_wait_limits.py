"""Device waits with a limit of one poll: every form of the sweeps gives up with
an error, and with the default limit the context solves as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gives_up_and_recovers(gpu, solve):
    want = solve()
    old = gpu.spin_limit(1)
    try:
        with pytest.raises(RuntimeError):
            solve()
    finally:
        gpu.spin_limit(old)
    np.testing.assert_array_equal(solve(), want)


def _batch(gpu, precision):
    from siconos_gb300.scene import lattice
    gpu.load_batch([lattice(*d, seed=40 + k) for k, d in enumerate([(20, 19, 9), (3, 3, 2), (12, 11, 6)])])

    def solve():
        gpu.zero_r()
        gpu.solve_batch(tol=1e-300, max_iter=12, precision=precision, fp32_only=1 - precision)
        return gpu.get()[0]

    return solve


@pytest.mark.parametrize("flow", [True, False], ids=["dataflow", "colours"])
def test_batch_fp32(gpu, flow):
    """The limit set after the batch's launches were recorded counts too."""
    gpu.flow(flow)
    try:
        _gives_up_and_recovers(gpu, _batch(gpu, 0))
    finally:
        gpu.flow(True)


@pytest.mark.parametrize("dims", [(3, 3, 2), (19, 18, 11)])
def test_fp64(gpu, dims):
    """From one contact a unit to several; rows of more than one round of slots."""
    from siconos_gb300.scene import lattice
    gpu.load(lattice(*dims, seed=2))

    def solve():
        gpu.zero_r()
        gpu.solve(tol=1e-300, max_iter=12, precision=1, lanes=1)
        return gpu.get()[0]

    _gives_up_and_recovers(gpu, solve)


def test_batch_fp64(gpu):
    _gives_up_and_recovers(gpu, _batch(gpu, 1))


def _context_recovers(ctx, n, solve):
    def run():
        ctx.set_r(np.zeros(n))
        solve()
        return ctx.get_r_u()[0]

    want = run()
    ctx.spin_limit(1)
    with pytest.raises(RuntimeError, match="poll limit"):
        run()
    ctx.spin_limit(0)
    np.testing.assert_array_equal(run(), want)
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("copies", [1, 100])
def test_rolling(built_lib, copies, precision):
    import siconos_gb300.numerics as sn
    from test_gpu_rfc3d import _ctx
    from test_rfc3d_oracle import load_rfc3d, tiled
    T = tiled(load_rfc3d("rfc3d_rockfall_21_54029")[0], copies, 7)
    ctx = _ctx(sn, T)
    ctx.set_precision(precision)
    _context_recovers(ctx, 5 * T.nc, lambda: ctx.solve(0.0, 6))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("problem,copies", [("FrictionContactProblem00727", 1),
                                            ("fc2d_granularflowonwall_07002_00801", 4)])
def test_2d(built_lib, problem, copies, precision):
    import siconos_gb300.numerics as sn
    from test_fc2d_oracle import load_fc2d, tiled2d
    from test_gpu_fc2d import _ctx
    P = tiled2d(load_fc2d("fc2d_" + problem)[0], copies, 4)
    ctx = _ctx(sn, P)
    ctx.set_precision(precision, 1e-30, 1 << 20)
    _context_recovers(ctx, 2 * P.nc, lambda: ctx.solve(1e-300, 8))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim", [2, 5])
def test_grid_barriers(built_lib, dim, precision):
    """By colours (a pattern that is not symmetric) on a grid: the barriers
    between colours, and that of an error evaluation."""
    import siconos_gb300.numerics as sn
    if dim == 2:
        from test_fc2d_oracle import load_fc2d, tiled2d
        from test_gpu_fc2d import _ctx
        from test_gpu_fc2d_shapes import _one_sided
        T = _one_sided(tiled2d(load_fc2d("fc2d_fc2d_granularflowonwall_07002_00801")[0], 4, 4), 0)
    else:
        from test_gpu_rfc3d import _ctx
        from test_gpu_rolling_lanes import _one_sided
        from test_rfc3d_oracle import load_rfc3d, tiled
        T = _one_sided(tiled(load_rfc3d("rfc3d_rockfall_21_54029")[0], 100, 7), 0)
    ctx = _ctx(sn, T)
    ctx.set_precision(precision, 1e-30, 1 << 20)
    error = ctx.compute_error(1.0)
    ctx.spin_limit(1)
    with pytest.raises(RuntimeError, match="poll limit"):
        ctx.compute_error(1.0)
    ctx.spin_limit(0)
    assert ctx.compute_error(1.0) == error
    _context_recovers(ctx, dim * T.nc, lambda: ctx.solve(1e-300, 6))
