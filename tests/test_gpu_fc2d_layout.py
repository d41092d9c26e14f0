"""The 2D solver's layout, built on the device: whether the block pattern is
symmetric (rows on both sides of the length up to which the device looks) decides
between dataflow and colours, and the sweeps are the oracle's either way, also
when one context takes problems of other sizes in turn."""
import numpy as np
import pytest

from test_gpu_fc2d import _ctx, _order, sn  # noqa: F401

pytestmark = pytest.mark.gpu


def _hub(O, nc, rows, change, seed=1):
    """A chain whose first contact is tied to so many others that its row has
    `rows` blocks; `change` drops one block of the pattern or doubles it."""
    g = np.random.default_rng(seed)
    adj = {i: {i} for i in range(nc)}
    for i, j in [(i, i + 1) for i in range(nc - 1)] + [(0, 2 * k) for k in range(1, rows - 1)]:
        adj[i].add(j)
        adj[j].add(i)
    assert len(adj[0]) == rows
    cols = [list(g.permutation(sorted(adj[i]))) for i in range(nc)]  # in any order
    if change == "drop":
        cols[7].remove(8)
    elif change == "double":
        cols[7].append(8)
    rowptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    colidx = np.concatenate(cols).astype(np.int64)
    blocks = 0.05 * g.standard_normal((len(colidx), 4))
    blocks[colidx == np.repeat(np.arange(nc), np.diff(rowptr))] = [2.0, 0.1, 0.1, 1.5]
    return O.Problem(nc, rowptr, colidx, blocks, g.standard_normal(2 * nc), g.uniform(0.1, 0.9, nc), 2)


def _check(sn, ctx, P):  # noqa: F811
    import oracle as O
    _, colour = ctx.colours()
    ctx.set_r(np.zeros(2 * P.nc))
    ctx.set_precision(1)
    ctx.solve(0.0, 5)
    ref = O.fc2d_nsgs_port(P, tol=0.0, maxiter=5, order=_order(colour))
    np.testing.assert_array_equal(ctx.get_r_u()[0], ref.r)
    ctx.set_precision(0, 1e-30, 1 << 20)
    ctx.set_r(np.zeros(2 * P.nc))
    ctx.solve(1e-300, 5)
    s32, s64 = ctx.last_sweeps()
    want = O.fc2d_sweeps_f32_port(P, np.zeros(2 * P.nc), s32, order=_order(colour))
    if s64:
        want = O.fc2d_nsgs_port(P, r0=want, tol=0.0, maxiter=s64, order=_order(colour)).r
    np.testing.assert_array_equal(ctx.get_r_u()[0], want)


@pytest.mark.parametrize("nc,rows", [(300, 20), (300, 64), (300, 100), (2698, 52), (2698, 53), (3000, 64), (3000, 65),
                                     (3000, 100)])
@pytest.mark.parametrize("change", ["none", "drop", "double"])
def test_pattern(sn, nc, rows, change):  # noqa: F811
    """Looked at by the device from 8,192 blocks on, with rows of up to 64."""
    import oracle as O
    P = _hub(O, nc, rows, change)
    ctx = _ctx(sn, P)
    ctx.set_precision(0)  # by colours FP32 sweeps of so few contacts have a cluster
    assert (ctx.launch_shape()[0] < 0) == (change == "none")  # a grid: dataflow
    _check(sn, ctx, P)
    ctx.close()


def test_problems_in_turn(sn):  # noqa: F811
    """Larger, a little smaller, much smaller, larger again, in one context."""
    import oracle as O
    ctx = None
    for nc, rows, change in [(300, 40, "none"), (3000, 70, "none"), (2900, 30, "drop"), (40, 10, "none"),
                             (2000, 64, "none")]:
        P = _hub(O, nc, rows, change, seed=nc)
        if ctx is None:
            ctx = _ctx(sn, P)
        else:
            rc = sn.lib().fc2dgpu_ctx_set_problem(ctx.ctx, nc, P.rowptr, P.colidx, P.blocks.reshape(-1), P.q, P.mu, 0)
            assert rc == 0, sn.last_error()
            ctx.nc = nc
        _check(sn, ctx, P)
    ctx.close()


@pytest.mark.parametrize("copies,shape", [(9, (1, 32, 1)), (9, (1, 64, 2)), (9, (2, 32, 2)), (9, (16, 32, 1)),
                                          (1, (1, 32, 0)), (1, (1, 64, 0)), (4, (1, 128, 2)), (4, (1, 160, 1)),
                                          (1100, (-1, 32, 0))])
def test_more_contacts_than_threads(sn, copies, shape):  # noqa: F811
    """Requested launches on both sides of the line from which FP64 contacts are
    one lane's (four a thread; 131 contacts in the largest colour of a copy)."""
    import oracle as O
    from test_fc2d_oracle import load_fc2d, tiled2d
    P = tiled2d(load_fc2d("fc2d_FrictionContactProblem00727")[0], copies, 4)
    ctx = _ctx(sn, P)
    _, colour = ctx.colours()
    ctx.set_launch(*shape)
    res = ctx.solve(0.0, 6)
    r, u = ctx.get_r_u()
    ctx.close()
    ref = O.fc2d_nsgs_port(P, tol=0.0, maxiter=6, order=_order(colour))
    np.testing.assert_array_equal(r, ref.r)
    np.testing.assert_array_equal(u, ref.u)
    assert res["error"] == pytest.approx(ref.error, rel=1e-12, abs=0)


@pytest.mark.parametrize("problem,copies", [("FrictionContactProblem00727", 9), ("FrictionContactProblem00071", 1)])
def test_launch_shape_is_that_of_the_precision(sn, problem, copies):  # noqa: F811
    """By colours: FP64 goes to a grid above 1,000 contacts a colour and takes two
    threads a contact, FP32 has a cluster and one."""
    from test_fc2d_oracle import load_fc2d, tiled2d
    from test_gpu_fc2d_shapes import _one_sided
    P = _one_sided(tiled2d(load_fc2d("fc2d_" + problem)[0], copies, 4), 0)
    ctx = _ctx(sn, P)
    fp64 = ctx.launch_shape()
    ctx.set_precision(0)
    fp32 = ctx.launch_shape()
    ctx.close()
    if copies > 1:
        assert fp64[0] < 0 < fp32[0]
    else:
        assert fp64 == (1, 2 * fp32[1], 2) and fp32[0] == 1
