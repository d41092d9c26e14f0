"""The 2D sweeps' automatic launches over their range: FP64 on two threads a
contact in one block, in clusters and on the grid, rows longer than the eight
slots fetched together, and colours that end inside a warp; the FP64 sweeps
and the FP32 ones bit for bit the oracle's in colour order.  As dataflow (a
symmetric pattern): units from one contact to as many as a warp takes."""
import numpy as np
import pytest

from test_fc2d_oracle import load_fc2d, tiled2d
from test_gpu_fc2d import _ctx, _order, sn  # noqa: F401

pytestmark = pytest.mark.gpu


def _one_sided(P, drop):
    """P without its `drop`-th block off the diagonal (the transpose stays): the
    sweeps go by colours."""
    from dataclasses import replace
    row = np.repeat(np.arange(P.nc), np.diff(P.rowptr))
    keep = np.ones(len(row), bool)
    keep[np.flatnonzero(row != P.colidx)[drop]] = False
    return replace(P, rowptr=np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=P.nc))]),
                   colidx=P.colidx[keep], blocks=P.blocks[keep])


def _dense_rows(O, nc, seed):
    """A chain with every contact also tied to one of a few hubs (rows of up
    to nc / 4 blocks)."""
    g = np.random.default_rng(seed)
    adj = {i: {i} for i in range(nc)}
    for i in range(nc):
        for j in (i - 1, i % 4):
            if 0 <= j != i:
                adj[i].add(j)
                adj[j].add(i)
    rowptr = np.concatenate([[0], np.cumsum([len(adj[i]) for i in range(nc)])]).astype(np.int64)
    colidx = np.concatenate([sorted(adj[i]) for i in range(nc)]).astype(np.int64)
    blocks = 0.05 * g.standard_normal((len(colidx), 4))
    blocks[colidx == np.repeat(np.arange(nc), np.diff(rowptr))] = [2.0, 0.1, 0.1, 1.5]
    return O.Problem(nc, rowptr, colidx, blocks, g.standard_normal(2 * nc), g.uniform(0.1, 0.9, nc), 2)


@pytest.mark.parametrize("problem,copies", [("FrictionContactProblem00031", 1), ("FrictionContactProblem00727", 1),
                                            ("FrictionContactProblem00727", 9),
                                            ("fc2d_granularflowonwall_07002_00801", 1),
                                            ("fc2d_granularflowonwall_07002_00801", 10), ("dense", 90),
                                            ("dense", 700)])
@pytest.mark.parametrize("one_sided", [False, True])
def test_sweeps_bit_exact(sn, problem, copies, one_sided):  # noqa: F811
    import oracle as O
    P = _dense_rows(O, copies, 3) if problem == "dense" else tiled2d(load_fc2d("fc2d_" + problem)[0], copies, 4)
    if one_sided:
        P = _one_sided(P, 0)
    ctx = _ctx(sn, P)
    _, colour = ctx.colours()
    res = ctx.solve(0.0, 8)
    r, _ = ctx.get_r_u()
    ref = O.fc2d_nsgs_port(P, tol=0.0, maxiter=8, order=_order(colour))
    np.testing.assert_array_equal(r, ref.r)
    assert res["error"] == pytest.approx(ref.error, rel=1e-12, abs=0)
    ctx.set_precision(0, 1e-30, 1 << 20)
    ctx.set_r(np.zeros(2 * P.nc))
    ctx.solve(1e-300, 8)
    rm, _ = ctx.get_r_u()
    s32, s64 = ctx.last_sweeps()
    ctx.close()
    # a problem whose FP32 sweeps settle earlier goes on in FP64 until it settles
    assert 1 <= s32 <= s32 + s64 <= 8
    want = O.fc2d_sweeps_f32_port(P, np.zeros(2 * P.nc), s32, order=_order(colour))
    if s64:
        want = O.fc2d_nsgs_port(P, r0=want, tol=0.0, maxiter=s64, order=_order(colour)).r
    np.testing.assert_array_equal(rm, want)
