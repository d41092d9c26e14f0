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


def _one_sided(P, drop):
    """P without the `drop`-th block off the diagonal: the block's transpose
    stays, so the pattern is not symmetric and the sweeps go by colours."""
    from dataclasses import replace
    row = np.repeat(np.arange(P.nc), np.diff(P.rowptr))
    off = np.flatnonzero(row != P.colidx)
    keep = np.ones(len(row), bool)
    keep[off[drop]] = False
    return replace(P, rowptr=np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=P.nc))]),
                   colidx=P.colidx[keep], blocks=P.blocks[keep])


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("copies,drop", [(1, 0), (1, 7), (40, 123), (700, 0)])
def test_pattern_not_symmetric(sn, copies, drop, precision):  # noqa: F811
    """FP64 sweeps bit for bit; after FP32 sweeps the FP64 loop from theirs."""
    import oracle as O
    P, _ = load_rfc3d("rfc3d_rockfall_21_54029")
    T = _one_sided(tiled(P, copies, 7), drop)
    ctx = _ctx(sn, T)
    ctx.set_precision(precision)
    _, colour = ctx.colours()
    assert all(colour[i] != colour[j] for i in range(T.nc) for j in T.colidx[T.rowptr[i]:T.rowptr[i + 1]] if i != j)
    res = ctx.solve(0.0, 12)
    r, u = ctx.get_r_u()
    s32, s64 = ctx.last_sweeps()
    start = None
    if s32:
        ctx.set_r(np.zeros(5 * T.nc))
        ctx.solve(0.0, s32)
        start = ctx.get_r_u()[0]
    ctx.close()
    assert s32 + s64 == res["iterations"] == 12
    ref = O.rfc3d_nsgs_port(T, r0=start, tol=0.0, maxiter=s64, order=_order(colour))
    np.testing.assert_array_equal(r, ref.r)
    assert res["error"] == pytest.approx(ref.error, rel=1e-12, abs=0)


@pytest.mark.parametrize("copies", [1, 90, 500, 2000])
def test_units_of_a_warp(sn, copies):  # noqa: F811
    """From one contact a unit to six (FP64) and beyond a dozen (FP32)."""
    import oracle as O
    P, _ = load_rfc3d("rfc3d_rockfall_21_54029")
    T = tiled(P, copies, 5)
    ctx = _ctx(sn, T)
    _, colour = ctx.colours()
    res = ctx.solve(0.0, 6)
    r, _ = ctx.get_r_u()
    ctx.set_precision(0)
    ctx.set_r(np.zeros(5 * T.nc))
    mixed = ctx.solve(0.0, 6)
    r32, _ = ctx.get_r_u()
    ctx.close()
    ref = O.rfc3d_nsgs_port(T, tol=0.0, maxiter=6, order=_order(colour))
    np.testing.assert_array_equal(r, ref.r)
    assert res["iterations"] == mixed["iterations"] == 6
    # FP32 sweeps of the same contraction: rounding of the entries, 6e-8, times
    # six sweeps and a one-contact conditioning of 1e3
    assert np.linalg.norm(r32 - ref.r) <= 1e-3 * np.linalg.norm(ref.r)
