"""The rolling solver's FP32 sweeps as dataflow against the sweeps by colours,
bit for bit.  A zero block without its transpose's place takes the pattern's
symmetry, so the sweeps go by colours; its products add zeros to sums that they
cannot change."""
from dataclasses import replace

import numpy as np
import pytest

from test_gpu_rfc3d import _ctx, sn  # noqa: F401
from test_rfc3d_oracle import load_rfc3d, tiled

pytestmark = pytest.mark.gpu


def _with_zero_block(sn, T, colour):  # noqa: F811
    """T with a zero block between two contacts that had none, of different
    colours, and such that the colouring stays."""
    i, at = 0, T.rowptr[1]
    have = set(T.colidx[:at].tolist())
    rowptr = T.rowptr + (np.arange(T.nc + 1) > i)
    for j in (k for k in range(T.nc) if k not in have and colour[k] != colour[i]):
        colidx = np.insert(T.colidx, at, j)
        if np.array_equal(sn.colour(rowptr, colidx)[1], colour):
            return replace(T, rowptr=rowptr, colidx=colidx,
                           blocks=np.insert(np.asarray(T.blocks).reshape(-1, 25), at, 0.0, axis=0))
    raise AssertionError("no such pair of contacts")


@pytest.mark.parametrize("copies", [1, 2, 37, 90, 500, 2000])
def test_equals_colours(sn, copies):  # noqa: F811
    T = tiled(load_rfc3d("rfc3d_rockfall_21_54029")[0], copies, 5)
    out, colours = [], []
    for P in (T, None):
        if P is None:
            P = _with_zero_block(sn, T, colours[0])
        ctx = _ctx(sn, P)
        colours.append(ctx.colours()[1])
        ctx.set_precision(0, 1e-30, 1 << 20)
        ctx.solve(1e-300, 9)
        assert ctx.last_sweeps() == (9, 0)
        out.append(ctx.get_r_u()[0])
        ctx.close()
    np.testing.assert_array_equal(colours[0], colours[1])
    np.testing.assert_array_equal(out[0], out[1])
