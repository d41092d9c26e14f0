"""Rows that store a second block on their diagonal: the dataflow sweeps read the
row's own last reaction there, as the sweeps by colours do, bit for bit."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _doubled(dims, seed, every):
    """A lattice whose contacts 0, every, 2 every, ... have a second diagonal
    block behind the others of their row."""
    from siconos_gb300.scene import lattice
    sc = lattice(*dims, seed=seed)
    at = np.asarray(sc.rowptr)[1:][::every]
    new = np.arange(0, sc.nc, every)
    blocks = sc.blocks.reshape(-1, 9)
    extra = 0.1 * blocks[[np.flatnonzero(sc.colidx[sc.rowptr[i]:sc.rowptr[i + 1]] == i)[0] + sc.rowptr[i] for i in new]]
    added = np.zeros(sc.nc + 1, np.int64)
    added[new + 1] = 1
    return SimpleNamespace(nc=sc.nc, rowptr=sc.rowptr + np.cumsum(added), colidx=np.insert(sc.colidx, at, new),
                           blocks=np.insert(blocks, at, extra, axis=0), q=sc.q, mu=sc.mu)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("dims,every", [((3, 3, 2), 1), ((12, 11, 9), 7), ((30, 31, 15), 5)])
@pytest.mark.parametrize("batch", [False, True], ids=["solo", "batch"])
def test_equals_colours(gpu, dims, every, precision, batch):
    scs = [_doubled(dims, 3, every)] + ([_doubled((5, 4, 3), 4, 2)] if batch else [])
    out = []
    for on in (True, False):
        gpu.flow(on)
        try:
            if batch:
                gpu.load_batch(scs)
                st = gpu.solve_batch(tol=1e-300, max_iter=12, precision=precision, fp32_only=1 - precision,
                                     switch_tol=0.0, stall_window=0)
                assert (st["sweeps64" if precision else "sweeps32"] == 12).all()
            else:
                gpu.load(scs[0])
                st = gpu.solve(tol=1e-300, max_iter=12, precision=precision, fp32_only=1 - precision, lanes=1,
                               switch_tol=0.0, stall_window=0)
                assert st["sweeps64" if precision else "sweeps32"] == 12
        finally:
            gpu.flow(True)
        out.append(gpu.get()[0])
    np.testing.assert_array_equal(*out)
