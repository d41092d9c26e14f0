"""The dataflow sweep on stamped reactions at the edges of its splits of a
slab (from one row a warp to several slabs a warp) and with rows longer than
the slots gathered together, in FP32 and in FP64 (from one contact a unit to
ten): the coloured kernel's iterates bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(gpu, load, sweeps, precision=0):
    how = dict(precision=1) if precision else dict(fp32_only=1, switch_tol=0.0)
    out = []
    for on in (True, False):
        gpu.flow(on)
        try:
            load()
            st = gpu.solve(tol=1e-300, max_iter=sweeps, lanes=1, stall_window=0, **how)
        finally:
            gpu.flow(True)
        out.append((st["sweeps32"], st["sweeps64"], gpu.get()[0]))
    return out


@pytest.mark.parametrize("dims", [(2, 2, 1), (3, 3, 2), (7, 6, 5), (12, 11, 9), (19, 18, 11), (30, 31, 15), (40, 41, 20)])
@pytest.mark.parametrize("warps", [8, 10, 12])
def test_lattices(gpu, dims, warps):
    from siconos_gb300.scene import lattice
    sc = lattice(*dims, seed=9)
    gpu.flow_warps(warps)
    try:
        (n, k, r), (m, j, want) = _both(gpu, lambda: gpu.load(sc), 15)
    finally:
        gpu.flow_warps(0)
    assert (n, k) == (m, j)
    np.testing.assert_array_equal(r, want)


@pytest.mark.parametrize("dims", [(2, 2, 1), (3, 3, 2), (12, 11, 9), (19, 18, 11), (30, 31, 15), (44, 44, 22),
                                  (46, 46, 23)])
def test_lattices_fp64(gpu, dims):
    """On both sides of the line beyond which the sweeps go by colours too."""
    from siconos_gb300.scene import lattice
    sc = lattice(*dims, seed=9)
    (_, n, r), (_, m, want) = _both(gpu, lambda: gpu.load(sc), 10, precision=1)
    assert n == m
    np.testing.assert_array_equal(r, want)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nc,degree", [(40, 4), (40, 5), (40, 11), (700, 12), (700, 13), (150, 64), (150, 66)])
def test_long_rows(gpu, nc, degree, precision):
    """A ring where every contact is tied to its `degree` nearest (more colours
    than a lattice; from 65 blocks on the pattern is not looked at)."""
    g = np.random.default_rng(nc + degree)
    near = [d for k in range(1, degree // 2 + 1) for d in (k, -k)] + ([nc // 2] if degree % 2 else [])
    blocks, cols, rowptr = {}, [], [0]
    for i in range(nc):
        js = sorted({(i + d) % nc for d in near} | {i})
        for j in js:
            if j == i:
                blocks[i, i] = np.eye(3) * 2.0 + 0.1 * np.diag(g.uniform(0, 1, 3))
            elif (j, i) in blocks:
                blocks[i, j] = blocks[j, i].T
            else:
                blocks[i, j] = 0.05 * g.standard_normal((3, 3))
        cols += js
        rowptr.append(len(cols))
    vals = np.concatenate([blocks[i, j].reshape(-1, order="F") for i in range(nc)
                           for j in cols[rowptr[i]:rowptr[i + 1]]])
    q = g.standard_normal(3 * nc)
    q[::3] -= 1.0
    mu = g.uniform(0.2, 0.8, nc)

    def load():
        gpu.set_W(nc, np.array(rowptr), np.array(cols), vals)
        gpu.set_q_mu(q, mu)
        gpu.set_r(np.zeros(3 * nc))

    (n, k, r), (m, j, want) = _both(gpu, load, 15, precision)
    assert (n, k) == (m, j)
    np.testing.assert_array_equal(r, want)
