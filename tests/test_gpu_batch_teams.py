"""Batched problems solved by teams of blocks (few problems of unequal sizes)
give a solo solve's iterates bit for bit, in both precisions; the largest
problem's colours do not divide evenly over its team."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[(20, 19, 9), (3, 3, 2), (12, 11, 6)], [(2, 2, 1), (25, 24, 12)]],
                         ids=["three", "tiny-and-large"])
@pytest.mark.parametrize("precision,flow", [(0, True), (0, False), (1, True), (1, False)],
                         ids=["fp32", "fp32-colours", "fp64", "fp64-colours"])
def test_team_equals_solo_bitwise(gpu, dims, precision, flow):
    from siconos_gb300 import scene
    from siconos_gb300.device import DeviceSolver
    scs = [scene.lattice(*d, seed=50 + k, mu=0.3 + 0.2 * k) for k, d in enumerate(dims)]
    kw = dict(tol=1e-300, max_iter=12, precision=precision, fp32_only=1 - precision)
    gpu.flow(flow)  # the sweeps as dataflow, or colour by colour
    try:
        gpu.load_batch(scs)
        st = gpu.solve_batch(**kw)
    finally:
        gpu.flow(True)
    rb, ub = gpu.get_batch()
    solo = DeviceSolver(0)
    solo.flow(False)  # the coloured kernels, whose stop rules the batch has (the dataflow stops a sweep later)
    for k, s in enumerate(scs):
        solo.load(s)
        one = solo.solve(lanes=1, **kw)
        r, u = solo.get()
        assert (st["sweeps32"][k], st["sweeps64"][k]) == (one["sweeps32"], one["sweeps64"])
        assert np.array_equal(rb[k], r) and np.array_equal(ub[k], u), k
        # the error's sums are over other blocks: some 1e5 terms, all positive
        assert abs(st["error"][k] - one["error"]) <= 1e-12 * one["error"]
    solo.close()
