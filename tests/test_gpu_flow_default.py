"""The number of warps the FP32 dataflow takes when none is asked for: the
iterates of the coloured kernel on both sides of its line (a slab a warp) and
at sizes where it takes 8, 10 and 12; a request stays a request."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(30, 31, 15), (32, 34, 17), (36, 36, 18), (40, 41, 20), (42, 42, 21)])
def test_default_warps(gpu, dims):
    from siconos_gb300.scene import lattice
    sc = lattice(*dims, seed=4)
    out = {}
    for on, warps in ((False, 0), (True, 0), (True, 10)):
        gpu.flow(on)
        prev = gpu.flow_warps(warps)
        try:
            gpu.load(sc)
            st = gpu.solve(tol=1e-300, max_iter=10, fp32_only=1, lanes=1, switch_tol=0.0, stall_window=0)
        finally:
            assert gpu.flow_warps(prev) == warps
            gpu.flow(True)
        out[on, warps] = (st["sweeps32"], gpu.get()[0])
    n, want = out[False, 0]
    for key in ((True, 0), (True, 10)):
        assert out[key][0] == n
        np.testing.assert_array_equal(out[key][1], want)
