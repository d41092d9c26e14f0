"""Timeline records and work counters: what they record, and the sweeps of a
context on which they were switched on and off again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def own(built_lib):
    from siconos_gb300.device import DeviceSolver
    d = DeviceSolver(0)
    yield d
    d.close()


def test_fp64_sweeps_after_a_timeline(own):
    """The dataflow's sweeps start with one launch more (the stamps): before a
    timeline was armed, not while it is, and again after it was switched off.
    The first solve, which also looks at the pattern, is not counted."""
    from siconos_gb300.scene import lattice
    own.load(lattice(6, 6, 4, seed=1))
    n = []
    for arm in (None, None, 2, 0):
        if arm is not None:
            own.timeline(arm)
        own.zero_r()
        before = own.launches()
        own.solve(tol=1e-300, max_iter=4, precision=1, lanes=1)
        n.append(own.launches() - before)
    assert n[2] == n[1] - 1 and n[3] == n[1]


def test_counters_of_a_batch_between_solves(own):
    """Switched on after a first batch solve they count its FP32 sweeps (one
    local solve or take-off a contact and sweep), switched off nothing; the
    reactions are the same throughout."""
    from siconos_gb300.scene import lattice
    own.load_batch([lattice(8, 7, 5, seed=1), lattice(3, 3, 2, seed=2)])
    kw = dict(tol=1e-300, max_iter=10, fp32_only=1, switch_tol=0.0, stall_window=0)

    def solve():
        own.zero_r()
        own.solve_batch(**kw)
        return own.get()[0]

    want = solve()
    own.counters(True)
    np.testing.assert_array_equal(solve(), want)
    on = own.counters(False)
    np.testing.assert_array_equal(solve(), want)
    assert 0 < on["solves"] <= 10 * own.nc and on["newton"] > 0
    assert own.counters(False)["solves"] == 0


@pytest.mark.parametrize("dims", [(3, 3, 2), (12, 11, 9)])
def test_timeline_of_a_slab(own, dims):
    """Scenes small enough for a slab's rows to be spread over several warps: one
    record a slab all the same, its stamps in order, and the local solves of all
    slabs those that the sweep by colours counts."""
    from siconos_gb300.scene import lattice
    own.load(lattice(*dims, seed=6))
    kw = dict(tol=1e-300, max_iter=8, fp32_only=1, lanes=1, switch_tol=0.0, stall_window=0)
    records = {}
    for on in (True, False):
        own.flow(on)
        own.timeline(5)
        own.zero_r()
        own.solve(**kw)
        records[on] = own.timeline(0).reshape(-1, 8)
    slabs = records[True][records[True][:, 0] > 0]
    n = own.nc
    assert (n + 31) // 32 <= len(slabs) <= n
    for a, b in ((0, 1), (1, 2), (2, 3), (3, 6), (6, 7), (7, 4)):
        assert (slabs[:, a] <= slabs[:, b]).all(), (a, b)
    assert slabs[:, 5].sum() == records[False][:, 3].sum() > 0
