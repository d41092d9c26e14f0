"""Reading results back takes its turn while two threads keep the device full of
cooperative sweeps: the three readers get their arrays throughout, not when the
sweeps end."""
import threading
import time

import pytest
from test_gpu_copy_order import _cases

pytestmark = pytest.mark.gpu
SECONDS = 2


def test_read_back_under_load(built_lib):
    import siconos_gb300.numerics as sn
    from siconos_gb300.device import DeviceSolver
    from siconos_gb300.scene import lattice
    stop, solves = threading.Event(), [0, 0]
    loads = []
    for s in (3, 4):
        loads.append(DeviceSolver(0))
        loads[-1].load(lattice(30, 31, 15, seed=s))

    def load(k):
        while not stop.is_set():
            loads[k].solve(tol=1e-300, max_iter=8, precision=1, lanes=1)
            solves[k] += 1

    ctxs = [make() for make, _, _ in _cases(sn)]
    reads = [0] * len(ctxs)

    def read(k):
        get = getattr(ctxs[k], "get_r_u", None) or ctxs[k].get
        while not stop.is_set():
            get()
            reads[k] += 1

    for k in range(2):  # each solver's first call allocates
        loads[k].solve(tol=1e-300, max_iter=1, precision=1, lanes=1)
    threads = [threading.Thread(target=load, args=(k,), daemon=True) for k in range(2)]
    threads += [threading.Thread(target=read, args=(k,), daemon=True) for k in range(len(ctxs))]
    for t in threads:
        t.start()
    time.sleep(SECONDS)
    under_load = list(reads)
    stop.set()
    for t in threads:
        t.join(60)
    assert not any(t.is_alive() for t in threads)
    for c in ctxs + loads:
        c.close()
    assert min(solves) > 10
    assert min(under_load) > 10, under_load
