"""Starts and problems given by the host reach the device before the kernels that
read them, with the device kept busy by other contexts' solves in threads of their
own: small problems (up to 64 KB an array, whose copies return when they are
staged) solved from alternating starts, in contexts made anew now and then, give
the bits they give alone."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SECONDS = 8


def _cases(sn):
    from siconos_gb300.scene import lattice_global
    from test_fc2d_oracle import load_fc2d, tiled2d
    from test_rfc3d_oracle import load_rfc3d, tiled
    R = tiled(load_rfc3d("rfc3d_rockfall_21_54029")[0], 2, 7)
    P = tiled2d(load_fc2d("fc2d_FrictionContactProblem00727")[0], 1, 4)
    G = lattice_global(3, 3, 2, seed=2)

    def rolling(ctx, r):
        ctx.set_r(r)
        ctx.solve(1e-300, 2)
        return ctx.get_r_u()[0]

    def flat(ctx, r):
        ctx.set_r(r)
        ctx.solve(1e-300, 2)
        return ctx.get_r_u()[0]

    def whole(ctx, r):
        ctx.set_start(r, None)
        ctx.solve(1e-300, 2)
        return ctx.get()[0]

    return [(lambda: sn.RollingContext(R.nc, R.rowptr, R.colidx, R.blocks, R.q, R.mu, R.mur), rolling, 5 * R.nc),
            (lambda: sn.Fc2dContext(P.nc, P.rowptr, P.colidx, P.blocks, P.q, P.mu), flat, 2 * P.nc),
            (lambda: sn.Gfc3dContext.from_problem(G), whole, 3 * G.nc)]


def test_same_bits_under_load(built_lib):
    import siconos_gb300.numerics as sn
    from siconos_gb300.device import DeviceSolver
    from siconos_gb300.scene import lattice
    g = np.random.default_rng(3)
    stop, failures, counts = threading.Event(), [], []

    def load(scenes, batch):
        d = DeviceSolver(0)
        d.load_batch(scenes) if batch else d.load(scenes[0])
        while not stop.is_set():
            d.zero_r()
            if batch:
                d.solve_batch(tol=1e-300, max_iter=6, precision=0, fp32_only=1)
            else:
                d.solve(tol=1e-300, max_iter=4, precision=1, lanes=1)
        d.close()

    def check(make, solve, starts, want):
        n, ctx = 0, make()
        while not stop.is_set():
            k = n % 2
            if not np.array_equal(solve(ctx, starts[k]), want[k]):
                failures.append((make, n))
            n += 1
            if n % 50 == 0:
                ctx.close()
                ctx = make()
        ctx.close()
        counts.append(n)

    def guarded(f, *a):
        try:
            f(*a)
        except Exception as e:  # a thread's error is the test's
            failures.append(e)

    threads = [threading.Thread(target=guarded, args=(load, [lattice(24, 24, 12, seed=3)], False), daemon=True),
               threading.Thread(target=guarded, args=(load, [lattice(12, 12, 6, seed=k) for k in range(6)], True),
                                daemon=True)]
    for make, solve, n in _cases(sn):
        starts = [np.zeros(n), g.standard_normal(n)]
        ctx = make()
        want = [solve(ctx, r) for r in starts]
        ctx.close()
        threads.append(threading.Thread(target=guarded, args=(check, make, solve, starts, want), daemon=True))
    for t in threads:
        t.start()
    time.sleep(SECONDS)
    stop.set()
    for t in threads:
        t.join(60)
    assert not any(t.is_alive() for t in threads)
    assert not failures, failures[:3]
    assert len(counts) == 3 and min(counts) > 10
