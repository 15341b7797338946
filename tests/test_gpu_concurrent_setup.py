"""Hierarchies of different sizes set up by several threads at once, each on a context of its own, equal the ones set
up alone: no thread's launches depend on what another thread is setting up."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_concurrent_setups_match_alone(native):
    from afepack_gb300 import workloads as W
    from afepack_gb300.amg import AMGSolver
    from afepack_gb300.fem import BoundaryConditionAdmin, Context, Space, assemble
    loads = [W.poisson3d_p1(9), W.poisson2d_p1(40), W.poisson3d_p1(14), W.elliptic2d_p2(20), W.poisson2d_p1(75),
             W.poisson3d_p2_multi(5, 1)]

    def solve(wl, out, i, reps):
        ctx = Context(0)
        space = Space(ctx, wl.space)
        for _ in range(reps):
            K, M = assemble(space, wl.acc_stiff, wl.acc_mass, wl.coef)
            b = M.vmult(np.ascontiguousarray(wl.f.reshape(wl.space.n_dof, -1)[:, 0]))
            bc = BoundaryConditionAdmin(wl.space)
            bc.add(1, 0.0)
            bc.apply(K, b)
            amg = AMGSolver(K, dense_tail=0)
            x, _ = amg.pcg(b, 1e-10)
            out[i].append((x, [amg.level_matrix(l) for l in range(1, amg.n_project() + 1)]))

    alone = [[] for _ in loads]
    for i, wl in enumerate(loads):
        solve(wl, alone, i, 1)
    together = [[] for _ in loads]
    threads = [threading.Thread(target=solve, args=(wl, together, i, 4)) for i, wl in enumerate(loads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, got in zip(alone, together):
        assert len(got) == 4
        for x, levels in got:
            assert np.array_equal(x, a[0][0])
            for l, m in zip(levels, a[0][1]):
                assert all(np.array_equal(u, v) for u, v in zip(l, m))
