"""The grid engine of mid-sized LPs against the tile engine, bit for bit.

The iterations between an epoch's first and its check run in one cooperative launch
(csrc/grid.cuh); a row's sum and the values made from it are the tile engine's, so a solve
gives the same bits with SP_PASS_ENGINE=tiles. The LPs sit at the edges of what a CTA keeps in
shared memory (row inputs and entries, row inputs, neither), with CTAs that have no rows, warp
rows, empty rows, and LPs that the engine leaves to launches.
"""
import os
import threading

import numpy as np
import pytest

from conftest import netlib_lp
from test_gpu_stream import assert_identical, ragged_lp, solve_with

pytestmark = pytest.mark.gpu


def sp():
    import saddlepoint_b200

    return saddlepoint_b200


def params(iters, **kw):
    return sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=iters, **kw)


LPS = {
    "one row, one column": lambda: sp().generate_random_lp(1, 1, 1, (1, 1)),
    "CTAs without rows": lambda: sp().generate_random_lp(2, 17, 33, (1, 5)),
    "5 CTAs": lambda: sp().generate_random_lp(3, 513, 1024, (8, 12)),
    "warp rows": lambda: sp().generate_transport_lp(9, 40, 60),
    "warp rows and empty rows": lambda: ragged_lp(11, 1100, 1500, 300, 300),
    "a row longer than a tile": lambda: ragged_lp(12, 1200, 2600, 100, 100),
    "power law": lambda: sp().generate_powerlaw_lp(6, 4000, 8000, 60000, 1.5, 2, 1500),
    "1024 columns and 512 rows a CTA": lambda: sp().generate_random_lp(4, 512 * 148, 1024 * 148, (2, 3)),
    "one column more": lambda: sp().generate_random_lp(5, 512 * 148, 1024 * 148 + 1, (2, 3)),
    "entries in global memory": lambda: sp().generate_random_lp(6, 40000, 80000, (11, 14)),
    "2560 columns and 1280 rows a CTA": lambda: sp().generate_random_lp(7, 1280 * 148, 2560 * 148, (2, 3)),
    "one row more": lambda: sp().generate_random_lp(8, 1280 * 148 + 1, 2560 * 148, (2, 3)),
    "long warp rows": lambda: sp().generate_transport_lp(5, 1100, 900),
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", LPS)
def test_grid_engine_equals_tile_engine(name, mixed, gpu_backend):
    lp = LPS[name]()
    p = params(300, precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)
    assert a.norm_estimate == b.norm_estimate


@pytest.mark.parametrize("check_every,iters", [(1, 40), (2, 41), (3, 40), (7, 100), (65, 1300), (200, 130), (0, 90)])
def test_grid_epochs_of_any_length(check_every, iters, gpu_backend):
    lp = sp().generate_random_lp(21, 3000, 6000, (3, 8))
    p = params(iters, check_every=check_every)
    assert_identical(solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend))


@pytest.mark.parametrize("name", ["80bau3b", "25fv47", "woodinfe"])
def test_grid_solve_of_netlib_equals_tile_engine(name, gpu_backend):
    """To the tolerance (or the infeasibility), the mixed form's switch to FP64 included."""
    lp = netlib_lp(name)
    for kw in ({}, {"precision": sp().Precision.Mixed}):
        p = sp().SolverParams(tolerance=1e-4, max_iterations=10_000, **kw)
        a, b = solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
        assert a.status == b.status
        assert_identical(a, b)


def test_grid_and_direct_launches_share_one_state(gpu_backend):
    """Epochs with the grid's launches, then with timed direct ones, then again the grid's, after
    a warm start."""
    lp = sp().generate_random_lp(22, 9000, 18000, (3, 8))
    rng = np.random.default_rng(5)
    x, y = rng.uniform(0, 1, lp.ncols), rng.uniform(-1, 1, lp.nrows)
    for precision in (sp().Precision.FP64, sp().Precision.Mixed):
        out = []
        for engine in ("grid", "tiles"):
            os.environ["SP_PASS_ENGINE"] = engine
            try:
                s = sp().Solver(lp, params(10**9, precision=precision), gpu_backend)
            finally:
                del os.environ["SP_PASS_ENGINE"]
            s.warm_start(x, y)
            s.run_epochs(3)
            s.set_timing(4 if engine == "grid" else 0)
            s.run_epochs(2)
            s.set_timing(0)
            s.run_epochs(5)
            s.sync()
            out.append((s.download(), s.trace(), s.info().iterations))
            s.close()
        (a, ta, ia), (b, tb, ib) = out
        assert ia == ib == 10 * 64 and ta == tb
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_grid_solves_beside_each_other(gpu_backend):
    """Solves of three backends (streams) from three threads, one of them on launches: each as
    when it is alone."""
    lps = [sp().generate_random_lp(30 + k, m, 2 * m, (4, 6)) for k, m in enumerate((9000, 20000, 300000))]
    p = params(640)
    alone = [sp().solve(lp, p, gpu_backend) for lp in lps]
    got = [None] * len(lps)

    def work(k):
        be = sp().CudaBackend(0)
        for _ in range(3):
            got[k] = sp().solve(lps[k], p, be)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(lps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got):
        assert b is not None
        assert_identical(a, b)


def test_grid_solve_beside_a_batch(gpu_backend):
    """The grid waits for the SMs that a batch on another stream holds; both as when alone."""
    lp = sp().generate_random_lp(40, 20000, 40000, (4, 6))
    p = params(640)
    alone = sp().solve(lp, p, gpu_backend)
    lps = [sp().generate_random_lp(50 + k, 30 + 3 * k, 60 + 6 * k, (3, 8)) for k in range(300)]
    b = sp().BatchSolver(lps, params(3000), gpu_backend)
    want = [(r.objective, r.iterations) for r in b.solve()[0]]
    got = []

    def work():
        be = sp().CudaBackend(0)
        for _ in range(6):
            got.append(sp().solve(lp, p, be))

    t = threading.Thread(target=work)
    t.start()
    for _ in range(3):
        assert [(r.objective, r.iterations) for r in b.solve()[0]] == want
    t.join()
    assert len(got) == 6
    for g in got:
        assert_identical(alone, g)


def test_grid_nonfinite_iterates_are_a_numerical_error(gpu_backend):
    """Costs near the largest number overflow the first residuals: the same error as on tiles."""
    lp = sp().generate_random_lp(23, 3000, 6000, (3, 5))
    lp.c = np.full(lp.ncols, 1e308)
    p = sp().SolverParams(bound_objective_rescaling=False, geometric_mean_passes=0, ruiz_iterations=0,
                          pock_chambolle_alpha=None)
    for engine in ("grid", "tiles"):
        with pytest.raises(sp().SolveError) as e:
            solve_with(engine, lp, p, gpu_backend)
        assert e.value.code == 5
