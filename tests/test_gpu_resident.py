"""The on-chip engine of small LPs against the tile engine, bit for bit.

A small LP's iterations run in one CTA or one cluster (csrc/resident.cuh); the sums, the
partial sums and the decisions are the tile engine's, so a solve gives the same bits with
SP_PASS_ENGINE=tiles. The LPs sit at the edges of what the engine holds: one CTA's rows and
columns, a cluster's, entries that do and do not fit in shared memory, warp rows, empty rows
and columns, and LPs that it leaves to the tile engine.
"""
import os

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
    "one CTA, its most columns and rows": lambda: sp().generate_random_lp(1, 512, 1024, (3, 3)),
    "one row more than a CTA's": lambda: sp().generate_random_lp(2, 513, 1024, (3, 3)),
    "one column": lambda: sp().generate_random_lp(3, 8, 1, (3, 3)),
    "33 columns": lambda: sp().generate_random_lp(4, 17, 33, (1, 5)),
    "a cluster": lambda: sp().generate_random_lp(5, 1417, 2834, (3, 8)),
    "a cluster, entries in L2": lambda: sp().generate_random_lp(6, 3500, 7000, (5, 9)),
    "a cluster's most columns": lambda: sp().generate_random_lp(7, 900, 8192, (2, 2)),
    "beyond a cluster": lambda: sp().generate_random_lp(8, 4200, 9000, (3, 3)),
    "warp rows": lambda: sp().generate_transport_lp(9, 40, 60),
    "warp rows and empty rows": lambda: ragged_lp(11, 1100, 1500, 300, 300),
    "a row longer than a tile": lambda: ragged_lp(12, 1200, 2600, 100, 100),
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", LPS)
def test_resident_engine_equals_tile_engine(name, mixed, gpu_backend):
    lp = LPS[name]()
    p = params(300, precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("resident", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)
    assert a.norm_estimate == b.norm_estimate


@pytest.mark.parametrize("check_every,iters", [(1, 40), (2, 41), (7, 100), (64, 64), (65, 1300), (200, 130)])
def test_resident_epochs_of_any_length(check_every, iters, gpu_backend):
    lp = sp().generate_random_lp(21, 300, 600, (3, 8))
    p = params(iters, check_every=check_every)
    assert_identical(solve_with("resident", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend))


@pytest.mark.parametrize("name", ["afiro", "israel", "25fv47", "woodinfe", "perold"])
def test_resident_solve_of_netlib_equals_tile_engine(name, gpu_backend):
    """To the tolerance (or the infeasibility), in both termination modes and both precisions."""
    lp = netlib_lp(name)
    for kw in ({}, {"termination": sp().Termination.StepImplied}, {"precision": sp().Precision.Mixed}):
        p = sp().SolverParams(tolerance=1e-4, max_iterations=20_000, **kw)
        a, b = solve_with("resident", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
        assert a.status == b.status
        assert_identical(a, b)


def test_resident_and_direct_launches_share_one_state(gpu_backend):
    """Epochs on chip, then direct launches with timing events, then on chip again, after a
    warm start: the state handed over in global memory is whole."""
    lp = sp().generate_random_lp(22, 700, 1400, (3, 8))
    rng = np.random.default_rng(5)
    x, y = rng.uniform(0, 1, lp.ncols), rng.uniform(-1, 1, lp.nrows)
    for precision in (sp().Precision.FP64, sp().Precision.Mixed):
        out = []
        for engine in ("resident", "tiles"):
            os.environ["SP_PASS_ENGINE"] = engine
            try:
                s = sp().Solver(lp, params(10**9, precision=precision), gpu_backend)
            finally:
                del os.environ["SP_PASS_ENGINE"]
            s.warm_start(x, y)
            s.run_epochs(3)
            s.set_timing(4 if engine == "resident" else 0)
            s.run_epochs(2)
            s.set_timing(0)
            s.run_epochs(20)
            s.sync()
            out.append((s.download(), s.trace(), s.info().iterations))
            s.close()
        (a, ta, ia), (b, tb, ib) = out
        assert ia == ib == 25 * 64 and ta == tb
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_resident_nonfinite_iterates_are_a_numerical_error(gpu_backend):
    """Costs near the largest number overflow the first residuals: the same error as on tiles."""
    lp = sp().generate_random_lp(23, 60, 120, (3, 5))
    lp.c = np.full(lp.ncols, 1e308)
    p = sp().SolverParams(bound_objective_rescaling=False, geometric_mean_passes=0, ruiz_iterations=0,
                          pock_chambolle_alpha=None)
    for engine in ("resident", "tiles"):
        with pytest.raises(sp().SolveError) as e:
            solve_with(engine, lp, p, gpu_backend)
        assert e.value.code == 5


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kw", [dict(max_iterations=300), dict(max_iterations=90, check_every=0),
                                dict(max_iterations=100, check_every=7)])
def test_batch_on_chip_equals_the_solo_solve(kw, mixed, gpu_backend):
    """Instances at the edges of the classes (clusters of 1, 2 and 4 CTAs), with warp rows, and
    one beyond them beside: each has the solo solve's bits, twice."""
    ms = [9, 60, 300, 512, 513, 1024, 1025, 2000, 2048]
    lps = [sp().generate_random_lp(40 + m, m, 2 * m, (3, 8)) for m in ms]
    lps += [sp().generate_random_lp(7, 8, 1, (3, 3)), sp().generate_transport_lp(9, 40, 60), netlib_lp("25fv47"),
            netlib_lp("israel")]
    beyond = sp().generate_random_lp(8, 2100, 4200, (3, 8))
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0,
                          precision=sp().Precision.Mixed if mixed else sp().Precision.FP64, **kw)
    b = sp().BatchSolver(lps + [beyond], p, gpu_backend)
    for _ in range(2):
        res, _ = b.solve()
        for i, lp in enumerate(lps):
            solo = sp().solve(lp, p, gpu_backend)
            x, y = b.solution(i)
            assert res[i].variant == "tiles" and not res[i].handed_off
            assert res[i].iterations == solo.iterations and res[i].restarts == solo.restarts, lp.name
            assert res[i].objective == solo.objective and res[i].status == int(solo.status), lp.name
            assert np.array_equal(x, solo.x) and np.array_equal(y, solo.y), lp.name
        assert res[len(lps)].iterations == kw["max_iterations"]


def test_batch_hand_off_from_a_cluster(gpu_backend, monkeypatch):
    """Stragglers on clusters stop at a check that all of the cluster's CTAs agree on, and get
    the solo solve's result."""
    monkeypatch.setenv("SP_BATCH_HANDOFF_S", "1e-9")
    lps = [sp().generate_random_lp(60 + m, m, 2 * m, (3, 8)) for m in (700, 900, 1500, 1900)]
    p = params(1000)
    b = sp().BatchSolver(lps, p, gpu_backend)
    res, _ = b.solve()
    assert sum(r.handed_off for r in res) >= len(lps) - 1
    for i, lp in enumerate(lps):
        solo = sp().solve(lp, p, gpu_backend)
        x, y = b.solution(i)
        assert res[i].iterations == solo.iterations == 1000 and res[i].objective == solo.objective
        assert np.array_equal(x, solo.x) and np.array_equal(y, solo.y)


def test_batch_solutions_in_any_order(gpu_backend):
    """Solutions fetched in order (a block ahead), out of order, twice, and after another solve
    are the same; an instance larger than a block is fetched by itself."""
    ms = [40, 2000, 9, 300, 25000, 700, 60, 2048, 80]
    lps = [sp().generate_random_lp(80 + i, m, 2 * m, (2, 4)) for i, m in enumerate(ms)]
    b = sp().BatchSolver(lps, params(40), gpu_backend)
    b.solve()
    ahead = [b.solution(i) for i in range(len(ms))]
    for i in (8, 3, 3, 4, 5, 6, 0, 1, 7, 2):
        x, y = b.solution(i)
        assert np.array_equal(x, ahead[i][0]) and np.array_equal(y, ahead[i][1])
    solo = sp().solve(lps[1], params(40), gpu_backend)
    assert np.array_equal(ahead[1][0], solo.x) and np.array_equal(ahead[1][1], solo.y)
    b.solve()
    for i in range(len(ms)):
        x, y = b.solution(i)
        assert len(x) == 2 * ms[i] and np.array_equal(x, ahead[i][0]) and np.array_equal(y, ahead[i][1])
