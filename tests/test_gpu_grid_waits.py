"""The ends of the grid engine's waits, without a fault on the GPU.

A launch of the grid engine whose CTAs cannot all start, since other streams' kernels hold SMs, is
left without effect and its iterations run by launches; the results keep their bits. The test
knob SP_TEST_GRID_WAIT (read when a solver is created) makes the first wait be for a CTA that is
not there ("start"), or the waits between passes give up at once ("pass").
"""
import threading
import time

import numpy as np
import pytest

from test_gpu_stream import assert_identical, solve_with

pytestmark = pytest.mark.gpu


def sp():
    import saddlepoint_b200

    return saddlepoint_b200


def params(iters, **kw):
    return sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=iters, **kw)


@pytest.fixture
def left_at_start(monkeypatch):
    monkeypatch.setenv("SP_TEST_GRID_WAIT", "start")


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("check_every,iters", [(2, 40), (3, 40), (64, 64 * 200 + 7), (0, 90)])
def test_epochs_left_to_launches_keep_their_bits(check_every, iters, mixed, left_at_start, gpu_backend):
    """More epochs than the first pause, so that the engine is tried again and left again."""
    lp = sp().generate_random_lp(21, 3000, 6000, (3, 8))
    p = params(iters, check_every=check_every, precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)
    assert a.norm_estimate == b.norm_estimate


@pytest.mark.parametrize("mixed", [False, True])
def test_epochs_left_to_the_large_problem_engines_keep_their_bits(mixed, left_at_start, gpu_backend):
    """1.2M nonzeros: the launches are the stream engine's and the SELL copy's, on two streams."""
    lp = sp().generate_random_lp(25, 120_000, 240_000, (5, 5))
    p = params(64 * 5, precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)


@pytest.mark.parametrize("read", ["sync", "info", "download", "trace", "solve"])
def test_every_read_finds_the_epochs_that_were_left(read, left_at_start, monkeypatch, gpu_backend):
    """Epochs queued behind the one that was left are run too, whatever asks first, with a warm
    start before and timed launches between."""
    lp = sp().generate_random_lp(22, 9000, 18000, (3, 8))
    rng = np.random.default_rng(5)
    x, y = rng.uniform(0, 1, lp.ncols), rng.uniform(-1, 1, lp.nrows)
    out = []
    for engine in ("grid", "tiles"):
        monkeypatch.setenv("SP_PASS_ENGINE", engine)
        s = sp().Solver(lp, params(70 * 64 if read == "solve" else 10**9), gpu_backend)
        monkeypatch.delenv("SP_PASS_ENGINE")
        for warm in (False, True):
            s.warm_start(x, y) if warm else s.reset()
            s.run_epochs(3)
            s.set_timing(4)
            s.run_epochs(2)
            s.set_timing(0)
            s.run_epochs(4)
            got = {"sync": s.sync, "info": s.info, "download": s.download, "trace": s.trace, "solve": s.solve}[read]()
            if read == "download":
                out.append(got)
            elif read == "trace":
                out.append(got)
            out.append((s.info().iterations, s.trace(), s.download()))
        if engine == "grid":
            assert s.epoch_engine()["engine"] == "grid" and s.epoch_engine()["left"] >= 2
        s.close()
    assert len(out) % 2 == 0
    for a, b in zip(out[:len(out) // 2], out[len(out) // 2:]):
        np.testing.assert_equal(a, b)


READS = {
    "solve": lambda s: s.solve(),
    "sync": lambda s: s.sync(),
    "info": lambda s: s.info(),
    "download": lambda s: s.download(),
    "trace": lambda s: s.trace(),
}


def assert_every_read_fails(s, message):
    for name, read in READS.items():
        with pytest.raises(sp().SolveError) as e:
            read(s)
        assert e.value.code == 1 and message in str(e.value), name


@pytest.mark.parametrize("mixed", [False, True])
def test_a_stalled_barrier_is_an_error_of_every_read(mixed, monkeypatch, gpu_backend):
    """The waits between passes give up at once: no caller gets the unfinished iterates as a
    result. A new solver of the same context gives a clean solve's bits."""
    lp = sp().generate_random_lp(24, 60000, 120000, (5, 5))  # its power iteration runs by launches
    p = params(640, precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    clean = solve_with("tiles", lp, p, gpu_backend)
    monkeypatch.setenv("SP_TEST_GRID_WAIT", "pass")
    s = sp().Solver(lp, p, gpu_backend)
    monkeypatch.delenv("SP_TEST_GRID_WAIT")
    assert s.epoch_engine()["engine"] == "grid"
    for _ in range(2):
        s.run_epochs(3)
        assert_every_read_fails(s, "the grid's barrier did not complete within its wait limit")
        s.reset()
    s.close()
    assert_identical(sp().solve(lp, p, gpu_backend), clean)


def test_a_stalled_barrier_of_the_power_iteration_is_an_error(monkeypatch, gpu_backend):
    lp = sp().generate_random_lp(24, 6000, 12000, (5, 5))
    monkeypatch.setenv("SP_TEST_GRID_WAIT", "pass")
    with pytest.raises(sp().SolveError) as e:
        sp().Solver(lp, params(640), gpu_backend)
    assert e.value.code == 1 and "the grid's barrier" in str(e.value)


def test_a_stalled_bulk_copy_is_an_error_of_every_read(monkeypatch, gpu_backend):
    """The stream engine's stall (its own test knob) on the same paths."""
    lp = sp().generate_powerlaw_lp(6, 4000, 8000, 60000, 1.5, 2, 1500)
    monkeypatch.setenv("SP_PASS_ENGINE", "stream")
    monkeypatch.setenv("SP_TEST_STREAM_WITHHOLD", "0")
    s = sp().Solver(lp, params(640), gpu_backend)
    monkeypatch.delenv("SP_PASS_ENGINE")
    monkeypatch.delenv("SP_TEST_STREAM_WITHHOLD")
    s.run_epochs(2)
    assert_every_read_fails(s, "a bulk copy of the pass pipeline did not complete")
    s.close()


def test_a_solve_beside_a_long_batch_runs(gpu_backend):
    """A kernel of another stream that holds an SM for seconds: the solve neither waits for it nor
    fails, and ends at its time limit; then the engine has the SMs again."""
    lp = sp().generate_random_lp(40, 20000, 40000, (5, 5))
    s = sp().Solver(lp, params(10**9, time_limit=0.5), gpu_backend)
    be = sp().CudaBackend(0)
    b = sp().BatchSolver([sp().generate_random_lp(41, 900, 1800, (3, 8))], params(1_000_000), be)
    took = []

    def work():
        t = time.time()
        b.solve()
        took.append(time.time() - t)

    thread = threading.Thread(target=work)
    try:
        assert s.epoch_engine()["engine"] == "grid" and b.engine(0)[0] == 1
        s.solve()
        assert s.epoch_engine()["left"] == 0
        thread.start()
        time.sleep(0.3)
        s.reset()
        t = time.time()
        beside = s.solve()
        dt = time.time() - t
        left = s.epoch_engine()["left"]
        thread.join()
        s.reset()
        s.solve()
        assert took[0] > 2.0 and dt < 1.5, (took, dt)
        assert beside.status.name == "TimeLimit" and beside.iterations > 1000
        assert left >= 1 and s.epoch_engine()["left"] == left
    finally:
        b.close()
        s.close()
        be.close()
