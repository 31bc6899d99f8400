"""Which epoch engine a solver gets, with what in shared memory: the cases of test_gpu_resident.py
and test_gpu_grid.py are at the edges that they name, and no engine is left out in silence."""
import numpy as np
import pytest

from test_gpu_grid import LPS as GRID_LPS
from test_gpu_resident import LPS as CHIP_LPS
from test_gpu_stream import assert_identical, solve_with

pytestmark = pytest.mark.gpu


def sp():
    import saddlepoint_b200

    return saddlepoint_b200


def engine(lp, backend, mixed=False):
    p = sp().SolverParams(precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    s = sp().Solver(lp, p, backend)
    e = s.epoch_engine()
    s.close()
    assert e["left"] == 0 and (mixed or e["fp32"] == 0)
    return e


# CTAs, and the level in FP64: 2 entries in shared memory, 1 row inputs only
CHIP = {
    "one CTA, its most columns and rows": (1, 2),
    "one row more than a CTA's": (8, 2),
    "one column": (1, 2),
    "33 columns": (1, 2),
    "a cluster": (8, 2),
    "a cluster, entries in L2": (8, 1),
    "a cluster's most columns": (8, 2),
    "beyond a cluster": None,
    "warp rows": (8, 2),
    "warp rows and empty rows": (8, 2),
    "a row longer than a tile": None,
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", CHIP_LPS)
def test_the_on_chip_engine_takes_its_cases(name, mixed, monkeypatch, gpu_backend):
    monkeypatch.setenv("SP_PASS_ENGINE", "resident")
    e = engine(CHIP_LPS[name](), gpu_backend, mixed)
    if CHIP[name] is None:
        assert e["engine"] == "launched"
        return
    assert (e["engine"], e["ctas"]) == ("on chip", CHIP[name][0])
    assert e["fp64"] == CHIP[name][1] or mixed  # the FP32 vectors take room too
    assert not mixed or e["fp32"] >= e["fp64"] >= 1


# the level in FP64: 2 row inputs and entries, 1 row inputs, 0 neither
GRID = {
    "one row, one column": 2,
    "CTAs without rows": 2,
    "5 CTAs": 2,
    "warp rows": 2,
    "warp rows and empty rows": 2,
    "a row longer than a tile": None,
    "power law": 2,
    "1024 columns and 512 rows a CTA": 2,
    "one column more": 1,
    "entries in global memory": 2,  # they fit after all: MORE has LPs whose entries do not
    "2560 columns and 1280 rows a CTA": 0,  # rows of uneven lengths are dealt unevenly: MORE has one that fits
    "one row more": 0,
    "long warp rows": 0,
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", GRID_LPS)
def test_the_grid_engine_takes_its_cases(name, mixed, monkeypatch, gpu_backend):
    monkeypatch.setenv("SP_PASS_ENGINE", "grid")
    lp = GRID_LPS[name]()
    e = engine(lp, gpu_backend, mixed)
    if GRID[name] is None:
        assert e["engine"] == "launched"
        return
    assert (e["engine"], e["ctas"]) == ("grid", min(148, max(4, lp.nnz // 1000)))
    assert e["fp64"] == GRID[name]
    assert not mixed or e["fp32"] >= e["fp64"]


# Columns of one length are dealt evenly: 2,560 to each of 148 CTAs, and one more.
MORE = {
    "entries in global memory": (lambda: sp().generate_random_lp(6, 40000, 80000, (20, 24)), 1),
    "2560 columns a CTA": (lambda: sp().generate_random_lp(7, 148000, 2560 * 148, (2, 2)), 1),
    "one column more": (lambda: sp().generate_random_lp(7, 148000, 2560 * 148 + 1, (2, 2)), 0),
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", MORE)
def test_grid_engine_with_less_in_shared_memory_equals_tile_engine(name, mixed, monkeypatch, gpu_backend):
    make, level = MORE[name]
    lp = make()
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=150,
                          precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("grid", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)
    monkeypatch.setenv("SP_PASS_ENGINE", "grid")
    e = engine(lp, gpu_backend, mixed)
    assert (e["engine"], e["ctas"], e["fp64"]) == ("grid", 148, level)


def long_columns(columns, rows):
    """`rows` rows of two entries, in columns of 2 * rows / columns."""
    k = np.arange(rows)
    ci = np.sort(np.stack([k % columns, (k % columns + 1 + k // columns % (columns - 1)) % columns], 1), 1)
    rng = np.random.default_rng(1)
    return sp().LpProblem(rows, columns, np.arange(0, 2 * rows + 1, 2, dtype=np.int64), ci.reshape(-1).astype(np.int32),
                          rng.standard_normal(2 * rows), rng.uniform(-1, 1, columns), np.full(rows, -np.inf),
                          rng.uniform(0, 1, rows), np.zeros(columns), np.ones(columns))


@pytest.mark.parametrize("make,want", [
    (lambda: sp().generate_random_lp(1, 200, 400, (3, 6)), "on chip"),
    (lambda: sp().generate_random_lp(1, 4096, 8192, (2, 2)), "on chip"),
    (lambda: sp().generate_random_lp(1, 4097, 8192, (2, 2)), "grid"),
    (lambda: sp().generate_powerlaw_lp(6, 20000, 40000, 300000, 1.5, 2, 1500), "grid"),
    (lambda: sp().generate_transport_lp(5, 1000, 1000), "grid"),
    (lambda: sp().generate_transport_lp(5, 1100, 1000), "launched"),  # long rows: the stream engine's
    (lambda: long_columns(2000, 1_200_000), "grid"),  # long columns: 28-35 % less an iteration on the grid
])
def test_the_engine_follows_from_the_size(make, want, monkeypatch, gpu_backend):
    for v in ("SP_PASS_ENGINE", "SP_PRIMAL_ENGINE", "SP_DUAL_ENGINE"):
        monkeypatch.delenv(v, raising=False)
    assert engine(make(), gpu_backend)["engine"] == want


@pytest.mark.parametrize("engines", ["tiles", "stream", "sell", "large"])
def test_other_engines_leave_the_iterations_to_launches(engines, monkeypatch, gpu_backend):
    monkeypatch.setenv("SP_PASS_ENGINE", engines)
    for m in (200, 9000):
        assert engine(sp().generate_random_lp(1, m, 2 * m, (3, 6)), gpu_backend)["engine"] == "launched"
