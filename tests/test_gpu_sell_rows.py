"""SELL passes over long warp rows against the tile engine, bit for bit.

A warp takes the warp rows that start in one block of 32 chunks (csrc/sell.cuh); a block inside
one long row has none, and rows of 16 or more chunks on average get their own launch shape
from 1M nonzeros on. The LPs have rows of one to several blocks, of a block's edge, and long rows
among short ones, on both sides of these rules.
"""
import pytest

from test_gpu_stream import assert_identical, ragged_lp, solve_with

pytestmark = pytest.mark.gpu


def sp():
    import saddlepoint_b200

    return saddlepoint_b200


LPS = {
    "rows of 64 chunks beside rows of 2": lambda: sp().generate_transport_lp(1, 40, 2048),
    "rows of 32 chunks": lambda: sp().generate_transport_lp(2, 70, 1024),
    "rows of 33 chunks": lambda: sp().generate_transport_lp(3, 33, 1025),
    "one warp row": lambda: sp().generate_transport_lp(4, 1, 900),
    "ragged": lambda: ragged_lp(5, 2100, 2048, 400, 500),
    "long rows, split launches": lambda: sp().generate_transport_lp(6, 800, 850),
    "15 chunks a row, one launch": lambda: sp().generate_transport_lp(7, 480, 1150),
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", LPS)
def test_sell_long_rows_equal_tile_engine(name, mixed, gpu_backend):
    lp = LPS[name]()
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=200,
                          precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    a, b = solve_with("sell", lp, p, gpu_backend), solve_with("tiles", lp, p, gpu_backend)
    assert_identical(a, b)
    assert a.norm_estimate == b.norm_estimate
