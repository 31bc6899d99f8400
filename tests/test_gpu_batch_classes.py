"""Which class of clusters a batch's instances run in, asserted, and each class's results.

An instance's class (csrc/batch.cu: res_class) follows from its rows' lengths alone; the result
of an instance on chip is the solo solve's, bit for bit.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sp():
    import saddlepoint_b200

    return saddlepoint_b200


# (LP, CTAs of its cluster, columns a CTA may have): the smallest and largest of each class; two
# LPs of 2,020 and 2,030 rows that two large parts cannot split evenly, for the class of four
CLASSES = [
    (lambda: sp().generate_random_lp(49, 9, 18, (3, 8)), 1, 1024),
    (lambda: sp().generate_random_lp(552, 512, 1024, (3, 8)), 1, 1024),
    (lambda: sp().generate_random_lp(553, 513, 1026, (3, 8)), 1, 2048),
    (lambda: sp().generate_random_lp(1064, 1024, 2048, (3, 8)), 1, 2048),
    (lambda: sp().generate_random_lp(1065, 1025, 2050, (3, 8)), 2, 2048),
    (lambda: sp().generate_random_lp(2088, 2048, 4096, (3, 8)), 2, 2048),
    (lambda: sp().generate_random_lp(14, 2030, 4060, (3, 8)), 4, 1024),
    (lambda: sp().generate_random_lp(553, 2020, 4040, (3, 8)), 4, 1024),
]


@pytest.mark.parametrize("mixed", [False, True])
def test_each_class_gives_the_solo_solve(mixed, gpu_backend):
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=200,
                          precision=sp().Precision.Mixed if mixed else sp().Precision.FP64)
    lps = [make() for make, _, _ in CLASSES]
    b = sp().BatchSolver(lps + [sp().generate_random_lp(8, 2100, 4200, (3, 8))], p, gpu_backend)
    assert b.engine(len(lps)) is None  # more rows than two CTAs take
    for i, (_, ctas, cols) in enumerate(CLASSES):
        assert b.engine(i)[:2] == (ctas, cols), i
    for _ in range(2):
        res, _ = b.solve()
        for i, lp in enumerate(lps):
            solo = sp().solve(lp, p, gpu_backend)
            x, y = b.solution(i)
            assert res[i].iterations == solo.iterations == 200 and res[i].objective == solo.objective, i
            assert np.array_equal(x, solo.x) and np.array_equal(y, solo.y), i


@pytest.mark.parametrize("m,ctas", [(40, 1), (700, 1), (1400, 2), (2300, None)])
def test_an_instance_without_a_first_iteration_has_a_zero_solution(m, ctas, gpu_backend, monkeypatch):
    """Coefficients of zero: the power iteration collapses before any iterate exists. The solution
    is zero, not what the scratch held of another instance, in any mix and on every solve."""
    monkeypatch.setenv("SP_BATCH_HANDOFF_S", "0")
    bad = sp().generate_random_lp(5, m, 2 * m, (2, 2))
    bad.values = np.zeros_like(bad.values)
    # others of its class that run before it on the same clusters, and smaller ones
    others = [sp().generate_random_lp(200 + i, m, 2 * m, (4, 6)) for i in range(160)]
    others += [sp().generate_random_lp(500 + i, 30, 60, (3, 5)) for i in range(5)]
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=64)
    for lps, at in (([bad], 0), (others + [bad], len(others))):
        b = sp().BatchSolver(lps, p, gpu_backend)
        assert (b.engine(at) or (None,))[0] == ctas
        for _ in range(2):
            res, _ = b.solve()
            assert res[at].status == -2  # a numerical breakdown of the power iteration
            x, y = b.solution(at)
            assert not x.any() and not y.any()
            assert all(r.status == 3 for i, r in enumerate(res) if i != at)
        b.close()


def test_the_largest_instances_run_beside_the_on_chip_ones(gpu_backend):
    """Instances beyond the on-chip classes start with them, not after them: together both take
    well under the sum of their times. And each has the result that it has without the
    others, on every solve (its values are scaled in place)."""
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=1000)
    small = [sp().generate_random_lp(600 + i, 1000, 2000, (3, 8)) for i in range(1200)]
    large = [sp().generate_random_lp(2300 + i, 2100 + 10 * i, 4200, (1, 2)) for i in range(4)]
    took, sols = {}, {}
    for name, lps in (("small", small), ("large", large), ("both", small + large)):
        b = sp().BatchSolver(lps, p, gpu_backend)
        assert [b.engine(i) is None for i in (0, len(lps) - 1)] == [name == "large", name != "small"]
        took[name] = min(b.solve()[1] for _ in range(4))
        sols[name] = [b.solution(i) for i in range(len(lps))]
        b.close()
    for (x, y), (u, v) in zip(sols["both"], sols["small"] + sols["large"]):
        assert np.array_equal(x, u) and np.array_equal(y, v)
    assert took["both"] < 0.85 * (took["small"] + took["large"]), took


def test_solutions_read_during_a_solve_do_not_outlive_it(gpu_backend, monkeypatch):
    """A thread that asks for solutions while another solves gets what is there; afterwards the
    solutions are the solve's, those of handed-off instances included."""
    monkeypatch.setenv("SP_BATCH_HANDOFF_S", "1e-9")
    lps = [sp().generate_random_lp(900 + i, 300 + 200 * i, 600 + 400 * i, (3, 8)) for i in range(4)]
    p = sp().SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=40_000)
    b = sp().BatchSolver(lps, p, gpu_backend)
    res = []
    t = threading.Thread(target=lambda: res.extend(b.solve()[0]))
    t.start()
    while t.is_alive():
        for i in range(len(lps)):
            b.solution(i)
    t.join()
    assert sum(r.handed_off for r in res) >= len(lps) - 1
    for i, lp in enumerate(lps):
        solo = sp().solve(lp, p, gpu_backend)
        x, y = b.solution(i)
        assert res[i].iterations == solo.iterations and np.array_equal(x, solo.x) and np.array_equal(y, solo.y), i
    b.close()
