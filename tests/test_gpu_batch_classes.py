"""Which class of clusters a batch's instances run in, asserted, and each class's results.

An instance's class (csrc/batch.cu: res_class) follows from its rows' lengths alone; the result
of an instance on chip is the solo solve's, bit for bit.
"""
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
