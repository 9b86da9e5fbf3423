"""Kernels at the sizes where they can go wrong: ends of tiles, remainders and
the smallest and largest lengths of each launch shape."""
import numpy as np
import pytest

from tests._helpers import rel_l2
from tests.test_gpu_step import make_case, make_ctx, run_oracle

pytestmark = pytest.mark.gpu


# x lengths of the partitioned lines: the shortest and longest of 4, 8, 16 and 32
# lanes, with equal and unequal partitions; odd y and z lengths.  Tolerance: the
# one every step is held to (test_gpu_step).
@pytest.mark.parametrize("n", [(12, 13, 12), (20, 14, 15), (24, 13, 18), (45, 17, 12),
                               (50, 15, 20), (125, 13, 12), (135, 13, 15), (250, 14, 12),
                               (270, 13, 12), (500, 13, 12)])
def test_x_lines_of_any_length_match_oracle(n):
    g, f, c1, par = make_case(*n)
    assert c1.any()
    ref = run_oracle(g, f, c1, par, 3)
    with make_ctx(g, f, c1, par) as ctx:
        ctx.step(3)
        for k in ("u", "v", "w", "p", "T", "u_ta", "T_pre"):
            assert rel_l2(ctx.download(k), ref.f[k]) < 1e-10, k
