"""Small fronts by a warp and by a block: pivot counts and row counts around the
limits (8 pivots; 32, 64 and 128 rows), children of one dense root.  Held to
the extend-add test's bound: the refinement's tolerance times the condition
number."""
import pytest

from test_gpu_ldlt_extend_add import test_children_meet_in_a_dense_root as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("k", [1, 7, 8, 9])
@pytest.mark.parametrize("rows", [(2, 24, 32), (33, 63, 64), (65, 127, 128, 129)])
def test_leaves_around_the_limits(k, rows, fronts):
    updates = tuple(max(1, m - k) for m in rows)
    _check(k, updates, 135, fronts)
