"""The inverse of a 64-pivot diagonal block where several small pivots lie inside
it, at the ends of its 16-pivot column groups: as for joined blocks, one
application must leave no more than four times the residual of substitution
with an inverse formed by substitution, in the geometric mean over six systems."""
import numpy as np
import pytest

from test_gpu_ldlt_growth import apply_and_solve, growth_case, growth_factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("n,tiny", [(200, [15, 31, 47]), (400, [15, 31, 47]), (150, [79, 95])])
def test_growth_inside_a_block(n, tiny, fronts):
    torch = pytest.importorskip("torch")
    ratios = []
    for seed in range(6):
        A, _, b, ref = growth_case(n, tiny, fronts, seed)
        one, _, info = apply_and_solve(torch, A, b, fronts)
        assert info["perturbed"] == 0
        ratios.append(np.linalg.norm(b - A @ one) / ref)
    assert np.exp(np.mean(np.log(ratios))) <= growth_factor(fronts)
