"""The mixed SOLID81 kernel widens its FP32 tangent with integer operations:
contributions near both ends of the range that a material may have (1e-20 .. 1e20), and ones
that are not finite.

A material scaled by a power of two scales every FP32 operation exactly; what
may differ are products that fall below 2^-149.  A K entry passes through
fewer than 2^9 such roundings, each multiplied by shape gradients, weights and
deformation gradients of at most 2^2 in all at unit spacing, and at most 2^3
elements meet in it: 2^14 half units, 2^-136."""
import numpy as np
import pytest

from nla3d_gb300 import meshgen as mg
from nla3d_gb300.storage import assemble_state

pytestmark = pytest.mark.gpu


def _tangent(scale, precision):
    c = (0.4 * scale, 0.1 * scale, 2000.0 * scale)
    mesh = mg.solid81_block(3, 2, 2, 1.0, mg.MAT_MOONEY_RIVLIN, c, clamp_z0=False)
    u, p = mg.twist_state(mesh, angle_deg=5.0, stretch=1.1, seed=4)
    return assemble_state(mesh, u, p * scale, precision)[2][2]


@pytest.mark.parametrize("exponent", [-60, 55])
def test_scaled_material_scales_the_tangent(exponent):
    scale = 2.0 ** exponent
    one, K = _tangent(1.0, "mixed"), _tangent(scale, "mixed")
    # the displacement entries: those that scale in FP64 (the pressure ones do not)
    d = _tangent(1.0, "fp64")
    uu = (_tangent(scale, "fp64") == d * scale) & (d != 0.0)
    assert uu.sum() > uu.size // 2
    assert np.abs(K[uu]).max() > scale / 64
    assert np.abs(K[uu] - one[uu] * scale).max() <= 2.0 ** -136


def test_nan_displacement_stays_nan():
    mesh = mg.solid81_block(3, 2, 2, 1.0, mg.MAT_NEO_HOOKEAN, (1.0, 1000.0), clamp_z0=False)
    u, p = mg.twist_state(mesh, angle_deg=5.0, stretch=1.1, seed=4)
    u[7, 1] = np.nan
    s32, _, K32, F32 = assemble_state(mesh, u, p, "mixed")
    s64, _, K64, F64 = assemble_state(mesh, u, p, "fp64")
    for b in K64:
        assert np.array_equal(np.isnan(K32[b]), np.isnan(K64[b]))
    assert np.array_equal(np.isnan(F32), np.isnan(F64)) and np.isnan(F64).any()
    assert s32.element_status() == s64.element_status()
