"""The PLANE41 kernel's material branches, rest state and element counts
around its 32-element blocks, and the sparse products' long rows: against the
CPU oracle, K and F at the parity bound (1e-12 of the largest entry), the
products bit for bit on the same K."""
import numpy as np
import pytest

from nla3d_gb300 import meshgen as mg
from nla3d_gb300.storage import FEStorage, assemble_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MATERIALS = {"nh": (mg.MAT_NEO_HOOKEAN, (1.0, 500.0)),
             "mr": (mg.MAT_MOONEY_RIVLIN, (0.4, 0.1, 800.0)),
             "bid": (mg.MAT_BIDERMAN, (0.4, 0.05, 0.01, 0.1, 800.0))}


@pytest.mark.parametrize("material", sorted(MATERIALS))
@pytest.mark.parametrize("n", [(1, 1), (31, 1), (8, 4), (11, 3), (13, 10)])
def test_distorted_plates_match_the_oracle(n, material):
    mat_id, c = MATERIALS[material]
    m = mg.plane41_plate(*n, 0.5, mat_id, c, clamp_y0=True)
    rng = np.random.default_rng(sum(n))
    m.xyz[:, :2] += rng.uniform(-0.08, 0.08, (m.n_nodes, 2))
    for scale in (0.0, 1.0):
        u, p = mg.plane_state(m, 1.25, 0.15, 0.02, seed=1)
        s, U, K, F = assemble_state(m, scale * u, p, "fp64")
        _, Uo, Ko, Fo = O.solve_state(m, scale * u, p, "port")
        assert np.array_equal(U, Uo)
        for b in K:
            if K[b].size:
                assert np.abs(K[b] - Ko[b]).max() <= 1e-12 * np.abs(Ko[b]).max(), (b, scale)
        assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max(), scale
        assert s.element_status() == (0, 0)


@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_mirrored_plates_keep_the_reference_values(material):
    """Elements numbered clockwise (det dX/dxi < 0) are flagged; K and F are
    still the reference's, which takes J = sqrt(det C) and a negative weight."""
    mat_id, c = MATERIALS[material]
    m = mg.plane41_plate(7, 5, 0.5, mat_id, c, clamp_y0=True)
    m.conn = np.ascontiguousarray(m.conn[:, [3, 2, 1, 0]])
    u, p = mg.plane_state(m, 1.2, 0.1, 0.02, seed=3)
    s, U, K, F = assemble_state(m, u, p, "fp64")
    _, Uo, Ko, Fo = O.solve_state(m, u, p, "port")
    for b in K:
        if K[b].size:
            assert np.abs(K[b] - Ko[b]).max() <= 1e-12 * np.abs(Ko[b]).max(), b
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    assert s.element_status() == (m.n_elems, 1)


@pytest.mark.parametrize("name", ["sheared by 100", "thin, oblique"])
@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_badly_shaped_plates_match_the_oracle(material, name):
    """Elements whose dX/dxi is badly conditioned, at small strains: F is as well
    conditioned as ever, so K and F stay within the parity bound (the oracle itself
    is within 1e-14 of extended precision here)."""
    mat_id, c = MATERIALS[material]
    m = mg.plane41_plate(7, 5, 0.25, mat_id, c, clamp_y0=False)
    rng = np.random.default_rng(8)
    m.xyz[:, :2] += rng.uniform(-0.005, 0.005, (m.n_nodes, 2))
    a = np.array([[1.0, 100.0], [0.0, 1.0]])
    if name == "thin, oblique":
        t, s = np.array([0.7, 1.9])
        a = np.array([[np.cos(t), -np.sin(t)], [np.sin(t), np.cos(t)]]) @ np.diag([1.0, 0.001]) \
            @ np.array([[np.cos(s), -np.sin(s)], [np.sin(s), np.cos(s)]])
    m.xyz[:, :2] = m.xyz[:, :2] @ a.T
    u = np.zeros((m.n_nodes, 3))
    u[:, :2] = m.xyz[:, :2] @ (1e-4 * rng.uniform(-1, 1, (2, 2))).T
    p = rng.normal(0.0, 0.1, m.n_elems)
    s, U, K, F = assemble_state(m, u, p, "fp64")
    _, Uo, Ko, Fo = O.solve_state(m, u, p, "port")
    for b in K:
        if K[b].size:
            assert np.abs(K[b] - Ko[b]).max() <= 1e-12 * np.abs(Ko[b]).max(), b
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    assert s.element_status() == (0, 0)


@pytest.mark.parametrize("n", [(5, 6, 1), (6, 6, 2), (9, 11, 2)])
def test_products_with_rows_above_and_below_the_long_limit(n):
    """A rigid-body end: the master's rows in K(2) hold one entry per slave
    DoF, here below, near and well above the limit for a thread of its own."""
    m = mg.solid81_bar_mpc(*n, 0.3)
    rng = np.random.default_rng(n[0])
    m.xyz[:-1] += rng.uniform(-0.02, 0.02, (m.n_nodes - 1, 3))
    u, p = mg.twist_state(m, 10.0, 1.1, seed=2)
    s, U, K, F = assemble_state(m, u, p, "fp64")
    o = O.OracleModel(m, "port", max_in_row=1024)
    o.set_U(U)
    o.update()
    o.assemble()
    import torch
    from nla3d_gb300.batch_newton import device_view
    for b in (1, 12, 2):                     # the oracle's K values on the device
        ptr, nv = s.device_K(b)
        if nv:
            device_view(torch, ptr, nv).copy_(torch.from_numpy(o.K(b)))
    torch.cuda.synchronize()
    shapes = {(1, 0): (s.n_con, s.n_con), (2, 0): (s.blocks[2][0],) * 2,
              (12, 0): (s.blocks[2][0], s.n_con), (12, 1): (s.n_con, s.blocks[2][0])}
    for (block, trans), (nx, ny) in shapes.items():
        x, y = rng.standard_normal(nx), rng.standard_normal(ny)
        x[rng.random(nx) < 0.2] = 0.0
        for coef in (1.0, -1.0, 0.7):
            got = s.block_mv(block, trans, x, coef, y)
            want = o.block_mv(block, trans, x, coef, y)
            assert np.array_equal(got.view(np.uint64), np.asarray(want).view(np.uint64)), (block, coef)
