"""The FP64 SOLID81 kernel where its four-element warps, its material branches
and its exact rest state can go wrong: element counts around a multiple of
four, distorted elements, each material (and two of them in one launch), and
states at rest or merely translated.  K and F against the CPU oracle at the
parity bound, 1e-12 of the largest entry."""
import numpy as np
import pytest

from nla3d_gb300 import meshgen as mg
from nla3d_gb300.batch import BatchAssembly
from nla3d_gb300.storage import assemble_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MATERIALS = {"nh": (mg.MAT_NEO_HOOKEAN, (1.0, 1000.0)),
             "mr": (mg.MAT_MOONEY_RIVLIN, (0.4, 0.1, 2000.0)),
             "bid": (mg.MAT_BIDERMAN, (0.4, 0.05, 0.01, 0.1, 2000.0))}


def _mesh(n, material, seed, clamp=True):
    mat_id, c = MATERIALS[material]
    m = mg.solid81_block(*n, 0.25, mat_id, c, clamp_z0=clamp)
    rng = np.random.default_rng(seed)
    m.xyz = m.xyz + rng.uniform(-0.04, 0.04, m.xyz.shape)
    return m


def _check(mesh, u, p):
    s, U, K, F = assemble_state(mesh, u, p, "fp64")
    _, Uo, Ko, Fo = O.solve_state(mesh, u, p, "port")
    assert np.array_equal(U, Uo)
    for b in K:
        if K[b].size:
            assert np.abs(K[b] - Ko[b]).max() <= 1e-12 * np.abs(Ko[b]).max(), b
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    assert s.element_status() == (0, 0)
    return K, F


@pytest.mark.parametrize("material", sorted(MATERIALS))
@pytest.mark.parametrize("n", [(1, 1, 1), (1, 1, 2), (3, 1, 1), (5, 1, 1), (3, 3, 1), (7, 3, 3)])
def test_distorted_blocks_match_the_oracle(n, material):
    mesh = _mesh(n, material, seed=sum(n))
    u, p = mg.twist_state(mesh, angle_deg=25.0, stretch=1.3, noise_frac=0.02, seed=3)
    _check(mesh, u, p)


@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_rest_and_translation_leave_no_residual(material):
    """At rest F = I: with zero pressures every entry of F is exactly zero, and
    a translation (exact in floating point) changes nothing."""
    mesh = _mesh((3, 2, 2), material, seed=1, clamp=False)
    zero, p0 = np.zeros((mesh.n_nodes, 3)), np.zeros(mesh.n_elems)
    K0, F0 = _check_zero(mesh, zero, p0)
    K1, F1 = _check_zero(mesh, zero + np.array([1.0, -2.0, 0.5]), p0)
    for b in K0:
        assert np.array_equal(K0[b], K1[b])
    rng = np.random.default_rng(2)
    _check(mesh, zero, rng.normal(0.0, 0.1, mesh.n_elems))


def _check_zero(mesh, u, p):
    s, U, K, F = assemble_state(mesh, u, p, "fp64")
    assert not F.any()
    return K, F


def test_two_materials_in_one_warp():
    """A batch of one-element meshes of different materials: the four elements
    of a warp take different branches."""
    names = ["nh", "mr", "bid", "nh", "mr"]
    meshes, states = [], []
    for k, name in enumerate(names):
        m = _mesh((1, 1, 1), name, seed=k)
        meshes.append(m)
        states.append(mg.twist_state(m, angle_deg=10.0 * k, stretch=1.2, seed=k))
    b = BatchAssembly(meshes, "fp64").init()
    b.set_U(b.state_vector(states))
    b.update()
    b.assemble()
    K, F = b.K_all(), b.F()
    for i, (m, (u, p)) in enumerate(zip(meshes, states)):
        _, _, Ko, Fo = O.solve_state(m, u, p, "port")
        for blk in Ko:
            if Ko[blk].size:
                assert np.abs(b.mesh_K(K, i, blk) - Ko[blk]).max() <= 1e-12 * np.abs(Ko[blk]).max()
        assert np.abs(b.mesh_F(F, i) - Fo).max() <= 1e-12 * np.abs(Fo).max()
    b.close()


@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_mirrored_elements_keep_the_reference_values(material):
    """Elements numbered left-handed (det dX/dxi < 0) are flagged; K and F are
    still the reference's, which takes J = sqrt(det C) and a negative weight."""
    m = _mesh((3, 2, 1), material, seed=6)
    m.conn = np.ascontiguousarray(m.conn[:, [3, 2, 1, 0, 7, 6, 5, 4]])
    u, p = mg.twist_state(m, angle_deg=20.0, stretch=1.2, noise_frac=0.02, seed=4)
    s, U, K, F = assemble_state(m, u, p, "fp64")
    _, Uo, Ko, Fo = O.solve_state(m, u, p, "port")
    for b in K:
        if K[b].size:
            assert np.abs(K[b] - Ko[b]).max() <= 1e-12 * np.abs(Ko[b]).max(), b
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    assert s.element_status() == (m.n_elems, 1)


def _stretched(name, rng):
    """A linear map of the mesh and a displacement gradient."""
    small = 1e-4 * rng.uniform(-1, 1, (3, 3))
    if name == "sheared by 100":
        return np.array([[1.0, 100.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]]), small
    q1, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    q2, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    a = q1 @ np.diag([1.0, 0.05, 0.001]) @ q2
    return a * np.sign(np.linalg.det(a)), small


@pytest.mark.parametrize("name", ["sheared by 100", "thin, oblique"])
@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_badly_shaped_elements_match_the_oracle(material, name):
    """Elements whose dX/dxi is badly conditioned, at small strains: F is as well
    conditioned as ever, so K and F stay within the parity bound (the oracle itself
    is within 1e-14 of extended precision here)."""
    mat_id, c = MATERIALS[material]
    m = mg.solid81_block(3, 2, 2, 0.25, mat_id, c, clamp_z0=False)
    rng = np.random.default_rng(8)
    m.xyz = m.xyz + rng.uniform(-0.005, 0.005, m.xyz.shape)
    a, grad = _stretched(name, rng)
    m.xyz = np.ascontiguousarray(m.xyz @ a.T)
    _check(m, m.xyz @ grad.T, rng.normal(0.0, 0.1, m.n_elems))
