"""The solve's inverted diagonal blocks and per-width kernels at the widths
where they can go wrong: fronts whose pivots end before, at and after a 64-,
128-, 256- and 512-pivot boundary, one dense front and a chain of two, for
every front type.  x against numpy's solution of the same dense matrix, held
to the refinement's tolerance times the matrix's condition number."""
import numpy as np
import pytest

from nla3d_gb300 import ldlt

pytestmark = pytest.mark.gpu


def _dense_upper(n):
    io = 1 + np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))])
    co = np.concatenate([np.arange(r, n) + 1 for r in range(n)])
    return io.astype(np.uint32), co.astype(np.uint32)


def _solve(torch, io, co, values, b, fronts, tol):
    s = ldlt.DeviceLDLT(io, co, None, fronts)
    v, bd = torch.from_numpy(values).cuda(), torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=30, tol=tol)
    info = s.info()
    out = x.cpu().numpy()
    s.close()
    assert info["nonfinite"] == 0 and info["perturbed"] == 0
    return out, info


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("n", [129, 191, 192, 193, 320, 511, 512, 513, 577, 1025, 1100])
def test_one_dense_quasi_definite_front(n, fronts):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n)) / np.sqrt(n)
    A = B @ B.T + np.eye(n)
    A[n // 2:, n // 2:] *= -1.0              # [P C; C^T -Q], P and Q positive definite
    io, co = _dense_upper(n)
    b = rng.standard_normal(n)
    tol = 1e-13 if fronts == "fp64" else 1e-12
    x, info = _solve(torch, io, co, A[np.triu_indices(n)], b, fronts, tol)
    assert info["max_front"] == n
    ref = np.linalg.solve(A, b)
    bound = 2 * np.linalg.cond(A) * (tol + 2.0 ** -52)
    assert np.linalg.norm(x - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("k1,u,k2", [(3, 140, 200), (40, 200, 130), (64, 300, 70), (65, 100, 600),
                                     (530, 90, 64)])
def test_two_fronts_in_a_chain(k1, u, k2, fronts):
    """k1 pivots coupled to the first u of k2 (u <= k2: clipped) others: a
    child with update rows under a root."""
    torch = pytest.importorskip("torch")
    u = min(u, k2)
    n = k1 + k2
    rng = np.random.default_rng(n + u)
    B = rng.standard_normal((n, n)) / np.sqrt(n)
    A = B @ B.T + np.eye(n)
    A[:k1, k1 + u:] = 0.0
    A[k1 + u:, :k1] = 0.0
    A += np.eye(n) * (np.abs(np.linalg.eigvalsh(A)).max())   # definite again after the cut
    iu = [(r, c) for r in range(n) for c in range(r, n) if not (r < k1 and c >= k1 + u)]
    rows = np.array([r for r, _ in iu])
    co = (np.array([c for _, c in iu]) + 1).astype(np.uint32)
    io = (1 + np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])).astype(np.uint32)
    b = rng.standard_normal(n)
    tol = 1e-13 if fronts == "fp64" else 1e-12
    x, _ = _solve(torch, io, co, A[rows, co - 1], b, fronts, tol)
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(x - ref) <= 2 * np.linalg.cond(A) * (tol + 2.0 ** -52) * np.linalg.norm(ref)
