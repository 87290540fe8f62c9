"""Extend-add: several children under one dense root, each child's update rows
a different subset of the root's, with update sizes around the 32 rows of a
warp and the 128 that it holds in flight, down to a single row.  x against
numpy's solution of the same matrix, held to the refinement's tolerance times
the condition number."""
import numpy as np
import pytest

from nla3d_gb300 import ldlt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("k,updates,root", [(3, (1, 31, 32), 40), (5, (33, 127), 200),
                                            (40, (128, 129, 64, 7), 260), (70, (255, 257), 300),
                                            (9, (2,) * 12, 130)])
def test_children_meet_in_a_dense_root(k, updates, root, fronts):
    torch = pytest.importorskip("torch")
    nc = len(updates)
    n = k * nc + root
    rng = np.random.default_rng(n + k)
    A = rng.standard_normal((n, n)) / np.sqrt(n)
    A = A + A.T
    keep = np.zeros((n, n), bool)
    keep[k * nc:, k * nc:] = True
    for c, u in enumerate(updates):
        piv = np.arange(k * c, k * c + k)
        rows = k * nc + np.sort(rng.permutation(root)[:u])
        keep[np.ix_(piv, piv)] = True
        keep[np.ix_(piv, rows)] = True
        keep[np.ix_(rows, piv)] = True
    A = np.where(keep, A, 0.0) + np.eye(n) * 4.0
    w = np.linalg.eigvalsh(A)
    A += np.eye(n) * max(0.0, 0.5 - w[0])              # definite
    r, c = np.nonzero(np.triu(keep))
    io = (1 + np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))])).astype(np.uint32)
    tol = 1e-13 if fronts == "fp64" else 1e-12
    b = rng.standard_normal(n)
    s = ldlt.DeviceLDLT(io, (c + 1).astype(np.uint32), np.arange(n, dtype=np.int32), fronts)
    v, bd = torch.from_numpy(A[r, c]).cuda(), torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=30, tol=tol)
    out = x.cpu().numpy()
    s.close()
    ref = np.linalg.solve(A, b)
    bound = 2 * np.linalg.cond(A) * (tol + 2.0 ** -52)
    assert np.linalg.norm(out - ref) <= bound * np.linalg.norm(ref)
