"""Fronts in which elimination grows: pivots of 1e-4 (FP64 fronts: 1e-7) at the
ends of 64-pivot blocks of one dense front, whose joined inverses cancel.  One
application of the factor must leave no more than four times the residual of
substitution by 64-pivot blocks in the same arithmetic, restated here with
numpy from the same unpivoted factorisation (four: two roundings of one factor
against another's), and the refined x must reach the tolerance.  Sizes: the
last 64-pivot block partial, single rows past a block, two 512-pivot blocks."""
import numpy as np
import pytest

from nla3d_gb300 import ldlt

pytestmark = pytest.mark.gpu


def _system(n, tiny, value):
    rng = np.random.default_rng(3)
    B = rng.standard_normal((n, n)) / np.sqrt(n)
    A = B @ B.T + np.eye(n)
    for j in tiny:      # the Schur complement of the pivots before j becomes `value`
        A[j, j] += value - (A[j, j] - A[j, :j] @ np.linalg.solve(A[:j, :j], A[:j, j]))
    return A, rng.standard_normal(n)


def _substitution(A, b, T):
    """x by an unpivoted LDL^T in T and 64-pivot blocks' inverses in T"""
    n = len(A)
    L, d = A.astype(T), np.zeros(n, T)
    for k in range(n):
        d[k] = L[k, k]
        l = L[k + 1:, k] / d[k]
        L[k + 1:, k + 1:] -= np.outer(l, L[k + 1:, k])
        L[k + 1:, k] = l
    X = []
    for q in range(0, n, 64):
        Lb = L[q:q + 64, q:q + 64]
        Y = np.eye(len(Lb), dtype=T)
        for i in range(len(Lb)):
            Y[i] -= Lb[i, :i] @ Y[:i]
        X.append(Y.astype(np.float64))
    L, y = L.astype(np.float64), b.copy()
    for k, q in enumerate(range(0, n, 64)):
        e = min(n, q + 64)
        y[q:e] = X[k] @ y[q:e]
        y[e:] -= L[e:, q:e] @ y[q:e]
    y /= d
    for k, q in reversed(list(enumerate(range(0, n, 64)))):
        e = min(n, q + 64)
        y[q:e] = X[k].T @ y[q:e]
        y[:q] -= L[q:e, :q].T @ y[q:e]
    return y


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("n,tiny", [(130, [63]), (200, [63]), (400, [63, 255]),
                                    (512, [63, 127, 191]), (513, [191]), (700, [255, 575])])
def test_growth_leaves_substitutions_residual(n, tiny, fronts):
    torch = pytest.importorskip("torch")
    fp64 = fronts == "fp64"
    A, x = _system(n, tiny, 1e-7 if fp64 else 1e-4)
    b = A @ x
    ref = b - A @ _substitution(A, b, np.float64 if fp64 else np.float32)
    io = 1 + np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))])
    co = np.concatenate([np.arange(r, n) + 1 for r in range(n)])
    s = ldlt.DeviceLDLT(io.astype(np.uint32), co.astype(np.uint32), np.arange(n, dtype=np.int32),
                        fronts)
    v, bd = torch.from_numpy(A[np.triu_indices(n)]).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty_like(bd)
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    s.solve_device(v.data_ptr(), bd.data_ptr(), out.data_ptr(), max_refine=0, tol=0.0, strict=False)
    one = out.cpu().numpy()
    info = s.info()
    s.solve_device(v.data_ptr(), bd.data_ptr(), out.data_ptr(), max_refine=30, tol=1e-13)
    got = out.cpu().numpy()
    s.close()
    assert info["perturbed"] == 0 and info["max_front"] == n
    # (the tensor cores' products: three TF32 terms, some units of 2^-21)
    factor = 32 if fronts == "fp32-tc" else 4
    assert np.linalg.norm(b - A @ one) <= factor * np.linalg.norm(ref)
    assert np.linalg.norm(got - x) <= 2 * np.linalg.cond(A) * 1e-13 * np.linalg.norm(x)
