"""Fronts in which elimination grows: pivots of 1e-4 (FP64 fronts: 1e-7) at the
ends of 64-pivot blocks of one dense front, whose joined inverses cancel.  One
application of the factor must leave, in the geometric mean over six systems,
no more than four times the residual of substitution by 64-pivot blocks in the
same arithmetic, restated here with numpy from the same unpivoted
factorisation (one rounding of such a factor against another's differs by up
to five either way; means differ by up to three), and the refined x must reach
the tolerance.  Sizes: the last 64-pivot block partial, single rows past a
block, two 512-pivot blocks."""
import numpy as np
import pytest

from nla3d_gb300 import ldlt

pytestmark = pytest.mark.gpu


def _system(n, tiny, value, seed=3):
    rng = np.random.default_rng(seed)
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


def growth_case(n, tiny, fronts, seed):
    fp64 = fronts == "fp64"
    A, x = _system(n, tiny, 1e-7 if fp64 else 1e-4, seed)
    b = A @ x
    ref = np.linalg.norm(b - A @ _substitution(A, b, np.float64 if fp64 else np.float32))
    return A, x, b, ref


def growth_factor(fronts):
    # (the tensor cores' products: three TF32 terms, some units of 2^-21)
    return 32 if fronts == "fp32-tc" else 4


def apply_and_solve(torch, A, b, fronts):
    """x after one application, the refined x, and the factor's statistics"""
    n = len(A)
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
    s.solve_device(v.data_ptr(), bd.data_ptr(), out.data_ptr(), max_refine=30, tol=1e-13)
    got, info = out.cpu().numpy(), s.info()
    s.close()
    return one, got, info


@pytest.mark.parametrize("fronts", ["fp64", "fp32", "fp32-tc"])
@pytest.mark.parametrize("n,tiny", [(130, [63]), (200, [63]), (400, [63, 255]),
                                    (512, [63, 127, 191]), (513, [191]), (700, [255, 575])])
def test_growth_leaves_substitutions_residual(n, tiny, fronts):
    torch = pytest.importorskip("torch")
    ratios = []
    for seed in range(6):
        A, x, b, ref = growth_case(n, tiny, fronts, seed)
        one, got, info = apply_and_solve(torch, A, b, fronts)
        assert info["perturbed"] == 0 and info["max_front"] == n
        ratios.append(np.linalg.norm(b - A @ one) / ref)
        assert np.linalg.norm(got - x) <= 2 * np.linalg.cond(A) * 1e-13 * np.linalg.norm(x)
    assert np.exp(np.mean(np.log(ratios))) <= growth_factor(fronts)
