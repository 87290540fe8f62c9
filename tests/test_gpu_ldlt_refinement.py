"""Accelerated refinement steps of FP32 fronts: systems whose condition number
makes several steps necessary, from one equation (every step parallel to the
first: null directions) past the eight directions that are kept.  b = A x for
a random x, so that the attainable residual (a few units of 2^-53 |A| |x|, with
|b| some |A| |x| / 4) is far below the tolerance.  The solve must reach it
within as many steps as allowed, and x the exact solution within the tolerance
times the condition number; steps past the attainable residual must not spoil
x."""
import numpy as np
import pytest

from nla3d_gb300 import ldlt

pytestmark = pytest.mark.gpu


def _system(n, cond):
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * np.logspace(0, -np.log10(cond), n)) @ q.T / 3.0
    a = 0.5 * (a + a.T)
    io = 1 + np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))])
    co = np.concatenate([np.arange(r, n) + 1 for r in range(n)])
    return a, io.astype(np.uint32), co.astype(np.uint32), a @ rng.standard_normal(n)


@pytest.mark.parametrize("fronts", ["fp32", "fp32-tc"])
@pytest.mark.parametrize("n,cond", [(1, 1.0), (2, 1e4), (37, 1e5), (300, 1e5), (700, 3e5)])
def test_steps_reach_the_tolerance_and_stay_there(n, cond, fronts):
    torch = pytest.importorskip("torch")
    a, io, co, b = _system(n, cond)
    s = ldlt.DeviceLDLT(io, co, None, fronts)
    v, bd = torch.from_numpy(a[np.triu_indices(n)]).cuda(), torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    ref = np.linalg.solve(a, b)
    tol = 1e-12
    s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=40, tol=tol)
    assert s.last_steps <= 40 and s.last_residual <= tol
    got = x.cpu().numpy()
    assert np.linalg.norm(b - a @ got) <= 2 * tol * np.linalg.norm(b)
    bound = 2 * np.linalg.cond(a) * (tol + 2.0 ** -52)
    assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref)
    for steps in (0, 1, 2, 12):      # an unattainable tolerance: every step is taken
        s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=steps, tol=0.0,
                       strict=False)
        assert s.last_residual == 0.0 or s.last_steps >= steps
    got = x.cpu().numpy()
    s.close()
    assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("fronts", ["fp32", "fp32-tc"])
def test_x_is_whole_when_the_steps_run_out(fronts):
    """An unattainable tolerance and every budget up to the directions that are
    kept: once the attainable residual is reached a last step is often worse than
    an earlier one, and the best x comes back.  Read on another stream right after
    the call, x must have the residual that the call reports: b - A x in FP64
    here and there differ by the rounding of n products a row, each n 2^-53 |A| |x|."""
    torch = pytest.importorskip("torch")
    n = 300
    a, io, co, b = _system(n, 1e5)
    s = ldlt.DeviceLDLT(io, co, None, fronts)
    v, bd = torch.from_numpy(a[np.triu_indices(n)]).cuda(), torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    spent = 0
    for steps in range(1, 31):
        with torch.cuda.stream(other):
            x.fill_(float("nan"))
            other.synchronize()
            s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=steps, tol=0.0,
                           strict=False)
            got = x.clone().cpu().numpy()
        rounding = n * 2.0 ** -53 * np.linalg.norm(np.abs(a) @ np.abs(got)) / np.linalg.norm(b)
        res = np.linalg.norm(b - a @ got) / np.linalg.norm(b)
        assert abs(res - s.last_residual) <= 2 * rounding, steps
        spent += s.last_residual > 0.0 and s.last_steps == steps   # no other way out
    s.close()
    assert spent > 0


@pytest.mark.parametrize("fronts", ["fp32", "fp32-tc"])
def test_gmres_after_the_steps_and_a_solve_after_it(fronts):
    """An unattainable tolerance with more steps than the accelerated ones take:
    GMRES goes on from the best x, its basis in the directions' memory.  The
    residual it ends with is rounding (n products a row, each 2^-53 |A| |x|), and
    the next solve on the handle repeats the first bit for bit."""
    torch = pytest.importorskip("torch")
    n = 300
    a, io, co, b = _system(n, 1e5)
    s = ldlt.DeviceLDLT(io, co, None, fronts)
    v, bd = torch.from_numpy(a[np.triu_indices(n)]).cuda(), torch.from_numpy(b).cuda()
    x, y = torch.empty_like(bd), torch.empty_like(bd)
    torch.cuda.synchronize()
    s.factor_device(v.data_ptr())
    s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=40, tol=1e-12)
    first = x.cpu().numpy()
    s.solve_device(v.data_ptr(), bd.data_ptr(), y.data_ptr(), max_refine=45, tol=0.0, strict=False)
    got = y.cpu().numpy()
    rounding = n * 2.0 ** -53 * np.linalg.norm(np.abs(a) @ np.abs(got))
    assert np.linalg.norm(b - a @ got) <= rounding
    s.solve_device(v.data_ptr(), bd.data_ptr(), x.data_ptr(), max_refine=40, tol=1e-12)
    assert np.array_equal(x.cpu().numpy(), first)
    s.close()
