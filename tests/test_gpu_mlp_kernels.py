"""The network's fused backward and optimiser kernels at the edges of their
tiles (128 rows, 32 columns, chunks of 128 along the sum): layer gradients
with the bias sums, input gradients through the tanh, and one Adam launch over
more tensors than one launch holds."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n_out,n_in", [(1, 1, 1), (37, 66, 256), (127, 129, 33),
                                              (128, 128, 32), (129, 65, 31), (300, 256, 132),
                                              (385, 130, 97)])
def test_layer_and_input_gradients(batch, n_out, n_in):
    """Against float64 products of the same inputs.  An FP32 operand enters as
    a BF16 pair, 2^-16 of itself; sums of FP32 terms add 2^-24 each."""
    torch = pytest.importorskip("torch")
    from nla3d_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(batch + 7 * n_out + n_in)
    d = rng.normal(size=(batch, n_out)).astype(np.float32)
    x = np.tanh(rng.normal(size=(batch, n_in))).astype(np.float32)
    w = torch.from_numpy(rng.normal(size=(n_out, n_in)).astype(np.float32)).to(torch.bfloat16)
    dd, xd, wd = torch.from_numpy(d).cuda(), torch.from_numpy(x).cuda(), w.cuda()
    dW, db = torch.full((n_out, n_in), 7.0).cuda(), torch.full((n_out,), 7.0).cuda()
    dX, dX0 = torch.full((batch, n_in), 7.0).cuda(), torch.full((batch, n_in), 7.0).cuda()
    torch.cuda.synchronize()
    assert lib.nla3d_mlp_layer_grads(batch, n_out, n_in, dd.data_ptr(), xd.data_ptr(),
                                     dW.data_ptr(), db.data_ptr(), None) == 0
    assert lib.nla3d_mlp_input_grad(batch, n_out, n_in, dd.data_ptr(), wd.data_ptr(),
                                    xd.data_ptr(), dX.data_ptr(), None) == 0
    assert lib.nla3d_mlp_input_grad(batch, n_out, n_in, dd.data_ptr(), wd.data_ptr(), None,
                                    dX0.data_ptr(), None) == 0
    torch.cuda.synchronize()
    t = ctypes.c_uint32()
    assert lib.nla3d_mlp_status(ctypes.byref(t)) == 0 and t.value == 0
    d, x, w = d.astype(np.float64), x.astype(np.float64), w.double().numpy()
    tol = 8 * 2.0 ** -16
    assert np.abs(dW.cpu().numpy() - d.T @ x).max() <= tol * ((np.abs(d).T @ np.abs(x)).max() + 1)
    assert np.abs(db.cpu().numpy() - d.sum(0)).max() <= batch * 2.0 ** -24 * np.abs(d).sum(0).max()
    scale = (np.abs(d) @ np.abs(w)).max() + 1
    assert np.abs(dX0.cpu().numpy() - d @ w).max() <= tol * scale
    assert np.abs(dX.cpu().numpy() - (d @ w) * (1 - x * x)).max() <= tol * scale


@pytest.mark.parametrize("n_in", [1, 66])
@pytest.mark.parametrize("batch", [8, 9, 127, 128, 129, 256, 300])
def test_gradients_of_a_one_output_layer(batch, n_in):
    """One output: the batch is contiguous along both indices of dY."""
    test_layer_and_input_gradients(batch, 1, n_in)


def test_adam_over_many_tensors_equals_one_at_a_time():
    torch = pytest.importorskip("torch")
    from nla3d_gb300 import _lib
    lib = _lib.load()
    sizes = [1, 255, 256, 257, 66 * 256] + [3] * 14          # 19 tensors: two launches
    rng = np.random.default_rng(0)
    make = lambda s: torch.from_numpy(s.astype(np.float32)).cuda()  # noqa: E731
    w = [make(rng.normal(size=n)) for n in sizes]
    g = [make(rng.normal(size=n)) for n in sizes]
    m = [make(rng.normal(size=n)) for n in sizes]
    v = [make(rng.random(size=n)) for n in sizes]
    b = [torch.zeros(n, dtype=torch.bfloat16).cuda() if k % 2 else None
         for k, n in enumerate(sizes)]
    ref = [[t.clone() for t in ts] for ts in (w, m, v)]
    rb = [None if t is None else t.clone() for t in b]
    torch.cuda.synchronize()
    for k, n in enumerate(sizes):
        assert lib.nla3d_mlp_adam(ref[0][k].data_ptr(), g[k].data_ptr(), ref[1][k].data_ptr(),
                                  ref[2][k].data_ptr(), n, 1e-3, 0.9, 0.999, 1e-8, 3,
                                  None if rb[k] is None else rb[k].data_ptr(), None) == 0
    ptr = lambda ts: (ctypes.c_void_p * len(ts))(  # noqa: E731
        *[None if t is None else t.data_ptr() for t in ts])
    assert lib.nla3d_mlp_adam_multi(len(sizes), ptr(w), ptr(g), ptr(m), ptr(v),
                                    (ctypes.c_int64 * len(sizes))(*sizes), ptr(b), 1e-3, 0.9,
                                    0.999, 1e-8, 3, None) == 0
    torch.cuda.synchronize()
    for got, want in zip((w, m, v, [t for t in b if t is not None]),
                         (*ref, [t for t in rb if t is not None])):
        for x, y in zip(got, want):
            assert torch.equal(x, y)
