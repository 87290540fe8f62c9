"""The work that users of this framework have it do, as measurable cases.

A case is one of six kinds of call, each through the package's public entry
points:

  assemble    one Newton iteration's assembly: vecU in, updateResults,
              assembleGlobalEqMatrices, K and F on the device; with
              "newton" also the right-hand side, residual and reaction
              products on the assembled blocks
  batch       the same for many meshes of uneven size in one context,
              replayed as the captured graph
  to_host     assembly with host buffers: vecU from the host, K and F to it
  solve       the equation solver on the assembled K(2): factorise and solve
              one right-hand side to a residual
  solve_batch the same for a block-diagonal system of equal meshes
  mlp         one training step of the learned Newton start's network
"""
import math

import numpy as np
import torch

from nla3d_gb300 import meshgen as mg

MATERIALS = {"nh": mg.MAT_NEO_HOOKEAN, "mr": mg.MAT_MOONEY_RIVLIN, "bid": mg.MAT_BIDERMAN}
CONSTANTS = {"nh": (1.0, 1000.0), "mr": (0.4, 0.1, 2000.0), "bid": (0.4, 0.05, 0.01, 0.1, 2000.0)}
MLP_SIZES = (132, 256, 256, 256, 256, 66)


def listed():
    return [
        # the smallest model of the benchmark: 1,000 elements, every launch's latency counts
        dict(name="cube10_fp64", kind="assemble", nx=10, ny=10, nz=10, precision="fp64",
             material="nh", state="stretch", clamp=False, jitter=0.0, mpc=False, newton=False),
        # a Newton iteration of a ragged, distorted bar with a rigid-body end: assembly, MPC rows
        # and the sparse products either side of the solve
        dict(name="bar_newton_fp64", kind="assemble", nx=9, ny=11, nz=43, precision="fp64",
             material="nh", state="twist", clamp=True, jitter=0.1, mpc=True, newton=True),
        # the large single mesh, 1e6 elements, in both precisions
        dict(name="block100_fp64", kind="assemble", nx=100, ny=100, nz=100, precision="fp64",
             material="mr", state="twist", clamp=False, jitter=0.0, mpc=False, newton=False),
        dict(name="block100_mixed", kind="assemble", nx=100, ny=100, nz=100, precision="mixed",
             material="mr", state="twist", clamp=False, jitter=0.0, mpc=False, newton=False),
        # parameter studies: many small uneven meshes, each with its own material
        dict(name="batch_mixed_graph", kind="batch", meshes=96, lo=4, hi=40, precision="mixed"),
        # a host program that owns K and F (the reference's own data flow)
        dict(name="to_host_60_fp64", kind="to_host", nx=60, ny=60, nz=60, precision="fp64",
             material="bid", state="twist", clamp=True, jitter=0.0),
        # plane strain: the four-node element of the 2D benchmark model
        dict(name="plane41_fp64", kind="assemble", nx=231, ny=173, nz=0, precision="fp64",
             material="mr", state="stretch", clamp=True, jitter=0.1, mpc=False, newton=False),
        # the solver with FP64 fronts on a small block (the linear drivers' and tests' size)
        dict(name="solve_block12_fp64", kind="solve", nx=12, ny=12, nz=12, fronts="fp64",
             material="mr", mpc=False),
        # the torsion bar of the Newton study, and the same bar refined
        dict(name="solve_bar20_tc", kind="solve", nx=20, ny=20, nz=80, fronts="fp32-tc",
             material="nh", mpc=True),
        dict(name="solve_bar30_tc", kind="solve", nx=30, ny=30, nz=120, fronts="fp32-tc",
             material="nh", mpc=True),
        # the lock-step training-set solves: copies of one block, different materials
        dict(name="solve_batch_fp32", kind="solve_batch", n=12, copies=24, fronts="fp32"),
        # one step of the network's training at its usual batch
        dict(name="mlp_train_256", kind="mlp", batch=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "plane", "batch", "to_host", "solve",
                       "solve", "solve_batch", "mlp"])
    material = rng.choice(["nh", "mr", "bid"])
    if kind in ("assemble", "to_host"):
        while True:
            n = [_log_int(rng, 5, 140) for _ in range(3)]
            if 200 <= n[0] * n[1] * n[2] <= (1000000 if kind == "assemble" else 216000):
                break
        c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], precision=rng.choice(["fp64", "mixed"]),
                 material=material, state=rng.choice(["stretch", "twist"]),
                 clamp=rng.random() < 0.7, jitter=rng.choice([0.0, 0.1]))
        if kind == "assemble":
            c["mpc"] = c["clamp"] and n[0] * n[1] * n[2] < 30000 and rng.random() < 0.6
            c["newton"] = c["clamp"] and n[0] * n[1] * n[2] < 30000 and rng.random() < 0.6
        return c
    if kind == "plane":
        return dict(kind="assemble", nx=_log_int(rng, 20, 400), ny=_log_int(rng, 20, 400), nz=0,
                    precision="fp64", material=material, state="stretch", clamp=rng.random() < 0.5,
                    jitter=rng.choice([0.0, 0.1]), mpc=False, newton=False)
    if kind == "batch":
        return dict(kind="batch", meshes=_log_int(rng, 8, 96), lo=rng.randint(3, 6),
                    hi=rng.randint(12, 40), precision=rng.choice(["fp64", "mixed"]))
    if kind == "solve":
        fronts = rng.choice(["fp64", "fp32", "fp32-tc"])
        s = _log_int(rng, 6, 13 if fronts == "fp64" else 24)
        return dict(kind="solve", nx=s, ny=s + rng.randint(0, 3), nz=s * rng.randint(1, 3),
                    fronts=fronts, material=material, mpc=rng.random() < 0.5)
    if kind == "solve_batch":
        return dict(kind="solve_batch", n=rng.randint(6, 14), copies=_log_int(rng, 4, 24),
                    fronts=rng.choice(["fp32", "fp64"]))
    return dict(kind="mlp", batch=_log_int(rng, 32, 2048))


# ---------------------------------------------------------------------------
# models as plain arrays (shared by prepare and exact)
# ---------------------------------------------------------------------------

def _grid(nx, ny, nz, h):
    """Nodes and elements (1-based) of a hexahedral block, or of a plate for nz = 0."""
    i, j, k = np.arange(nx + 1.0), np.arange(ny + 1.0), np.arange(nz + 1.0)
    kk, jj, ii = np.meshgrid(k, j, i, indexing="ij")
    xyz = np.stack([ii.ravel(), jj.ravel(), kk.ravel()], axis=1) * h
    ek, ej, ei = np.meshgrid(np.arange(max(nz, 1)), np.arange(ny), np.arange(nx), indexing="ij")
    n0 = (1 + ei + (nx + 1) * (ej + (ny + 1) * ek)).ravel()
    quad = np.array([0, 1, nx + 2, nx + 1])
    local = quad if nz == 0 else np.concatenate([quad, quad + (nx + 1) * (ny + 1)])
    return xyz, (n0[:, None] + local[None, :]).astype(np.uint32)


def _model(nx, ny, nz, material, constants, clamp, jitter, mpc, fix_master, rng, h=None):
    h = 1.0 / max(nx, ny, nz) if h is None else h
    xyz, conn = _grid(nx, ny, nz, h)
    dims = 2 if nz == 0 else 3
    axis = dims - 1                      # the axis that carries the load
    ends = (xyz[:, axis] < 1e-9 * h, xyz[:, axis] > xyz[:, axis].max() - 1e-9 * h)
    base, top = np.nonzero(ends[0])[0] + 1, np.nonzero(ends[1])[0] + 1
    if jitter:
        free = ~(ends[0] | ends[1])
        xyz[free, :dims] += rng.uniform(-jitter * h, jitter * h, (int(free.sum()), dims))
    m = dict(xyz=xyz, conn=conn, dims=dims, h=h, material=material, constants=constants, top=top,
             fix_nodes=np.zeros(0, np.uint32), fix_dofs=np.zeros(0, np.int32), master=0)
    if clamp:
        m["fix_nodes"] = np.repeat(base, dims).astype(np.uint32)
        m["fix_dofs"] = np.tile(np.arange(dims, dtype=np.int32), base.size)
    if mpc:
        centre = xyz[top - 1].mean(axis=0)
        m["xyz"] = np.vstack([xyz, centre[None]])
        m["master"] = m["xyz"].shape[0]
        if fix_master:
            m["fix_nodes"] = np.r_[m["fix_nodes"], np.full(6, m["master"])].astype(np.uint32)
            m["fix_dofs"] = np.r_[m["fix_dofs"], np.arange(6)].astype(np.int32)
    return m


def _mesh(m):
    mesh = mg.Mesh(mg.ELEM_PLANE41 if m["dims"] == 2 else mg.ELEM_SOLID81, m["xyz"], m["conn"],
                   mat_id=MATERIALS[m["material"]], mat_c=m["constants"])
    if m["fix_nodes"].size:
        mesh.fix_nodes, mesh.fix_dofs = m["fix_nodes"], m["fix_dofs"]
    if m["master"]:
        mesh.rigid_bodies.append(mg.RigidBody(m["master"], m["top"].astype(np.uint32)))
    return mesh


def _numbering(m):
    """Equation numbers (1-based): constrained DoFs first, then the element pressures, the free
    node DoFs node by node, and the MPC equations."""
    N, E = m["xyz"].shape[0], m["conn"].shape[0]
    used = np.zeros((N, 6), bool)
    used[: N - 1 if m["master"] else N, : m["dims"]] = True
    if m["master"]:
        used[m["master"] - 1] = True
    fixed = np.zeros((N, 6), bool)
    fixed[m["fix_nodes"].astype(np.int64) - 1, m["fix_dofs"]] = True
    nc = int(fixed.sum())
    eq = np.zeros((N, 6), np.int64)
    eq[fixed] = 1 + np.arange(nc)
    free = used & ~fixed
    eq[free] = nc + E + 1 + np.arange(int(free.sum()))
    n_dofs = E + int(used.sum())
    n_mpc = 3 * m["top"].size if m["master"] else 0
    return dict(node=eq, p=nc + 1 + np.arange(E), nc=nc, n_unk=n_dofs - nc, n_mpc=n_mpc,
                n=n_dofs + n_mpc, mpc=n_dofs + 1 + np.arange(n_mpc))


def _state(m, num, kind, rng, scale=1.0):
    """vecU of a deformed state with seeded noise (displacements, pressures, multipliers)."""
    x, h, dims = m["xyz"], m["h"], m["dims"]
    u = np.zeros_like(x)
    L = x[:, dims - 1].max()
    angle = 0.0
    if kind == "twist":
        angle = scale * math.pi / 6
        th = angle * x[:, 2] / L
        c = 0.5 * (x[:, :2].min(axis=0) + x[:, :2].max(axis=0))
        d = x[:, :2] - c
        u[:, 0] = np.cos(th) * d[:, 0] - np.sin(th) * d[:, 1] - d[:, 0]
        u[:, 1] = np.sin(th) * d[:, 0] + np.cos(th) * d[:, 1] - d[:, 1]
        u[:, 2] = 0.5 * scale * x[:, 2]
        noise = 0.005
    else:
        u[:, dims - 1] = 0.2 * scale * x[:, dims - 1]
        noise = 0.01
    u[:, :dims] += rng.uniform(-noise * h, noise * h, (x.shape[0], dims))
    full = np.zeros((x.shape[0], 6))
    full[:, :3] = u
    if m["master"]:
        full[m["master"] - 1, 5] = angle
    U = np.zeros(num["n"])
    sel = num["node"] > 0
    U[num["node"][sel] - 1] = full[sel]
    U[num["p"] - 1] = rng.normal(0.0, 0.1, num["p"].size)
    if num["n_mpc"]:
        U[num["mpc"] - 1] = rng.normal(0.0, 0.1, num["n_mpc"]) * h * h
    return U


def _assembly_problem(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    m = _model(case["nx"], case["ny"], case["nz"], case["material"], CONSTANTS[case["material"]],
               case["clamp"], case["jitter"], case.get("mpc", False), False, rng)
    num = _numbering(m)
    U = _state(m, num, case["state"], rng)
    out = dict(m=m, num=num, U=U)
    if case.get("newton"):
        out["dUc"] = 1e-3 * m["h"] * rng.standard_normal(num["nc"])
        out["dUsl"] = 1e-3 * m["h"] * rng.standard_normal(num["n"] - num["nc"])
    return out


def _batch_problems(case, seed):
    """Side lengths are the case's own (log-uniform); materials and states the seed's."""
    shape = np.random.default_rng([case["meshes"], case["lo"], case["hi"]])
    rng = np.random.default_rng([seed, case["meshes"]])
    out = []
    for _ in range(case["meshes"]):
        n = np.rint(np.exp(shape.uniform(math.log(case["lo"]), math.log(case["hi"]), 3)))
        c10 = rng.uniform(0.2, 1.0)
        m = _model(*(int(v) for v in n), "nh", (2 * c10, c10 * rng.uniform(500.0, 5000.0)), False,
                   0.0, False, False, rng)
        num = _numbering(m)
        out.append(dict(m=m, num=num, U=_state(m, num, "stretch", rng, rng.uniform(0.5, 4.0))))
    return out


def _increment(m, num, rng):
    """A solution of the linear system as Newton meets it: a smooth displacement increment with
    some noise, pressures and multipliers of its scale."""
    x = _state(m, num, "twist", rng, 0.02)[num["nc"]:]
    return 10.0 * x / np.abs(x).max()


def _solve_problem(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    m = _model(case["nx"], case["ny"], case["nz"], case["material"], CONSTANTS[case["material"]],
               True, 0.0, case["mpc"], case["mpc"], rng, h=1.0 if case["mpc"] else None)
    num = _numbering(m)
    return dict(m=m, num=num, U=_state(m, num, "twist", rng, 0.3), x=_increment(m, num, rng))


def _solve_batch_problems(case, seed):
    rng = np.random.default_rng([seed, case["n"], case["copies"]])
    out = []
    for _ in range(case["copies"]):
        c10, k, s = rng.uniform(0.2, 1.0), rng.uniform(500.0, 5000.0), rng.uniform(1.0, 2.0)
        m = _model(case["n"], case["n"], case["n"], "nh", (2 * c10, k), True, 0.0, False, False, rng)
        m["fix_nodes"] = np.r_[m["fix_nodes"], m["top"]].astype(np.uint32)
        m["fix_dofs"] = np.r_[m["fix_dofs"], np.full(m["top"].size, 2)].astype(np.int32)
        num = _numbering(m)
        out.append(dict(m=m, num=num, U=_state(m, num, "stretch", rng, 2.0 * (s - 1.0)),
                        x=_increment(m, num, rng)))
    return out


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

class _Array:
    """Device memory of the library as a tensor (not owned)."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<f8", "strides": None,
                                         "data": (int(ptr), False), "version": 2}


def _view(ptr, n, keep):
    t = torch.as_tensor(_Array(ptr, n), device="cuda")
    t._keep = keep
    return t


def _device_K_F(s, lib, h):
    import ctypes
    p, n = ctypes.c_void_p(), ctypes.c_uint64()
    assert lib.nla3d_device_K(h, 0, ctypes.byref(p), ctypes.byref(n)) == 0
    K = _view(p.value, n.value, s)
    assert lib.nla3d_device_F(h, ctypes.byref(p), ctypes.byref(n)) == 0
    return K, _view(p.value, n.value, s)


def _symmetric_product(io, co, values, x):
    """b = A x of a symmetric matrix held as its upper CSR (1-based), fixed-order sums."""
    io, co = (torch.as_tensor(v.astype(np.int64), device="cuda") for v in (io, co))
    n = io.numel() - 1
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), io[1:] - io[:-1])
    col = co - 1
    off = row != col
    r, c = torch.cat([row, col[off]]), torch.cat([col, row[off]])
    order = torch.argsort(r * n + c)
    r, c, v = r[order], c[order], torch.cat([values, values[off]])[order]
    counts = torch.bincount(r, minlength=n)
    return torch.segment_reduce(v * x[c], "sum", lengths=counts, initial=0.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        from nla3d_gb300.learned import MLP
        X, T = _mlp_data(case, seed)
        return dict(kind=kind, mlp=MLP(MLP_SIZES, seed=seed % 1000), X=torch.from_numpy(X).cuda(),
                    T=torch.from_numpy(T).cuda())
    stream = torch.cuda.Stream()
    if kind == "batch":
        from nla3d_gb300.batch import BatchAssembly
        pbs = _batch_problems(case, seed)
        ba = BatchAssembly([_mesh(p["m"]) for p in pbs], case["precision"],
                           stream=stream.cuda_stream).init()
        U = torch.from_numpy(np.concatenate([p["U"] for p in pbs])).cuda()
        torch.cuda.synchronize()
        ba.set_U_device(U.data_ptr(), U.numel())
        ba.update()
        ba.assemble()
        ba.capture_graph()
        ba.synchronize()
        return dict(kind=kind, ba=ba, U=U, stream=stream, out=_device_K_F(ba, ba.lib, ba.h))
    if kind == "solve_batch":
        return _prepare_solve_batch(case, seed, stream)
    from nla3d_gb300.storage import FEStorage
    pb = _solve_problem(case, seed) if kind == "solve" else _assembly_problem(case, seed)
    s = FEStorage(_mesh(pb["m"]), case.get("precision", "fp64"),
                  stream=stream.cuda_stream).initSolutionData()
    num = pb["num"]
    assert (s.n_con, s.n_unk, s.n_mpc, s.n_total) == (num["nc"], num["n_unk"], num["n_mpc"], num["n"])
    st = dict(kind=kind, s=s, stream=stream, num=num)
    if kind == "to_host":
        st["U"] = torch.from_numpy(pb["U"]).pin_memory()
        st["host"] = [torch.empty(n, dtype=torch.float64).pin_memory()
                      for n in [s.blocks[b][2] for b in (1, 12, 2)] + [s.n_total]]
        st["np"] = [t.numpy() for t in st["host"]]
        return st
    st["U"] = torch.from_numpy(pb["U"]).cuda()
    st["out"] = _device_K_F(s, s.lib, s.h)
    if kind == "assemble":
        for k in ("dUc", "dUsl"):
            if k in pb:
                st[k] = torch.from_numpy(pb[k]).cuda()
        torch.cuda.synchronize()
        return st
    from nla3d_gb300.ldlt import DeviceLDLT, fill_reducing_order
    from nla3d_gb300.newton import row_points
    torch.cuda.synchronize()
    s.setU_device(st["U"].data_ptr(), s.n_total)
    s.updateResults()
    s.assembleGlobalEqMatrices()
    s.synchronize()
    io, co = s.pattern(2)
    order = fill_reducing_order(io, co, row_points(s, s.n_con, s.n_unk, s.n_mpc), s.n_unk)
    st["ldlt"] = DeviceLDLT.for_storage(s, order, case["fronts"])
    st["values"], n2 = s.device_K(2)
    st["tol"] = 1e-13 if case["fronts"] == "fp64" else 1e-12
    st["b"] = _symmetric_product(io, co, _view(st["values"], n2, s), torch.from_numpy(pb["x"]).cuda())
    st["x"] = torch.empty_like(st["b"])
    torch.cuda.synchronize()
    return st


def _prepare_solve_batch(case, seed, stream):
    from nla3d_gb300.batch import BatchAssembly
    from nla3d_gb300.batch_newton import BlockSolver
    from nla3d_gb300.ldlt import fill_reducing_order
    pbs = _solve_batch_problems(case, seed)
    ba = BatchAssembly([_mesh(p["m"]) for p in pbs], "fp64", stream=stream.cuda_stream).init()
    U = torch.from_numpy(np.concatenate([p["U"] for p in pbs])).cuda()
    torch.cuda.synchronize()
    ba.set_U_device(U.data_ptr(), U.numel())
    ba.update()
    ba.assemble()
    ba.synchronize()
    io, co = ba.pattern(0, 2)
    m, num = pbs[0]["m"], pbs[0]["num"]
    pts = np.zeros((num["n"] - num["nc"], 3))
    for d in range(3):
        sel = num["node"][:, d] > num["nc"]
        pts[num["node"][sel, d] - num["nc"] - 1] = m["xyz"][sel]
    pts[num["p"] - num["nc"] - 1] = m["xyz"][m["conn"].astype(np.int64) - 1].mean(axis=1)
    bs = BlockSolver(io, co, fill_reducing_order(io, co, pts, num["n_unk"]), case["copies"],
                     case["fronts"], stream)
    K, _ = _device_K_F(ba, ba.lib, ba.h)
    n1, n12, n2 = (int(ba.info[0, k]) for k in (6, 9, 12))
    values = torch.cat([K[int(o) + n1 + n12: int(o) + n1 + n12 + n2] for o in ba.k_off[:-1]])
    b = torch.cat([_symmetric_product(io, co, values[k * n2:(k + 1) * n2],
                                      torch.from_numpy(p["x"]).cuda()) for k, p in enumerate(pbs)])
    # as the lock-step driver has them: each problem's right-hand side of unit norm
    scale = torch.linalg.vector_norm(b.view(case["copies"], -1), dim=1)
    st = dict(kind="solve", ldlt=bs.ldlt, bs=bs, values=values.data_ptr(), v=values, stream=stream,
              b=(b.view(case["copies"], -1) / scale[:, None]).ravel(), scale=scale,
              tol=(1e-13 if case["fronts"] == "fp64" else 1e-12))
    st["x"] = torch.empty_like(st["b"])
    torch.cuda.synchronize()
    ba.close()
    return st


def run(st):
    kind = st["kind"]
    if kind == "mlp":
        mlp = st["mlp"]
        acts = mlp.forward(st["X"])
        gW, gb = mlp.backward(acts, mlp.loss_grad(acts[-1], st["T"]))
        mlp.adam(gW, gb, lr=1e-3)
        return dict(out=acts[-1], gW=gW, gb=gb, W=mlp.W, b=mlp.b)
    if kind == "batch":
        st["ba"].set_U_device(st["U"].data_ptr(), st["U"].numel())
        st["ba"].graph_launch()
        return st["out"]
    if kind == "solve":
        st["ldlt"].factor_device(st["values"])
        st["ldlt"].solve_device(st["values"], st["b"].data_ptr(), st["x"].data_ptr(), max_refine=100,
                                tol=st["tol"])
        if "scale" not in st:
            return st["x"]
        with torch.cuda.stream(st["stream"]):
            return (st["x"].view(st["scale"].numel(), -1) * st["scale"][:, None]).ravel()
    s = st["s"]
    if kind == "to_host":
        s.setU(st["U"].numpy())
        s.updateResults()
        s.assemble_to_host(*st["np"])
        return st["np"]
    s.setU_device(st["U"].data_ptr(), s.n_total)
    s.updateResults()
    s.assembleGlobalEqMatrices()
    if "dUc" not in st:
        return st["out"]
    nc, K, F = s.n_con, *st["out"]
    with torch.cuda.stream(st["stream"]):
        rhs = F[nc:].clone()
        s.block_mv_device(12, 1, st["dUc"].data_ptr(), -1.0, rhs.data_ptr())
        res = rhs.clone()
        if s.n_mpc:
            lam = torch.zeros_like(rhs)
            lam[s.n_unk:] = st["U"][nc + s.n_unk:]
            s.block_mv_device(2, 0, lam.data_ptr(), -1.0, res.data_ptr())
        reac = torch.zeros(nc, dtype=torch.float64, device="cuda")
        s.block_mv_device(1, 0, st["dUc"].data_ptr(), 1.0, reac.data_ptr())
        s.block_mv_device(12, 0, st["dUsl"].data_ptr(), 1.0, reac.data_ptr())
        reac -= F[:nc]
    return [K, F, rhs, res, reac]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def _solve_work(n, fronts, copies=1):
    # three-dimensional nested dissection: about 12.4 n^2 flop and 16.6 n^(4/3) factor entries,
    # written once and read by one forward and one backward substitution; K read once (30 a row)
    size = 8 if fronts == "fp64" else 4
    return {"bytes": copies * (n * 30 * 8 + 3 * size * 16.6 * n ** (4 / 3) + 16 * n),
            "flops": copies * (12.4 * n * n + 4 * 16.6 * n ** (4 / 3))}


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        p = sum(a * b + b for a, b in zip(MLP_SIZES[:-1], MLP_SIZES[1:]))
        w = sum(a * b for a, b in zip(MLP_SIZES[:-1], MLP_SIZES[1:]))
        B = case["batch"]
        first = MLP_SIZES[0] * MLP_SIZES[1]
        # weights and moments read and written, gradients written; data read, output written
        return {"bytes": 4 * p * 7 + 2 * w * 2 + 4 * B * (MLP_SIZES[0] + 2 * MLP_SIZES[-1]),
                "flops": 2 * B * (3 * w - first) + 12 * p}
    if kind == "solve":
        e = case["nx"] * case["ny"] * case["nz"]
        n = e + 3 * (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + (1 if case["mpc"] else 0))
        return _solve_work(n, case["fronts"])
    if kind == "solve_batch":
        c = case["n"]
        return _solve_work(c ** 3 + 3 * (c + 1) ** 2 * c - (c + 1) ** 2, case["fronts"], case["copies"])
    if kind == "batch":
        shape = np.random.default_rng([case["meshes"], case["lo"], case["hi"]])
        sides = [[int(v) for v in np.rint(np.exp(shape.uniform(math.log(case["lo"]),
                                                               math.log(case["hi"]), 3)))]
                 for _ in range(case["meshes"])]
    else:
        sides = [[case["nx"], case["ny"], case["nz"]]]
    total = {"bytes": 0.0, "flops": 0.0}
    for nx, ny, nz in sides:
        if nz:
            E, N = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
            # node pairs that share an element, each once, 9 values (6 on the diagonal)
            pairs = ((3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1) - N) / 2
            nnz, npe, dims, per = 9 * pairs + 6 * N + 25 * E, 8, 3, 12000
        else:
            E, N = nx * ny, (nx + 1) * (ny + 1)
            pairs = ((3 * nx + 1) * (3 * ny + 1) - N) / 2
            nnz, npe, dims, per = 4 * pairs + 3 * N + 9 * E, 4, 2, 1500
        n = dims * N + E
        # connectivity, coordinates, vecU in; K and F out
        total["bytes"] += 4 * npe * E + 8 * dims * N + 8 * n + 8 * (nnz + n)
        total["flops"] += per * E
        if case.get("newton"):
            total["bytes"] += 8 * 2 * nnz
            total["flops"] += 4 * nnz
    return total


# ---------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------

def _shape_derivatives(dims):
    """dN/dxi at the 2^dims Gauss points: (points, nodes, dims)."""
    a = 1.0 / math.sqrt(3.0)
    corners = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                        [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)[: 2 ** dims, :dims]
    pts = np.array([[(a if g >> d & 1 else -a) for d in range(dims)] for g in range(2 ** dims)])
    out = np.zeros((2 ** dims, 2 ** dims, dims))
    for g, xi in enumerate(pts):
        f = 1.0 + corners * xi
        for d in range(dims):
            rest = np.prod(np.delete(f, d, axis=1), axis=1)
            out[g, :, d] = corners[:, d] * rest / 2 ** dims
    return torch.as_tensor(out, device="cuda")


def _elements(m, num, U, e0, e1):
    """K and F contributions of elements e0 .. e1: equation pairs and values."""
    dims, dev = m["dims"], "cuda"
    conn = torch.as_tensor(m["conn"][e0:e1].astype(np.int64), device=dev) - 1
    X = torch.as_tensor(m["xyz"][:, :dims], device=dev)[conn]
    eq = torch.as_tensor(num["node"][:, :dims], device=dev)[conn]          # (E, nodes, dims)
    peq = torch.as_tensor(num["p"][e0:e1], device=dev)
    u, p = U[eq - 1], U[peq - 1]
    dN = _shape_derivatives(dims)
    Jm = torch.einsum("gni,enj->egij", dN, X - X[:, :1])
    w = torch.linalg.det(Jm)
    G = torch.einsum("egij,gnj->egni", torch.linalg.inv(Jm), dN)           # (E, g, nodes, dims)
    H = torch.einsum("eni,egnj->egij", u - u[:, :1], G)
    F = torch.eye(3, dtype=torch.float64, device=dev).repeat(*w.shape, 1, 1)
    F[..., :dims, :dims] += H
    C = F.transpose(-1, -2) @ F
    I = torch.eye(3, dtype=torch.float64, device=dev)
    I1 = C.diagonal(dim1=-2, dim2=-1).sum(-1)
    I2 = 0.5 * (I1 ** 2 - (C * C).sum((-1, -2)))
    J = torch.linalg.det(F)
    Ci = torch.linalg.inv(C)
    c = m["constants"]
    pp, pppp = J ** (-2.0 / 3.0), J ** (-4.0 / 3.0)
    a2, a11 = torch.zeros_like(J), torch.zeros_like(J)
    if m["material"] == "nh":
        a1, kb = torch.full_like(J, 0.5 * c[0]), c[1]
    elif m["material"] == "mr":
        a1, a2, kb = torch.full_like(J, c[0]), torch.full_like(J, c[1]), c[2]
    else:
        d = I1 * pp - 3.0
        a1, a2, a11, kb = c[0] + 2 * c[1] * d + 3 * c[2] * d * d, torch.full_like(J, c[3]), \
            2 * c[1] + 6 * c[2] * d, c[4]
    q = lambda v: v[..., None, None]  # noqa: E731
    A = I - q(I1 / 3) * Ci
    B = q(I1) * I - C - q(2 * I2 / 3) * Ci
    pj = p[:, None] * J
    S = q(2 * a1 * pp) * A + q(2 * a2 * pppp) * B + q(pj) * Ci
    k11, k1, k2 = 4 * a11 * pppp, 4 / 3 * a1 * pp, 8 / 3 * a2 * pppp
    P = q(k11) * A - q(k1) * Ci
    R = -q(k1) * A - q(k2) * B + q(pj - k1 * I1 / 3 - k2 * 2 * I2 / 3) * Ci
    o = lambda x, y: torch.einsum("egij,egkl->egijkl", x, y)  # noqa: E731
    s = lambda x: 0.5 * (torch.einsum("egik,egjl->egijkl", x, x) +  # noqa: E731
                         torch.einsum("egil,egjk->egijkl", x, x))
    q4 = lambda v: v[..., None, None, None, None]  # noqa: E731
    II = I.expand_as(C)
    D = o(A, P) - q4(k2) * o(B, Ci) + o(Ci, R) - q4(2 * pj - k1 * I1 - k2 * I2) * s(Ci) \
        + q4(1.5 * k2) * (o(II, II) - s(II))
    T = torch.einsum("egij,egjlmn,egkm->egilkn", F, D, F)
    T = T + torch.einsum("ik,egln->egilkn", I, S)
    Kuu = torch.einsum("eg,egal,egilkn,egbn->eaibk", w, G, T[:, :, :dims, :dims, :dims, :dims], G)
    Finv = torch.linalg.inv(F)[..., :dims, :dims]
    Kup = torch.einsum("eg,egji,egaj->eai", w * J, Finv, G)
    Fu = -torch.einsum("eg,egij,egaj->eai", w, (F @ S)[..., :dims, :dims], G)
    E, nn = conn.shape
    nd = nn * dims
    r, cc = torch.triu_indices(nd, nd, device=dev)
    fe = eq.reshape(E, nd)
    pairs = [(fe[:, r], fe[:, cc], Kuu.reshape(E, nd, nd)[:, r, cc]),
             (fe, peq[:, None].expand(E, nd), Kup.reshape(E, nd)),
             (peq[:, None], peq[:, None], -(w.sum(1) / kb)[:, None])]
    rows, cols, vals = (torch.cat([t[k] for t in pairs], dim=1).reshape(-1) for k in range(3))
    f = torch.zeros(num["n"], dtype=torch.float64, device=dev)
    f.index_add_(0, fe.reshape(-1) - 1, Fu.reshape(-1))
    f[peq - 1] = -((J - 1 - p[:, None] / kb) * w).sum(1)
    return torch.minimum(rows, cols), torch.maximum(rows, cols), vals, f


def _rigid_rows(m, num, U):
    """Rows of the rigid-body equations u_s = u_m + (C(theta) - I)(x_s - x_m)."""
    U = U.cpu().numpy()
    mast, top = m["master"] - 1, m["top"] - 1
    me = num["node"][mast]
    w0, th = U[me[:3] - 1], U[me[3:] - 1]
    t = float(np.linalg.norm(th))
    eps = np.zeros((3, 3, 3))
    for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        eps[i, j, k], eps[i, k, j] = 1.0, -1.0
    sn, cs = math.sin(t), math.cos(t)
    c1, c2, c3, c4 = ((1.0, 0.5, -1 / 3, -1 / 12) if t < 1e-3 else
                      (sn / t, (1 - cs) / t ** 2, (t * cs - sn) / t ** 3,
                       (t * sn - 2 + 2 * cs) / t ** 4))
    spin = np.einsum("imj,m->ij", eps, th)
    I = np.eye(3)
    C = cs * I + c1 * spin + c2 * np.outer(th, th)
    dC = (-c1 * np.einsum("ij,l->ijl", I, th) + c3 * np.einsum("l,ij->ijl", th, spin)
          + c1 * np.einsum("ilj->ijl", eps) + c4 * np.einsum("l,i,j->ijl", th, th, th)
          + c2 * (np.einsum("il,j->ijl", I, th) + np.einsum("i,jl->ijl", th, I)))
    rows, cols, vals, f = [], [], [], np.zeros(num["n"])
    for k, s in enumerate(top):
        d = m["xyz"][s] - m["xyz"][mast]
        for i in range(3):
            e = int(num["mpc"][3 * k + i])
            terms = [(num["node"][s, i], 1.0), (me[i], -1.0)] + \
                    [(me[3 + l], -float(dC[i, :, l] @ d)) for l in range(3)]
            for q, v in terms:
                rows.append(min(int(q), e)), cols.append(max(int(q), e)), vals.append(v)
            f[e - 1] = w0[i] + (C[i] - I[i]) @ d - U[num["node"][s, i] - 1]
    dev = "cuda"
    return (torch.tensor(rows, device=dev), torch.tensor(cols, device=dev),
            torch.tensor(vals, dtype=torch.float64, device=dev), torch.as_tensor(f, device=dev))


def _assembled(pb):
    """K as (rows, cols, values) in storage order: block(1), block(1,2), block(2); and F."""
    m, num = pb["m"], pb["num"]
    U = torch.as_tensor(pb["U"], device="cuda")
    E, n, nc = m["conn"].shape[0], num["n"], num["nc"]
    keys, vals = [], []
    F = torch.zeros(n, dtype=torch.float64, device="cuda")

    def add(r, c, v, f):
        nonlocal F
        blk = (r > nc).long() + (c > nc).long()
        keys.append((blk * (n + 1) + r) * (n + 1) + c)
        vals.append(v)
        F = F + f

    for e0 in range(0, E, 40000):
        add(*_elements(m, num, U, e0, min(E, e0 + 40000)))
    if m["master"]:
        add(*_rigid_rows(m, num, U))
    keys, vals = torch.cat(keys), torch.cat(vals)
    keys, order = torch.sort(keys)
    vals = vals[order]
    del order
    first = torch.ones_like(keys, dtype=torch.bool)
    first[1:] = keys[1:] != keys[:-1]
    start = torch.nonzero(first).ravel()
    counts = torch.diff(start, append=torch.tensor([keys.numel()], device="cuda"))
    V = torch.segment_reduce(vals, "sum", lengths=counts)
    keys = keys[start]
    return (keys // (n + 1)) % (n + 1), keys % (n + 1), V, F


def _mlp_data(case, seed):
    rng = np.random.default_rng([seed, case["batch"]])
    return (rng.standard_normal((case["batch"], MLP_SIZES[0])).astype(np.float32),
            rng.standard_normal((case["batch"], MLP_SIZES[-1])).astype(np.float32))


def _mlp_exact(case, seed):
    rng = np.random.default_rng(seed % 1000)
    W = []
    for i, o in zip(MLP_SIZES[:-1], MLP_SIZES[1:]):
        lim = math.sqrt(6.0 / (i + o))
        W.append(rng.uniform(-lim, lim, (o, i)).astype(np.float32))
    X, T = (v.astype(np.float64) for v in _mlp_data(case, seed))
    Wb = [torch.from_numpy(w).to(torch.bfloat16).double().numpy() for w in W]
    acts = [X]
    for l, w in enumerate(Wb):
        z = acts[-1] @ w.T
        acts.append(np.tanh(z) if l < len(Wb) - 1 else z)
    d = 2.0 * (acts[-1] - T) / T.size
    gW, gb = [None] * len(W), [None] * len(W)
    for l in range(len(W) - 1, -1, -1):
        if l < len(W) - 1:
            d = d * (1.0 - acts[l + 1] ** 2)
        gW[l], gb[l] = d.T @ acts[l], d.sum(axis=0)
        d = d @ Wb[l]
    step = lambda g: 1e-3 * g / (np.abs(g) + 1e-8)  # noqa: E731  (the first Adam step)
    return dict(out=acts[-1], gW=gW, gb=gb, W=[w.astype(np.float64) - step(g) for w, g in zip(W, gW)],
                b=[-step(g) for g in gb])


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _mlp_exact(case, seed)
    if kind == "solve":
        # the right-hand side is the product of K with this vector
        return torch.from_numpy(_solve_problem(case, seed)["x"])
    if kind == "solve_batch":
        return torch.from_numpy(np.concatenate([p["x"] for p in _solve_batch_problems(case, seed)]))
    if kind == "batch":
        parts = [_assembled(p) for p in _batch_problems(case, seed)]
        return torch.cat([p[2] for p in parts]), torch.cat([p[3] for p in parts])
    pb = _assembly_problem(case, seed)
    r, c, K, F = _assembled(pb)
    nc = pb["num"]["nc"]
    blk = (r > nc).long() + (c > nc).long()
    if kind == "to_host":
        return [K[blk == b] for b in range(3)] + [F]
    if not case.get("newton"):
        return K, F
    dUc, dUsl = (torch.as_tensor(pb[k], device="cuda") for k in ("dUc", "dUsl"))
    nsl = F.numel() - nc

    def product(b, trans, x, y, coef):
        s = blk == b
        rr, cc, v = r[s] - 1, c[s] - 1, K[s]
        if b:
            cc = cc - nc
        if b == 2:
            rr = rr - nc
        if b != 1:                      # symmetric: both triangles
            y.index_add_(0, cc[rr != cc], coef * (v * x[rr])[rr != cc])
        if trans:
            return y.index_add_(0, cc, coef * v * x[rr])
        return y.index_add_(0, rr, coef * v * x[cc])

    rhs = product(1, True, dUc, F[nc:].clone(), -1.0)
    res = rhs.clone()
    if pb["num"]["n_mpc"]:
        lam = torch.zeros(nsl, dtype=torch.float64, device="cuda")
        nu = pb["num"]["n_unk"]
        lam[nu:] = torch.as_tensor(pb["U"], device="cuda")[nc + nu:]
        product(2, False, lam, res, -1.0)
    reac = product(0, False, dUc, torch.zeros(nc, dtype=torch.float64, device="cuda"), 1.0)
    product(1, False, dUsl, reac, 1.0)
    return [K, F, rhs, res, reac - F[:nc]]
