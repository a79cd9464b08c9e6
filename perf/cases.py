"""Performance cases: the work a program of this framework has it do, through
its public entry points.

Each kind of case stands for a call, or a short run of calls, that the drivers
make: whole Picard and time steps, and the blocks they are made of (element
build and assembly, matrix products, incomplete factorisation and its sweeps,
AMG V-cycle, learned preconditioner).  Sizes run from the 64 x 64 transport
mesh of the reference's own configuration to the 2048 x 1024 one; the drawn
cases spread over the same ranges, ragged sizes and the other storage schemes,
solvers and precisions among them.
"""
import ctypes
import math
import os

import numpy as np
import torch

import fem_codes_gb300 as fg
from fem_codes_gb300 import learned
from fem_codes_gb300.mesh import (cavity_problem, euler_cfl_dt, refletido_problem, skew_problem,
                                  structured_mesh)

_vp = ctypes.c_void_p
_WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(fg.__file__)), "weights", "gnn_transport.npy")


def listed():
    return [
        # The smallest whole run: the reference's own transport configuration
        # (CSR, ILU(0), GMRES(30)), two Picard iterations through the host
        # call; launches and latency are what counts.
        {"name": "picard_64x64", "kind": "picard", "nx": 64, "ny": 64, "reorder": "NOT", "kmax": 30, "steps": 2},
        # The largest whole run: one Picard iteration (build, factorisation,
        # solve to 1e-8) of the 4.2M-triangle transport configuration, block
        # ILU(0) x32 and FGMRES(80), continuing from the previous iterate.
        {"name": "step_2048x1024", "kind": "step", "nx": 2048, "ny": 1024, "blocks": 32, "kmax": 80},
        # One implicit Euler time step (predictor, two correctors: build,
        # nodal block-diagonal set-up, FGMRES(50) in FP64) of the oblique
        # shock reflection, a few steps in.
        {"name": "euler_step_256x64", "kind": "euler_step", "nx": 256, "ny": 64, "solver": "FGMRES"},
        # The Krylov operator of that transport configuration on its own.
        {"name": "product_csr_2048x1024", "kind": "product", "nx": 2048, "ny": 1024, "scheme": "CSR", "fused": True},
        # The edge-by-edge product on a mid-sized mesh with odd sides.
        {"name": "product_ede_1001x703", "kind": "product", "nx": 1001, "ny": 703, "scheme": "EDE", "fused": False},
        # Element build and CSR assembly, what every Picard iteration starts with.
        {"name": "build_csr_1200x900", "kind": "build", "nx": 1200, "ny": 900, "scheme": "CSR"},
        # The reference's preconditioner as it has it: ILU(0) of the whole
        # matrix in SYMRCM order, F := M^-1 F, and one more application.
        {"name": "ilu_global_400x300", "kind": "ilu", "nx": 400, "ny": 300, "blocks": 0, "solver": "GMRES"},
        # Euler element Jacobians and residual at the full configuration's
        # size, the state a few time steps in.
        {"name": "euler_build_1024x256", "kind": "euler_build", "nx": 1024, "ny": 256},
        # What one Newton iteration of the lid-driven cavity sets up: VMS
        # build, CSR assembly, ILU(0) and F := M^-1 F.
        {"name": "ns_setup_96", "kind": "ns_setup", "n": 96},
        # One V-cycle of the double pairwise aggregation preconditioner.
        {"name": "amg_cycle_300x200", "kind": "amg", "nx": 300, "ny": 200, "ncl": 3},
        # One application of the learned preconditioner, bf16 activations,
        # trained weights, at the largest training mesh's size.
        {"name": "gnn_apply_1024x1024", "kind": "gnn_apply", "nx": 1024, "ny": 1024, "bf16": True},
        # One training gradient of that network on the smallest training mesh.
        {"name": "gnn_grad_256x256", "kind": "gnn_grad", "nx": 256, "ny": 256, "bf16": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, most):
    """Two mesh sides in [lo, hi], their product at most `most` cells."""
    while True:
        nx, ny = _log(rng, lo, hi), _log(rng, lo, hi)
        if nx * ny <= most and nx <= 8 * ny and ny <= 8 * nx:
            return nx, ny


def draw(rng):
    kind = rng.choice(["picard", "step", "euler_step", "product", "product", "build", "ilu", "ilu", "euler_build",
                       "euler_product", "ns_setup", "amg", "gnn_apply", "gnn_grad"])
    if kind == "picard":
        nx, ny = _sides(rng, 16, 160, 160 * 100)
        return {"kind": kind, "nx": nx, "ny": ny, "reorder": rng.choice(["NOT", "SYMRCM"]),
                "kmax": rng.choice([20, 30, 50]), "steps": rng.choice([1, 2, 3])}
    if kind == "step":
        nx, ny = _sides(rng, 96, 2048, 1 << 20)
        return {"kind": kind, "nx": nx, "ny": ny, "blocks": rng.choice([8, 16, 32]), "kmax": rng.choice([60, 80])}
    if kind == "euler_step":
        nx, ny = _sides(rng, 24, 320, 320 * 80)
        return {"kind": kind, "nx": nx, "ny": ny, "solver": rng.choice(["GMRES", "FGMRES"])}
    if kind == "product":
        nx, ny = _sides(rng, 48, 2048, 1 << 21)
        scheme = rng.choice(["CSR", "EDE", "EBE"])
        return {"kind": kind, "nx": nx, "ny": ny, "scheme": scheme,
                "fused": scheme == "CSR" and rng.random() < 0.5}
    if kind == "build":
        nx, ny = _sides(rng, 48, 2048, 1 << 21)
        return {"kind": kind, "nx": nx, "ny": ny, "scheme": "CSR"}
    if kind == "ilu":
        nx, ny = _sides(rng, 48, 1024, 1 << 18)
        return {"kind": kind, "nx": nx, "ny": ny, "blocks": rng.choice([0, 8, 16, 32]),
                "solver": rng.choice(["GMRES", "FGMRES"])}
    if kind == "euler_build":
        nx, ny = _sides(rng, 24, 1024, 1 << 18)
        return {"kind": kind, "nx": nx, "ny": ny}
    if kind == "euler_product":
        nx, ny = _sides(rng, 24, 1024, 1 << 18)
        return {"kind": kind, "nx": nx, "ny": ny, "precision": rng.choice(["FP64", "MIXED_IR"])}
    if kind == "ns_setup":
        return {"kind": kind, "n": _log(rng, 16, 160)}
    if kind == "amg":
        nx, ny = _sides(rng, 32, 512, 1 << 16)
        return {"kind": kind, "nx": nx, "ny": ny, "ncl": rng.choice([2, 3])}
    if kind == "gnn_apply":
        nx, ny = _sides(rng, 48, 1400, 1 << 20)
        return {"kind": kind, "nx": nx, "ny": ny, "bf16": rng.random() < 0.75}
    nx, ny = _sides(rng, 48, 1024, 1 << 18)
    return {"kind": "gnn_grad", "nx": nx, "ny": ny, "bf16": rng.random() < 0.75}


# ------------------------------------------------------------------ helpers
class _Buffer:
    """A device array of a context, kept alive with it (CUDA array interface)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3}


def _view(owner, ptr, *shape):
    return torch.as_tensor(_Buffer(owner, ptr, shape), device="cuda")


_streams = []


def _stream():
    """The one stream this program launches on, as bench.py has it: every
    context is bound to it."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _check(rc, what):
    if rc:
        raise fg.FemGpuError(rc, what)


def _normal(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def _transport(c, seed, scheme="CSR", reorder="NOT", **kw):
    """A skew-advection context on a mesh perturbed from the seed."""
    m = structured_mesh(c["nx"], c["ny"], perturb=0.2, seed=int(seed))
    p = skew_problem(m)
    T = fg.SSTransport.from_problem(m, p, scheme=scheme, reorder=reorder, **kw)
    T.set_stream(_stream().cuda_stream)
    return m, p, T


def _front(m, p, T, seed):
    """A nodal state such as a Picard iterate has: the inflow values carried
    along the flow, the front smeared over a few cells, with a little noise;
    in the context's numbering (neq + 1 values, the last one 0)."""
    h = 1.0 / min(m.nx, m.ny)
    d = m.y - 0.5 / 0.86602540378443865 * m.x - 0.3
    u = 0.5 * (1.0 + np.tanh(d / (2.0 * h)))
    u += 1e-4 * np.random.default_rng(seed).standard_normal(u.size)
    ids = T.pattern()["node_id"]
    out = np.zeros(T.neq + 1)
    out[ids[ids >= 0]] = u[ids >= 0]
    return out


def _fem_csr(nx, ny, seed):
    """The 7-point matrix of linear triangles on an nx x ny node grid with
    upwinded, seed-perturbed coefficients: (IA, JA, AA), ascending columns."""
    rng = np.random.default_rng(seed)
    n = nx * ny
    i = np.arange(n)
    x, y = i % nx, i // nx
    off = [(-1, -1), (0, -1), (-1, 0), (0, 0), (1, 0), (0, 1), (1, 1)]
    base = np.array([-0.35, -0.9, -1.2, 4.0, -0.6, -0.5, -0.25])
    ok = np.stack([(x + a >= 0) & (x + a < nx) & (y + b >= 0) & (y + b < ny) for a, b in off], axis=1)
    col = np.stack([i + a + b * nx for a, b in off], axis=1)
    val = base * (1.0 + 0.2 * rng.uniform(-1.0, 1.0, (n, 7)))
    IA = np.zeros(n + 1, np.int32)
    IA[1:] = np.cumsum(ok.sum(axis=1))
    return IA, col[ok].astype(np.int32), val[ok]


def _euler(c, seed, **kw):
    """A reflected-shock context a few implicit time steps in, on a mesh
    perturbed from the seed; the state is left on the device."""
    m = structured_mesh(c["nx"], c["ny"], lx=4.0, ly=1.0, perturb=0.05, seed=int(seed))
    p = refletido_problem(m)
    E = fg.Euler.from_problem(m, p, alpha=0.5, dt=euler_cfl_dt(m, 5.0), stab_tol=1e-6, kmax=50, lmax=100, ncorr=2,
                              **kw)
    E.set_stream(_stream().cuda_stream)
    return m, p, E


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    c, k = case, case["kind"]
    st = {"kind": k, "case": dict(case)}
    if k == "picard":
        m, p, st["T"] = _transport(c, seed, reorder=c["reorder"], precond="ILU0", kmax=c["kmax"], lmax=1000, tol=1e-8,
                                   solver="GMRES")
    elif k == "step":
        m, p, T = _transport(c, seed, reorder="SYMRCM", precond="ILU0", kmax=c["kmax"], lmax=25, tol=1e-8,
                             solver="FGMRES", ilu_blocks=c["blocks"])
        T.build_dev()                                    # the previous Picard iteration, from u = 0
        T.precond_setup_dev(1)
        T.solve_dev()
        u = _view(T, T.u_dev(), T.neq + 1)
        torch.cuda.synchronize()
        st.update(T=T, u=u, u0=u.clone())
    elif k == "product":
        m, p, T = _transport(c, seed, scheme=c["scheme"], reorder="SYMRCM" if c["fused"] else "NOT", precond="NOT",
                             kmax=4, lmax=1, solver="FGMRES")
        T.Build(_front(m, p, T, seed))
        st.update(T=T, x=_normal(T.neq + 1, seed), y=torch.zeros(T.neq + 1, dtype=torch.float64, device="cuda"))
        st["x"][T.neq] = 0.0
    elif k == "build":
        m, p, T = _transport(c, seed, scheme=c["scheme"], precond="NOT", kmax=4, lmax=1, solver="FGMRES")
        T.Build(_front(m, p, T, seed))
        st.update(T=T, A=_view(T, T.csr_dev()[2], T.nnzero), F=_view(T, fg.load().femgpu_transport_F_dev(T.handle), T.neq))
    elif k == "ilu":
        m, p, T = _transport(c, seed, reorder="SYMRCM", precond="ILU0", kmax=4, lmax=1, solver=c["solver"],
                             ilu_blocks=c["blocks"])
        F0, _ = T.Build(_front(m, p, T, seed))
        st.update(T=T, F=_view(T, fg.load().femgpu_transport_F_dev(T.handle), T.neq + 1),
                  F0=torch.from_numpy(F0).cuda(), p=_normal(T.neq + 1, seed),
                  z=torch.zeros(T.neq + 1, dtype=torch.float64, device="cuda"))
        st["p"][T.neq] = 0.0
    elif k == "euler_step":
        m, p, E = _euler(c, seed, solver=c["solver"], tol=1e-8)
        u, _ = E.Predictor(p.u0, 2)
        st.update(E=E, u0=u[-1].copy())
    elif k == "euler_build":
        m, p, E = _euler(c, seed, solver="FGMRES", precision="MIXED_IR", tol=1e-4)
        E.Predictor(p.u0, 2)
        A = fg.load().femgpu_ebe_A_dev
        A.restype, A.argtypes = _vp, [_vp]
        st.update(E=E, A=_view(E, A(fg.load().femgpu_euler_ebe(E.handle)), E.nel, 144),
                  R=torch.zeros(E.neq + 1, dtype=torch.float64).pin_memory())
    elif k == "euler_product":
        m, p, E = _euler(c, seed, solver="FGMRES", precision=c["precision"], tol=1e-4)
        E.Predictor(p.u0, 2)
        L = fg.load()
        f = L.femgpu_ebe_matvec_dev if c["precision"] == "FP64" else L.femgpu_ebe_matvec32_dev
        f.restype, f.argtypes = ctypes.c_int, [_vp, _vp, _vp]
        x = _normal(E.neq + 1, seed)
        x[E.neq] = 0.0
        st.update(E=E, product=f, ebe=_vp(L.femgpu_euler_ebe(E.handle)), x=x if c["precision"] == "FP64" else x.float(),
                  y=torch.zeros(E.neq + 1, dtype=torch.float64, device="cuda"))
    elif k == "ns_setup":
        m = structured_mesh(c["n"], c["n"], perturb=0.1, seed=int(seed))
        p = cavity_problem(m, 1000.0)
        N = fg.NavierStokes.from_problem(m, p, solver="FGMRES", kmax=50, lmax=40, scheme="CSR", precond="ILU0")
        N.set_stream(_stream().cuda_stream)
        # a developing cavity flow: a vortex with the lid's speed and a smooth pressure
        u = np.zeros((m.nnodes, 3))
        u[:, 0] = -0.4 * np.sin(np.pi * m.x) ** 2 * np.sin(2.0 * np.pi * m.y)
        u[:, 1] = 0.4 * np.sin(2.0 * np.pi * m.x) * np.sin(np.pi * m.y) ** 2
        u[:, 2] = 0.1 * np.cos(np.pi * m.x) * np.cos(np.pi * m.y)
        u *= 1.0 + 0.05 * np.random.default_rng(seed).standard_normal(u.shape)
        free = p.node_id >= 0
        v = np.zeros(p.neq + 1)
        v[p.node_id[free]] = u[free]
        st.update(N=N, u=v)
    elif k == "amg":
        m, p, T = _transport(c, seed, precond="NOT", kmax=4, lmax=1, solver="FGMRES")
        _, A = T.Build(_front(m, p, T, seed), want_matrix=True)
        pat = T.pattern()
        T.close()
        G = fg.AMG(ncl=c["ncl"], beta=-1.0, omega=1.0, nr=2)
        _check(fg.load().femgpu_amg_set_stream(G.handle, _vp(_stream().cuda_stream)), "set_stream")
        G.setup(pat["IA"], pat["JA"], A[:len(pat["JA"])])
        st.update(G=G, q=_normal(G.n, seed), z=torch.zeros(G.n, dtype=torch.float64, device="cuda"))
    else:
        net = learned.MeshGNN(np.load(_WEIGHTS), bf16=c["bf16"])
        net.set_stream(_stream().cuda_stream)
        net.attach_csr(*_fem_csr(c["nx"], c["ny"], seed))
        st.update(net=net, r=_normal(net.n, seed), z=torch.zeros(net.n, dtype=torch.float64, device="cuda"))
        if k == "gnn_grad":
            net.set_loss("residual")
            st["t"] = 0.25 * st["r"]
    return st


# ---------------------------------------------------------------------- run
def run(st):
    k, L = st["kind"], fg.load()
    if k == "picard":
        u, _ = st["T"].Process(st["case"]["steps"])
        return u
    if k == "step":
        T = st["T"]
        with torch.cuda.stream(_stream()):
            st["u"].copy_(st["u0"])
        T.build_dev()
        T.precond_setup_dev(2)
        T.solve_dev()
        return st["u"]
    if k == "product":
        f = L.femgpu_transport_operator_dev if st["case"]["fused"] else L.femgpu_transport_matvec_dev
        _check(f(st["T"].handle, _vp(st["x"].data_ptr()), _vp(st["y"].data_ptr())), "product")
        return st["y"]
    if k == "build":
        st["T"].build_dev()
        return {"A": st["A"], "F": st["F"]}
    if k == "ilu":
        T = st["T"]
        with torch.cuda.stream(_stream()):
            st["F"].copy_(st["F0"])
        T.precond_setup_dev(2)
        _check(L.femgpu_transport_precond_dev(T.handle, _vp(st["p"].data_ptr()), _vp(st["z"].data_ptr())), "precond")
        return {"F": st["F"], "z": st["z"]}
    if k == "euler_step":
        u, _ = st["E"].Predictor(st["u0"], 1)
        return u
    if k == "euler_build":
        _check(L.femgpu_euler_build(st["E"].handle, None, None, None, _vp(st["R"].data_ptr())), "build")
        return {"A": st["A"], "R": st["R"]}
    if k == "euler_product":
        _check(st["product"](st["ebe"], _vp(st["x"].data_ptr()), _vp(st["y"].data_ptr())), "product")
        return st["y"]
    if k == "ns_setup":
        N = st["N"]
        N.reset()
        F, _ = N.Build(st["u"])
        return {"F": F, "MF": N.precond_setup()}
    if k == "amg":
        st["G"].apply_dev(st["q"].data_ptr(), st["z"].data_ptr())
        return st["z"]
    net = st["net"]
    if k == "gnn_apply":
        net.apply_dev(st["r"].data_ptr(), st["z"].data_ptr())
        return st["z"]
    net.loss_grad_dev(st["r"].data_ptr(), st["t"].data_ptr(), st["z"].data_ptr(), False)
    return {"grad": net.grad(), "z": st["z"]}


# --------------------------------------------------------------------- work
def work(case):
    """Bytes and floating-point operations of one pass that no implementation
    does without: the mesh or matrix read once (a solve: the matrix and its
    factors once), vectors read and written once; 12 bytes per CSR entry, FP64
    values elsewhere."""
    k = case["kind"]
    nx, ny = case.get("nx", case.get("n")), case.get("ny", case.get("n"))
    n, ne = (nx + 1) * (ny + 1), 2 * nx * ny
    nnz = 7 * n
    mesh = 16 * n + 12 * ne + 12 * n                     # coordinates, vertices, numbering and state
    if k in ("picard", "step"):
        steps = case.get("steps", 1)
        return {"bytes": steps * (mesh + 2 * 12 * nnz + 8 * nnz + 16 * n), "flops": steps * (200 * ne + 8 * nnz)}
    if k == "product":
        b = {"CSR": 12 * nnz, "EDE": 40 * 3 * n, "EBE": 84 * ne}[case["scheme"]]
        f = {"CSR": 2 * nnz, "EDE": 8 * 3 * n, "EBE": 18 * ne}[case["scheme"]]
        return {"bytes": b + 16 * n, "flops": f}
    if k == "build":
        return {"bytes": mesh + 8 * nnz + 8 * n, "flops": 200 * ne}
    if k == "ilu":
        return {"bytes": 12 * nnz + 8 * nnz + 12 * nnz + 32 * n, "flops": 6 * nnz}
    if k == "euler_build":
        return {"bytes": 12 * ne + 16 * n + 3 * 32 * n + 144 * 8 * ne, "flops": 2500 * ne}
    if k == "euler_product":
        w = 8 if case["precision"] == "FP64" else 4
        return {"bytes": 144 * w * ne + 48 * ne + 4 * n * (w + 8), "flops": 288 * ne}
    if k == "euler_step":
        return {"bytes": 2 * (12 * ne + 16 * n + 2 * 144 * 8 * ne + 4 * 32 * n), "flops": 2 * 2800 * ne}
    if k == "ns_setup":
        return {"bytes": 12 * ne + 16 * n + 24 * n + 2 * 9 * 12 * nnz + 48 * n, "flops": 2500 * ne + 9 * 40 * nnz}
    if k == "amg":
        # two sweeps down, two up and a residual on every level, level sizes 1, 1/4, 1/16, ...
        return {"bytes": 1.33 * (12 * nnz + 24 * n), "flops": 1.33 * 10 * nnz}
    e = 6 * nx * ny                                      # off-diagonal entries of the graph
    f = nx * ny * 3 * (2 * 96 * 32) + 3 * 2 * 64 * e
    if k == "gnn_apply":
        return {"bytes": 12 * e + 24 * nx * ny, "flops": f}
    return {"bytes": 12 * e + 32 * nx * ny + 4 * 9441, "flops": 3 * f}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """The products, the transport build and the network in 64-bit torch;
    None for solves, factorisations and the Euler and Navier-Stokes builds."""
    k = case["kind"]
    if k == "product":
        return _exact_product(case, seed)
    if k == "euler_product":
        st = prepare(case, seed)
        E = st["E"]
        A = fg.load().femgpu_ebe_A_dev
        A.restype, A.argtypes = _vp, [_vp]
        A = _view(E, A(fg.load().femgpu_euler_ebe(E.handle)), E.nel, 12, 12)
        vert, ids = E._keep[2].reshape(-1, 3), E._keep[3].reshape(-1, 4)
        lm = torch.from_numpy(np.where(ids[vert] < 0, E.neq, ids[vert]).reshape(-1, 12).astype(np.int64)).cuda()
        y = torch.zeros(E.neq + 1, dtype=torch.float64, device="cuda")
        y.index_add_(0, lm.reshape(-1), torch.einsum("eij,ej->ei", A, st["x"].double()[lm]).reshape(-1))
        y[E.neq] = 0.0
        return y
    if k == "build":
        return _exact_build(case, seed)
    if k in ("gnn_apply", "gnn_grad"):
        return _exact_network(case, seed)
    return None


def _exact_product(case, seed):
    st = prepare(case, seed)
    T, x = st["T"], st["x"]
    _, A = T.Build(None, want_matrix=True)
    A, pat, n = torch.from_numpy(A).cuda(), T.pattern(), T.neq
    y = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    if case["scheme"] == "CSR":
        row = np.repeat(np.arange(n), np.diff(pat["IA"]))
        y.index_add_(0, torch.from_numpy(row).cuda(), A[:T.nnzero] * x[torch.from_numpy(pat["JA"]).cuda().long()])
    elif case["scheme"] == "EDE":
        a, e = A.reshape(-1, 4)[:T.nedge], torch.from_numpy(pat["lm2"].astype(np.int64)).cuda()
        p, q = x[e[:, 0]], x[e[:, 1]]
        y.index_add_(0, e[:, 0], a[:, 0] * p + a[:, 1] * q)
        y.index_add_(0, e[:, 1], a[:, 2] * p + a[:, 3] * q)
    else:
        ids = pat["node_id"][T._keep[3].reshape(-1, 3)]
        lm = torch.from_numpy(np.where(ids < 0, n, ids).astype(np.int64)).cuda()
        y.index_add_(0, lm.reshape(-1), torch.einsum("eij,ej->ei", A.reshape(-1, 3, 3), x[lm]).reshape(-1))
    y[n] = 0.0
    return y


def _exact_build(case, seed):
    """SUPG with CAU shock capturing on linear triangles, assembled into CSR:
    grad-grad, convection, streamline and shock terms of each element from the
    basis gradients (zero source and reaction)."""
    st = prepare(case, seed)
    T = st["T"]
    m = structured_mesh(case["nx"], case["ny"], perturb=0.2, seed=int(seed))
    p = skew_problem(m)
    pat, n = T.pattern(), T.neq
    dev = {"dtype": torch.float64, "device": "cuda"}
    vert = torch.from_numpy(m.vert.astype(np.int64)).cuda()
    X, Y = torch.from_numpy(m.x).cuda()[vert], torch.from_numpy(m.y).cuda()[vert]
    ids = torch.from_numpy(pat["node_id"].astype(np.int64)).cuda()
    u = torch.from_numpy(_front(m, p, T, seed)).cuda()
    presc = torch.from_numpy(p.upresc).cuda()
    ue = torch.where(ids >= 0, u[ids.clamp(min=0)], presc)[vert]
    b = torch.stack([Y[:, 1] - Y[:, 2], Y[:, 2] - Y[:, 0], Y[:, 0] - Y[:, 1]], 1)
    c = torch.stack([X[:, 2] - X[:, 1], X[:, 0] - X[:, 2], X[:, 1] - X[:, 0]], 1)
    area = 0.5 * (c[:, 2] * b[:, 1] - c[:, 1] * b[:, 2])
    G = torch.stack([b, c], 2) / (2.0 * area)[:, None, None]             # basis gradients [e, 3, 2]
    beta = torch.tensor(p.beta[0], **dev)
    bg = G @ beta                                                        # beta . grad N_i
    h = torch.sqrt((2.0 * area).abs())
    tau = 0.5 * h / beta.norm()
    gu = torch.einsum("ei,eid->ed", ue, G)
    ru, ng2 = (bg * ue).sum(1), (gu * gu).sum(1)
    ng = ng2.sqrt()
    par = ru[:, None] * gu / torch.where(ng2 > 0, ng2, 1.0)[:, None]     # velocity along grad u
    npar = par.norm(dim=1)
    pe = 0.5 * h * npar ** 3 / torch.where(npar > 0, p.k * npar ** 2, 1.0)
    delta = 0.5 * h * torch.minimum(pe / 3.0, torch.tensor(0.7, **dev)) * ru.abs() / torch.where(ng > 0, ng, 1.0)
    delta = torch.where(ng > 0, delta, 0.0)
    K = torch.einsum("eid,ejd->eij", G, G) * ((p.k + delta) * area)[:, None, None]
    K = K + (area / 3.0)[:, None, None] * bg[:, None, :] + (tau * area)[:, None, None] * bg[:, :, None] * bg[:, None, :]
    eq = ids[vert]
    free = (eq[:, :, None] >= 0) & (eq[:, None, :] >= 0)
    key = (eq[:, :, None] * n + eq[:, None, :])[free]
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(pat["IA"]))
    keys = torch.from_numpy(row * n + pat["JA"]).cuda()
    A = torch.zeros(T.nnzero, **dev)
    A.index_add_(0, torch.searchsorted(keys, key), K[free])
    lift = torch.where(eq[:, None, :] >= 0, 0.0, -K * presc[vert][:, None, :]).sum(2)
    F = torch.zeros(n, **dev)
    F.index_add_(0, eq[eq >= 0], lift[eq >= 0])
    return {"A": A, "F": F}


def _exact_network(case, seed):
    IA, JA, AA = _fem_csr(case["nx"], case["ny"], seed)
    n = IA.size - 1
    row = torch.from_numpy(np.repeat(np.arange(n, dtype=np.int64), np.diff(IA))).cuda()
    col, val = torch.from_numpy(JA.astype(np.int64)).cuda(), torch.from_numpy(AA).cuda()
    d = torch.zeros(n, dtype=torch.float64, device="cuda")
    on = row == col
    d[row[on]] = val[on]
    A = torch.sparse_coo_tensor(torch.stack([row, col]), val, (n, n)).coalesce()
    i, j, v = row[~on], col[~on], val[~on]
    wA = torch.sparse_coo_tensor(torch.stack([i, j]), v / d[i], (n, n)).coalesce()
    wT = torch.sparse_coo_tensor(torch.stack([j, i]), v / d[i], (n, n)).coalesce()
    r = _normal(n, seed)
    theta = torch.from_numpy(np.load(_WEIGHTS).astype(np.float64)).cuda().requires_grad_(case["kind"] == "gnn_grad")
    part, o = {}, 0
    for name, shape in learned.param_shapes():
        size = int(np.prod(shape))
        part[name] = theta[o:o + size].reshape(shape)
        o += size
    s, dbar = r.square().mean().sqrt(), d.abs().mean()
    x = torch.stack([r / s, r / s * dbar / d], 1)
    h = torch.relu(x @ part["We"] + part["be"])
    for l in range(learned.LAYERS):
        u = h @ part[f"Wh{l}"] + torch.sparse.mm(wA, h) @ part[f"W1{l}"] + torch.sparse.mm(wT, h) @ part[f"W2{l}"]
        h = h + torch.relu(u + part[f"b{l}"])
    z = s * (h @ part["Wd"] + part["bd"]) * dbar / d
    if case["kind"] == "gnn_apply":
        return z
    loss = (torch.sparse.mm(A, z[:, None])[:, 0] - r).square().sum() / r.square().sum()
    grad, = torch.autograd.grad(loss, theta)
    return {"grad": grad.cpu().numpy(), "z": z.detach()}
