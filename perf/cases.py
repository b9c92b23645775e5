"""What a program that uses this framework has it do, as timed cases over the public entry
points of ``cfdv_b200.gpu`` (``FDVSolver`` and the C ABI's ``cfdv_ebe_matvec_static``).

The ranges: quad4 meshes from the 8x8 cavity to the twice-refined flat plate, hex8 meshes from
a few hundred elements to the 128x64x32 compression ramp; odd and ragged extents; the textbook
solve in FP64 and mixed precision, cold and warm-started, and the reference-mode solve; the
discrete adjoint with its two products (VJP, JVP); the element-by-element product on a caller's
device buffers, plain and transposed.

Every input follows from the seed: the mesh generators' initial state with 1e-3 relative
Gaussian density noise (the flat plate's configuration asks for it), drawn anew per seed.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from cfdv_b200 import gpu as G
from cfdv_b200 import meshgen as mg

RTOL = 1e-8      # relative residual of every textbook solve, the configurations' tolerance
RESTARTS = 200   # restart limit of the textbook solves
# per family: CFL number and GMRES restart length
FAMILY = {"lid": (0.5, 20), "plate": (1.0, 30), "ramp": (0.25, 50), "duct": (0.5, 40), "cylinder": (0.5, 40)}
# EBE products that one solve of a kind takes (what its work is counted with); the smaller
# plates need fewer than the 200x100 one, the larger ones more
PRODUCTS = {("step", "lid"): 31, ("step", "plate"): 61, ("step", "ramp"): 40, ("step", "duct"): 46,
            ("march", "lid"): 30, ("march", "duct"): 35, ("reference", "lid"): 21, ("reference", "plate"): 27,
            ("reference", "ramp"): 8, ("adjoint", "cylinder"): 60}
PREC = {"fp64": G.PREC_FP64, "mixed": G.PREC_MIXED}


def listed():
    return [
        # the host driver's default step (reference-mode GMRES) on the smallest configuration:
        # the lid-driven cavity, bound by latency and launches
        dict(name="lid_reference", kind="reference", family="lid", nx=32, ny=32, nz=0, prec="fp64"),
        # the flat plate at its configured size, FP64: the plain form the mixed one is held against
        dict(name="plate_fp64", kind="step", family="plate", nx=200, ny=100, nz=0, prec="fp64"),
        # the same in mixed precision: the configuration the headline figure is quoted on
        dict(name="plate_mixed", kind="step", family="plate", nx=200, ny=100, nz=0, prec="mixed"),
        # a refinement study's next plate, ragged: its Krylov basis no longer fits on chip
        dict(name="plate_fine_mixed", kind="step", family="plate", nx=391, ny=203, nz=0, prec="mixed"),
        # a short run on a small ragged duct, each solve after the first started from the last dU
        dict(name="duct_small_march", kind="march", family="duct", nx=25, ny=13, nz=7, prec="mixed"),
        # the reference-mode step of the host driver in 3D
        dict(name="ramp_reference", kind="reference", family="ramp", nx=64, ny=32, nz=32, prec="fp64"),
        # the compression ramp at its configured size, mixed: the largest step
        dict(name="ramp_mixed", kind="step", family="ramp", nx=128, ny=64, nz=32, prec="mixed"),
        # a jittered duct with ragged extents, FP64
        dict(name="duct_fp64", kind="step", family="duct", nx=97, ny=53, nz=29, prec="fp64"),
        # gradient of the cylinder's drag: forward steps, then the reverse sweep
        dict(name="cylinder_adjoint", kind="adjoint", family="cylinder", nx=48, ny=64, nz=9, prec="mixed"),
        # the residual's vector-Jacobian product for a program with its own adjoint solver
        dict(name="cylinder_vjp", kind="vjp", family="cylinder", nx=96, ny=128, nz=16, prec="fp64"),
        # the residual's Jacobian-vector product (tangent runs, matrix-free Newton)
        dict(name="cylinder_jvp", kind="jvp", family="cylinder", nx=48, ny=64, nz=9, prec="fp64"),
        # the EBE product on a caller's device buffers, near the entry point's size limit
        dict(name="matvec", kind="matvec", family="ramp", nx=50, ny=32, nz=32, prec="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reference", "step", "step", "step", "march", "adjoint", "vjp", "jvp", "matvec", "matvec"])
    family = {"reference": ["lid", "plate", "ramp"], "step": ["lid", "plate", "ramp", "duct"],
              "march": ["lid", "duct"], "adjoint": ["cylinder"], "vjp": ["cylinder", "duct", "plate"],
              "jvp": ["cylinder", "duct", "plate"], "matvec": ["plate", "ramp"]}[kind]
    family = rng.choice(family)
    prec = rng.choice(["fp64", "mixed"]) if kind in ("step", "march", "adjoint") else "fp64"
    if family == "lid":
        nx = ny = _log(rng, 8, 64)
        nz = 0
    elif family == "plate":
        nx = _log(rng, 24, 400 if kind in ("step", "vjp") else 200)
        ny, nz = max(10, int(nx * rng.uniform(0.45, 0.55))), 0
    else:
        top = {"step": 250_000, "vjp": 180_000, "reference": 60_000, "matvec": 52_000, "march": 20_000}.get(kind, 27_000)
        e = math.exp(rng.uniform(math.log(300), math.log(top)))
        s = (e / 4.0) ** (1.0 / 3.0)  # about 2 : 2 : 1, each extent off by up to a fifth
        nx, ny, nz = (max(4, int(k * s * rng.uniform(0.8, 1.0))) for k in (2.0, 2.0, 1.0))
        if family == "cylinder":
            nz = max(3, nz)
            ny = max(8, ny)
    case = dict(kind=kind, family=family, nx=nx, ny=ny, nz=nz, prec=prec)
    if kind == "matvec":
        case["transpose"] = rng.random() < 0.5
    return case


def _mesh(case, seed):
    """The family's mesh, its density carrying 1e-3 relative Gaussian noise drawn from the seed."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["family"] == "lid":
        c = mg.lid(nx)
    elif case["family"] == "plate":  # the wall spacing of 100 layers at ratio 1.05, whatever their number
        c = mg.plate(nx, ny, ratio=1.05 ** (100.0 / ny))
    elif case["family"] == "ramp":
        c = mg.ramp(nx, ny, nz)
    elif case["family"] == "duct":
        c = mg.duct(nx, ny, nz)
    else:
        c = mg.cylinder(nx, ny, nz)
    rng = np.random.default_rng(seed)
    c.nodes[:, c.ndim] *= 1.0 + 1e-3 * rng.standard_normal(c.n_nodes)
    return c, rng


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    c, rng = _mesh(case, seed)
    if case["kind"] == "matvec":
        return _prepare_matvec(case, c, seed)
    s = G.FDVSolver(c)
    s.load_node_records()
    st = {"case": case, "solver": s}
    if case["kind"] in ("step", "march", "reference"):
        u_in, u_out = _pinned(s.n_dof), _pinned(s.n_dof)
        u_in.numpy()[:] = s.get_state()
        st.update(keep=(u_in, u_out), u_in=u_in.numpy(), u_out=u_out.numpy())
    elif case["kind"] in ("vjp", "jvp"):
        cfl = FAMILY[case["family"]][0]
        s.form(s.cfl(cfl))  # fixes the step's dt
        n = s.n_dof
        st["du"] = 1e-3 * rng.standard_normal(n)
        st["v"] = rng.standard_normal(n) if case["kind"] == "vjp" else 1e-3 * rng.standard_normal(n)
    return st


def _prepare_matvec(case, c, seed):
    """Connectivity, node CSR, element matrices and x on the GPU, as the entry point takes them."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    conn = torch.from_numpy(np.ascontiguousarray(c.conn, dtype=np.int32)).to(dev)
    flat = conn.reshape(-1).long()
    idx = torch.argsort(flat, stable=True).to(torch.int32)  # entries of a node in element order
    ptr = torch.zeros(c.n_nodes + 1, dtype=torch.int32, device=dev)
    ptr[1:] = torch.cumsum(torch.bincount(flat, minlength=c.n_nodes), 0).to(torch.int32)
    ke, neqn = c.nnod * c.neqn, c.neqn
    R = torch.randn(c.n_elements, ke, ke, dtype=torch.float64, device=dev, generator=gen)  # column-major blocks
    x = torch.randn(c.n_nodes * neqn, dtype=torch.float64, device=dev, generator=gen)
    return {"case": case, "ndim": c.ndim, "n_nodes": c.n_nodes, "n_elements": c.n_elements, "conn": conn, "ptr": ptr,
            "idx": idx, "R": R, "x": x, "y": torch.empty_like(x)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matvec":
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = G.lib().cfdv_ebe_matvec_static(state["ndim"], state["n_nodes"], state["n_elements"], p(state["conn"]),
                                            p(state["ptr"]), p(state["idx"]), p(state["R"]), p(state["x"]),
                                            p(state["y"]), int(case.get("transpose", False)),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise G.CfdvError(rc, "ebe_matvec_static")
        return {"y": state["y"]}
    s = state["solver"]
    cfl, m = FAMILY[case["family"]]
    prec = PREC[case["prec"]]
    opts = dict(mode=G.GMRES_CORRECT, m=m, restarts=RESTARTS, rtol=RTOL, precision=prec)
    if kind == "step":  # one step with the state passed in and out in pinned host memory
        rep = s.step_host(cfl, state["u_in"], state["u_out"], **opts)
        return {"U": state["u_out"], "dt": rep["dt"]}
    if kind == "march":  # a cold step, then three that start from the last dU
        dt = [s.step_host(cfl, state["u_in"], None, **opts)["dt"]]
        dt += [s.step(cfl, warm_start=True, **opts)["dt"] for _ in range(2)]
        dt += [s.step_host(cfl, None, state["u_out"], warm_start=True, **opts)["dt"]]
        return {"U": state["u_out"], "dt": np.array(dt)}
    if kind == "reference":  # the host driver's calls of one iteration
        s.set_state(state["u_in"])
        dt = s.cfl(cfl)
        s.form(dt)
        rep = s.gmres(mode=G.GMRES_REFERENCE, m=m, restarts=1)
        s.update()
        rms = s.rms()
        return {"U": s.get_state(), "dt": dt, "est": rep["est"], "rms": rms}
    if kind == "adjoint":  # two steps, checkpointed every step
        r = s.adjoint(2, cfl, checkpoint_every=1, m=m, restarts=RESTARTS, rtol=1e-10, precision=prec)
        return {k: r[k] for k in ("J", "dJ_dmach", "dJ_dtwall", "wall_nodes", "dJ_dtnode")}
    if kind == "vjp":
        g, g_dt, g_mach = s.vjp(state["v"], state["du"])
        return {"g": g, "g_dt": g_dt, "g_mach": g_mach}
    return {"dr": s.jvp(state["du"], state["v"], t_dt=1e-4, t_mach=1e-3)}


def _counts(case):
    """(elements, unknowns, Ke) of a case's mesh."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["family"] == "cylinder":
        return nx * ny * (nz - 1), (nx + 1) * ny * nz * 5, 40
    if nz == 0:
        return nx * ny, (nx + 1) * (ny + 1) * 4, 16
    return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1) * 5, 40


def work(case):
    """Per product the element matrices streamed once (they are the solve's operator and far
    larger than the chip's memory in the cases that matter) and 2 Ke^2 flops an element; per
    formation the matrices written once and the flops of the factored Gauss-point contraction;
    the state and the vectors of an interface read and written once."""
    E, n, ke = _counts(case)
    form_flops = (13_824 if ke == 16 else 158_800) * E
    K2 = float(E) * ke * ke
    kind = case["kind"]
    sr = 4.0 if case["prec"] == "mixed" else 8.0
    if kind == "matvec":
        return {"bytes": 8.0 * K2 + 16.0 * n, "flops": 2.0 * K2}
    if kind in ("vjp", "jvp"):  # state, direction and dU in, one vector out; one residual and its derivative
        return {"bytes": 32.0 * n, "flops": 40_000.0 * E * (1.0 if ke == 40 else 0.1)}
    P = PRODUCTS[kind, case["family"]]
    steps = {"march": 4, "adjoint": 4}.get(kind, 1)  # an adjoint's two steps and two reverse steps
    formed = 8.0 * K2 + (4.0 * K2 if case["prec"] == "mixed" else 0.0)
    return {"bytes": steps * (formed + P * sr * K2 + 16.0 * n), "flops": steps * (form_flops + 2.0 * P * K2)}


def exact(case, seed):
    """The product of the caller's matrices in 64 bits.  The other kinds have no such value to
    compare with: a step is defined by its iteration stopping at a residual, and the formation,
    tangent and gradient only through the framework's own discretisation."""
    if case["kind"] != "matvec":
        return None
    c, _ = _mesh(case, seed)
    st = _prepare_matvec(case, c, seed)
    E, neqn = st["n_elements"], c.neqn
    dof = (st["conn"].long()[:, :, None] * neqn + torch.arange(neqn, device=st["x"].device)).reshape(E, -1)
    R = st["R"] if case.get("transpose", False) else st["R"].transpose(1, 2)  # R[e, j, i] holds entry (i, j)
    ye = torch.einsum("eij,ej->ei", R, st["x"][dof])
    return {"y": torch.zeros_like(st["x"]).index_add_(0, dof.reshape(-1), ye.reshape(-1))}
