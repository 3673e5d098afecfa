"""The work a user of this framework has it do, as timed cases.

Every case goes through a public entry point (``Solver``, ``Ensemble``, the
closure's ``Network`` and data functions, the C ABI) on inputs a user's
program holds on the device:

  step      n SSP-RK3 steps of one mesh, any precision pipeline, flux scheme,
            wall and viscosity choice; with the learned closure attached or not
  rhs       one right-hand side without a context (od_rhs_noalloc)
  ensemble  n steps of many boxes of uneven size, states back on the host
  train     minibatch Adam steps of the closure network
  data      a training snapshot: fine state -> coarse projection -> features
  diag      volume integrals and plane-averaged profiles
  fields    the ParaView point-field conversion's device part

``exact`` restates the discretisation in float64 torch on its own.
"""

import ctypes
import math

import numpy as np
import torch

from opendynamo_b200 import _native as N
from opendynamo_b200.forms import closure as C
from opendynamo_b200.forms.ensemble import Box, Ensemble
from opendynamo_b200.solver import Solver, make_params

DEV = "cuda"
PI = math.pi
CHANNEL = (2 * PI, 2.0, PI)     # the production channel's box (slip walls in y)
CUBE = (2 * PI,) * 3            # the Taylor-Green box (periodic)
NET_SIZES = [(256, 896), (256, 256), (256, 256), (384, 256)]


# ---------------------------------------------------------------- the cases
def _step(name, nx, ny, nz, pipeline, flux, wall, visc, steps, closure=False):
    c = {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "pipeline": pipeline, "flux": flux, "wall": wall,
         "visc": visc, "steps": steps, "closure": closure}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the small validation run: Taylor-Green, 8^3, inviscid Euler, Rusanov, f64
        _step("tgv8-f64-euler", 8, 8, 8, "f64", "rusanov", False, "inviscid", 10),
        # the production channel, the headline workload (141.6 MB of state)
        _step("channel48-f32", 48, 48, 48, "f32", "slau2", True, "constant", 5),
        # the all-f64 pipeline on a production mesh
        _step("channel40-f64", 40, 40, 40, "f64", "slau2", True, "constant", 2),
        # the default precision of a config without a [precision] table (f64 state,
        # f32 arithmetic) on a mesh whose sides divide by nothing, Sutherland's law
        _step("ragged37x29x23-u64c32", 37, 29, 23, "u64c32", "ausm+", True, "sutherland", 4),
        # the precision form at its own size, the largest mesh a user runs here
        _step("channel96-mixed", 96, 96, 96, "mixed", "slau2", True, "constant", 2),
        # a coarse run with the learned closure in every stage
        _step("closure24-f32", 24, 24, 24, "f32", "slau2", True, "constant", 10, True),
        # a right-hand side inside another framework's step callback: one tiny call
        {"name": "rhs4-f64", "kind": "rhs", "nx": 4, "ny": 4, "nz": 4, "pipeline": "f64", "flux": "rusanov",
         "wall": False, "visc": "constant"},
        # a parameter sweep: boxes of 8^3 to 32^3 elements, a run between two dumps
        {"name": "ensemble16", "kind": "ensemble", "boxes": 16, "n_min": 8, "n_max": 32, "steps": 100, "pick": 7},
        # training the closure network with its own batch size
        {"name": "train8192", "kind": "train", "batch": 8192, "steps": 4},
        # one snapshot of the closure's training data: 96^3 onto 24^3
        {"name": "data96to24", "kind": "data", "coarse": 24, "factor": 4},
        # the monitoring a run does beside its dumps
        {"name": "diag48-f32", "kind": "diag", "nx": 48, "ny": 48, "nz": 48, "pipeline": "f32"},
        # post-processing of a dump for ParaView
        {"name": "fields48-f32", "kind": "fields", "nx": 48, "ny": 48, "nz": 48, "pipeline": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi, most):
    while True:
        m = [_log_int(rng, lo, hi) for _ in range(3)]
        if m[0] * m[1] * m[2] <= most:
            return m


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["closure", "rhs", "ensemble", "train", "data", "diag", "fields"])
    if kind in ("step", "closure"):
        closure = kind == "closure"
        pipe = "f32" if closure else rng.choice(["f32", "f32", "f64", "u64c32", "u32c64", "mixed"])
        m = _mesh(rng, 4, 32, 24000) if closure else _mesh(rng, 2, 80, 200000)
        ne = m[0] * m[1] * m[2]
        steps = max(1, min(20, 400000 // ne))
        return _step(None, *m, pipe, rng.choice(["slau2", "ausm+", "rusanov"]), rng.random() < 0.6,
                     "constant" if closure else rng.choice(["constant", "inviscid", "sutherland"]), steps, closure)
    if kind == "rhs":
        m = _mesh(rng, 2, 20, 4800)
        return {"kind": "rhs", "nx": m[0], "ny": m[1], "nz": m[2], "pipeline": "f64",
                "flux": rng.choice(["slau2", "ausm+", "rusanov"]), "wall": rng.random() < 0.5,
                "visc": rng.choice(["constant", "inviscid", "sutherland"])}
    if kind == "ensemble":
        lo = _log_int(rng, 3, 12)
        return {"kind": "ensemble", "boxes": rng.randint(2, 24), "n_min": lo, "n_max": rng.randint(lo, 30),
                "steps": rng.randint(10, 60), "pick": rng.randrange(1000)}
    if kind == "train":
        return {"kind": "train", "batch": _log_int(rng, 100, 16384), "steps": rng.randint(1, 4)}
    if kind == "data":
        f = rng.randint(2, 4)
        return {"kind": "data", "coarse": _log_int(rng, 4, 96 // f), "factor": f}
    m = _mesh(rng, 3, 80, 200000)
    return {"kind": kind, "nx": m[0], "ny": m[1], "nz": m[2], "pipeline": rng.choice(["f32", "f64"])}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return np.random.default_rng(int(seed))


def _coords(n, ext):
    """Solution-point coordinates per axis, broadcastable over [z, y, x, k, j, i]."""
    xi = torch.tensor(np.polynomial.legendre.leggauss(4)[0], device=DEV)
    out = []
    for d in range(3):
        e = (torch.arange(n[d], device=DEV, dtype=torch.float64)[:, None] + 0.5 + 0.5 * xi[None, :]) * (ext[d] / n[d])
        shape = [1] * 6
        shape[2 - d], shape[5 - d] = n[d], 4
        out.append(e.reshape(shape))
    return out


def _flow(n, ext, wall, mach, seed, amp=0.05, modes=8):
    """A laminar channel (walls) or Taylor-Green flow (periodic) plus a
    solenoidal, wall-damped Fourier trip drawn from the seed: [5 x npts] float64."""
    rng = _gen(seed)
    x, y, z = _coords(n, ext)
    full = (n[2], n[1], n[0], 4, 4, 4)
    if wall:
        eta = y / (0.5 * ext[1]) - 1.0
        damp = 1.0 - eta * eta
        u = (1.5 * mach * damp).expand(full).clone()
        v = torch.zeros(full, device=DEV, dtype=torch.float64)
        w = torch.zeros(full, device=DEV, dtype=torch.float64)
        p = torch.full(full, 1.0 / 1.4, device=DEV, dtype=torch.float64)
    else:
        damp = 1.0
        u = mach * torch.sin(x) * torch.cos(y) * torch.cos(z)
        v = -mach * torch.cos(x) * torch.sin(y) * torch.cos(z)
        w = torch.zeros(full, device=DEV, dtype=torch.float64)
        p = 1.0 / 1.4 + mach * mach / 16.0 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)
    for _ in range(modes):
        kx, kz = 2 * PI * int(rng.integers(1, 7)) / ext[0], 2 * PI * int(rng.integers(1, 5)) / ext[2]
        a = amp * mach * float(rng.uniform(-1, 1)) / math.sqrt(modes) / math.hypot(kx, kz)
        th = damp * torch.cos(kx * x + kz * z + float(rng.uniform(0, 2 * PI)))
        u += kz * a * th
        w -= kx * a * th
        v += amp * mach * float(rng.uniform(-1, 1)) / math.sqrt(modes) * damp * torch.cos(kx * x + 0.7)
    E = p / 0.4 + 0.5 * (u * u + v * v + w * w)
    return torch.stack([torch.ones_like(u), u, v, w, E]).reshape(-1)


PREC = {"f32": dict(u_real="f32"), "f64": dict(u_real="f64"),
        "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "u32c64": dict(u_real="f32", q_real="f64", rhs_real="f64", compute_real="f64"),
        "mixed": dict(u_real="f64", mixed=True)}


def _dtype(pipeline):
    return torch.float64 if pipeline in ("f64", "u64c32", "mixed") else torch.float32


def _setup(case):
    """Mesh, physics and time step of a single-mesh case."""
    n = (case["nx"], case["ny"], case["nz"])
    wall = case.get("wall", True)
    ext = CHANNEL if wall else CUBE
    mach = 0.2 if wall else 0.1
    visc = case.get("visc", "constant")
    h = min(ext[d] / n[d] for d in range(3))
    return {"n": n, "ext": ext, "wall": wall, "mach": mach, "mu": 0.0 if visc == "inviscid" else 1.6e-4,
            "forcing": 1e-3 if wall else 0.0, "suth": 110.4 / 273.15 if visc == "sutherland" else -1.0,
            "flux": case.get("flux", "slau2"), "dt": float(np.float32(0.2 * h / (7.0 * 1.4)))}


def _params(case):
    s = _setup(case)
    return make_params(*s["n"], *s["ext"], flux=s["flux"], y_wall=s["wall"], mu=s["mu"], forcing=s["forcing"],
                       viscosity_model="sutherland" if s["suth"] >= 0 else "fixed", **PREC[case["pipeline"]])


def _input(case, seed):
    s = _setup(case)
    return _flow(s["n"], s["ext"], s["wall"], s["mach"], seed).to(_dtype(case["pipeline"])).contiguous()


def _boxes(case, seed):
    """Meshes from the case, flow parameters from the seed (as a sweep varies them)."""
    pick = _gen(case["pick"])
    rng = _gen(seed)
    out = []
    for b in range(case["boxes"]):
        n = int(round(math.exp(pick.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        wall = bool(pick.random() < 0.5)
        flux = "rusanov" if pick.random() < 0.5 else "slau2"
        mach, re = float(rng.uniform(0.05, 0.3)), float(rng.uniform(400.0, 1600.0))
        ext = CHANNEL if wall else CUBE
        dt = 0.3 * min(ext[d] / n for d in range(3)) / (7.0 * ((1.5 if wall else 1.0) * mach + 1.0))
        out.append(Box((n, n, n), ext, flux, wall, mach / re, 1e-3 if wall else 0.0, dt, "", mach, re, b))
    return out


# a network's standardisation: means and scales of a Mach-0.2 channel
FEAT_MEAN = np.array([1.0, 0.2, 0.0, 0.0, 1.81] + [0.0] * 9, np.float32)
FEAT_SCALE = np.array([1e-2, 0.1, 1e-2, 1e-2, 2e-2] + [0.3] * 9, np.float32)
OUT_SCALE = np.array([0.01, 0.02, 0.02, 0.02, 0.05], np.float32)


def _net_params(seed):
    return C.init_params(_gen(seed))


def _pools(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    rows = 4 * case["batch"]
    X = torch.randn(rows, 896, device=DEV, generator=g).clamp_(-8, 8).to(torch.bfloat16)
    T = torch.randn(rows, 320, device=DEV, generator=g).to(torch.bfloat16)
    picks = _gen(seed).permutation(rows).astype(np.int64)
    return X, T, [picks[k * case["batch"]:(k + 1) * case["batch"]] for k in range(case["steps"])]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("step", "diag"):
        s = _setup(case)
        st["u"] = _input(case, seed)
        st["solver"] = Solver(_params(case))
        st["stream"] = torch.cuda.ExternalStream(st["solver"].stream)
        if kind == "step":
            st["out"] = torch.empty_like(st["u"])
            st["dt"] = s["dt"]
            if case["closure"]:
                net = C.Network(case["nx"] * case["ny"] * case["nz"])
                net.set_params(_net_params(seed))
                net.set_scaling(FEAT_MEAN, FEAT_SCALE, OUT_SCALE)
                net.attach(st["solver"])
                st["net"] = net
        else:
            torch.cuda.synchronize()
            st["solver"].set_state_device(st["u"].data_ptr(), st["solver"].state_bytes)
            st["solver"].sync()
    elif kind == "rhs":
        st["u"] = _input(case, seed)
        st["out"] = torch.empty_like(st["u"])
        st["params"] = _params(case)
        st["lib"] = N.lib()
    elif kind == "ensemble":
        boxes = _boxes(case, seed)
        st["ens"] = Ensemble(boxes)
        for b, x in enumerate(boxes):
            st["ens"].set_state(b, _flow(x.n, x.extent, x.y_wall, x.mach, seed + 1000 * b).float().cpu().numpy())
    elif kind == "train":
        st["X"], st["T"], st["rows"] = _pools(case, seed)
        st["net"] = C.Network(case["batch"])
        st["net"].set_params(_net_params(seed))
    elif kind == "data":
        n = case["coarse"] * case["factor"]
        nc = case["coarse"]
        st["u"] = _flow((n, n, n), CHANNEL, True, 0.2, seed).float()
        st["coarse"] = torch.empty(5 * nc ** 3 * 64, device=DEV)
        st["X"] = torch.empty(nc ** 3, 896, device=DEV, dtype=torch.bfloat16)
    elif kind == "fields":
        st["u"] = _input(case, seed)
        st["out"] = torch.empty(7, 4 * case["nx"], 4 * case["ny"], 4 * case["nz"], device=DEV)
        st["lib"] = N.lib()
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------- one pass
def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "step":
        # the solver's own stream, ordered with the caller's on both sides
        sol, u, out = state["solver"], state["u"], state["out"]
        here = torch.cuda.current_stream()
        state["stream"].wait_stream(here)
        sol.set_state_device(u.data_ptr(), sol.state_bytes)
        sol.step(case["steps"], state["dt"])
        sol.get_state_device(out.data_ptr(), sol.state_bytes)
        here.wait_stream(state["stream"])
        return out
    if kind == "rhs":
        u, out = state["u"], state["out"]
        rc = state["lib"].od_rhs_noalloc(ctypes.byref(state["params"]), ctypes.c_void_p(u.data_ptr()),
                                         ctypes.c_void_p(out.data_ptr()), u.numel() * u.element_size(),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        N.check(rc, None, "od_rhs_noalloc")
        return out
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        return [state["ens"].get_state(b) for b in range(case["boxes"])]
    if kind == "train":
        loss = [state["net"].train_step(state["X"], state["T"], r, 1e-3) for r in state["rows"]]
        return {"loss": loss, "params": state["net"].get_params()}
    if kind == "data":
        nc = case["coarse"]
        C.project(state["u"], nc, nc, nc, case["factor"], state["coarse"])
        C.features_device(state["coarse"], nc, CHANNEL, FEAT_MEAN, FEAT_SCALE, state["X"])
        return {"coarse": state["coarse"], "features": state["X"]}
    if kind == "diag":
        return state["solver"].diagnostics()
    u, out = state["u"], state["out"]
    rc = state["lib"].od_point_fields(ctypes.c_void_p(u.data_ptr()), int(u.dtype == torch.float64), case["nx"],
                                      case["ny"], case["nz"], ctypes.c_void_p(out.data_ptr()),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    N.check(rc, None, "od_point_fields")
    return out


def work(case):
    kind = case["kind"]
    stage = 950.0   # floating-point operations a dof and stage: gradients, faces, fluxes, divergence, lifting, RK
    if kind == "train":
        mac = 896 * 256 + 2 * 256 * 256 + 256 * 320
        par = sum(r * (c + 1) for r, c in NET_SIZES)
        return {"bytes": case["steps"] * (case["batch"] * (896 + 320) * 2.0 + par * 24.0),
                "flops": case["steps"] * case["batch"] * (6.0 * mac - 2.0 * 896 * 256)}
    if kind == "data":
        nf, nc = case["coarse"] * case["factor"], case["coarse"]
        return {"bytes": 20.0 * 64 * nf ** 3 + (20.0 + 28.0) * 64 * nc ** 3,
                "flops": 5 * 64 * nf ** 3 * 2.0 * (4 + 4 / case["factor"]) + 64 * nc ** 3 * 150.0}
    if kind == "ensemble":
        dofs = sum(b.dofs for b in _boxes(case, 1))
        return {"bytes": case["steps"] * dofs * 160.0, "flops": case["steps"] * 3 * dofs * stage}
    dofs = 64.0 * case["nx"] * case["ny"] * case["nz"]
    size = 8.0 if _dtype(case["pipeline"]) == torch.float64 else 4.0
    if kind == "step":
        # stage 1 reads u and writes u'; stages 2 and 3 read u0 and u and write u'
        w = {"bytes": case["steps"] * dofs * 40.0 * size, "flops": case["steps"] * 3 * dofs * stage}
        if case["closure"]:
            w["flops"] += case["steps"] * 3 * dofs / 64 * 2.0 * (896 * 256 + 2 * 256 * 256 + 256 * 320)
        return w
    if kind == "rhs":
        return {"bytes": dofs * 10.0 * size, "flops": dofs * stage}
    if kind == "diag":
        return {"bytes": dofs * 5.0 * size, "flops": dofs * 200.0}
    return {"bytes": dofs * (5.0 * size + 28.0), "flops": dofs * 20.0}


# ---------------------------------------------------------------- in 64 bits
def _lagrange(xi, x):
    return np.array([np.prod([(x - xi[m]) / (xi[i] - xi[m]) for m in range(4) if m != i]) for i in range(4)])


def _operators():
    """Gauss-Legendre FR operators of degree 3: D, end traces, Radau g'."""
    L = np.polynomial.legendre
    xi = L.leggauss(4)[0]
    V = np.stack([L.legval(xi, np.eye(4)[k]) for k in range(4)], axis=1)
    dV = np.stack([L.legval(xi, L.legder(np.eye(4)[k])) if k else np.zeros(4) for k in range(4)], axis=1)
    D = dV @ np.linalg.inv(V)
    d3, d4 = (L.legval(xi, L.legder(np.eye(5)[k])) for k in (3, 4))
    return xi, D, _lagrange(xi, -1.0), _lagrange(xi, 1.0), 0.5 * (d4 - d3), 0.5 * (d3 + d4)


GAM, PRN = 1.4, 0.72


def _prim(q):
    ir = 1.0 / q[0]
    vel = [q[1] * ir, q[2] * ir, q[3] * ir]
    praw = (GAM - 1) * (q[4] - 0.5 * (q[1] * vel[0] + q[2] * vel[1] + q[3] * vel[2]))
    return ir, vel, praw, praw.clamp_min(1e-7)


def _euler(q, d):
    _, vel, _, p = _prim(q)
    f = [q[1 + d], q[1] * vel[d], q[2] * vel[d], q[3] * vel[d], vel[d] * (q[4] + p)]
    f[1 + d] = f[1 + d] + p
    return torch.stack(f)


def _viscous(q, g, d, mu0, suth):
    """Viscous flux along axis d; g[v][b] = d q_v / d x_b."""
    ir, vel, praw, p = _prim(q)
    mu = mu0
    if suth >= 0:
        T = GAM * p * ir
        mu = mu0 * T * torch.sqrt(T) * (1 + suth) / (T + suth)
    dv = lambda a, b: (g[1 + a][b] - vel[a] * g[0][b]) * ir   # noqa: E731
    div = dv(0, 0) + dv(1, 1) + dv(2, 2)
    tau = [mu * (dv(a, d) + dv(d, a) - (2.0 / 3.0 * div if a == d else 0.0)) for a in range(3)]
    ke = 0.5 * (q[1] * vel[0] + q[2] * vel[1] + q[3] * vel[2])
    dke = (q[1] * g[1][d] + q[2] * g[2][d] + q[3] * g[3][d]) * ir - ke * g[0][d] * ir
    heat = -mu * GAM / (PRN * (GAM - 1)) * ((GAM - 1) * (g[4][d] - dke) * ir - praw * g[0][d] * ir * ir)
    return torch.stack([torch.zeros_like(ir), *tau, vel[0] * tau[0] + vel[1] * tau[1] + vel[2] * tau[2] - heat])


def _interface(flux, L, R, d):
    irL, vL, _, pL = _prim(L)
    irR, vR, _, pR = _prim(R)
    cL, cR = torch.sqrt(GAM * pL * irL), torch.sqrt(GAM * pR * irR)
    a, b = vL[d], vR[d]
    if flux == "rusanov":
        s = torch.maximum(a.abs() + cL, b.abs() + cR)
        return 0.5 * (_euler(L, d) + _euler(R, d) - s * (R - L))
    one, zero = torch.ones_like(a), torch.zeros_like(a)
    if flux == "ausm+":
        cm = torch.maximum(cL, cR)
        mL, mR = a / cm, b / cm
        bL, bR = mL * mL - 1, mR * mR - 1
        mp = torch.where(mL.abs() >= 1, 0.5 * (mL + mL.abs()), 0.25 * (mL + 1) ** 2 + 0.125 * bL * bL)
        pp = torch.where(mL.abs() >= 1, torch.where(mL > 0, one, zero),
                         0.25 * (mL + 1) ** 2 * (2 - mL) + 0.1875 * mL * bL * bL)
        mm = torch.where(mR.abs() >= 1, 0.5 * (mR - mR.abs()), -0.25 * (mR - 1) ** 2 - 0.125 * bR * bR)
        pm = torch.where(mR.abs() >= 1, torch.where(mR < 0, one, zero),
                         0.25 * (mR - 1) ** 2 * (2 + mR) - 0.1875 * mR * bR * bR)
        m = mp + mm
        pf = pp * pL + pm * pR
        up = m > 0
        mdot = m * cm * torch.where(up, L[0], R[0])
    else:
        q2L, q2R = sum(x * x for x in vL), sum(x * x for x in vR)
        cf = 0.5 * (cL + cR)
        mL, mR = a / cf, b / cf
        qbar = torch.sqrt(0.5 * (q2L + q2R))
        chi = (1 - (qbar / cf).clamp_max(1.0)) ** 2
        g = -mL.clamp(-1, 0) * mR.clamp(0, 1)
        vbar = (L[0] * a.abs() + R[0] * b.abs()) / (L[0] + R[0])
        mdot = 0.5 * (L[0] * (a + (1 - g) * vbar + g * a.abs()) + R[0] * (b - (1 - g) * vbar - g * b.abs())
                      - chi / cf * (pR - pL))
        bL = torch.where(mL.abs() < 1, 0.25 * (2 - mL) * (mL + 1) ** 2, torch.where(mL >= 0, one, zero))
        bR = torch.where(mR.abs() < 1, 0.25 * (2 + mR) * (mR - 1) ** 2, torch.where(mR >= 0, zero, one))
        pf = 0.5 * (pL + pR) + 0.5 * (bL - bR) * (pL - pR) + qbar * (bL + bR - 1) * cf * 0.5 * (L[0] + R[0])
        up = mdot > 0
    W = torch.where(up, L, R)
    irW, vW, _, pW = _prim(W)
    f = [mdot, mdot * vW[0], mdot * vW[1], mdot * vW[2], mdot * (W[4] + pW) * irW]
    f[1 + d] = f[1 + d] + pf
    return torch.stack(f)


class _Exact:
    """The FR P=3 right-hand side and SSP-RK3 of one mesh, float64 torch."""

    def __init__(self, n, ext, wall, flux, mu, forcing, suth):
        self.n, self.wall, self.flux = n, wall, flux
        self.mu, self.forcing, self.suth = mu, forcing, suth
        _, self.D, self.eL, self.eR, self.gL, self.gR = _operators()
        self.jac = [2.0 * n[d] / float(np.float32(ext[d])) for d in range(3)]

    @staticmethod
    def _sum(q, w, ax):
        return sum(float(w[m]) * q.select(ax, m) for m in range(4))

    def _deriv(self, q, ax):
        return torch.stack([self._sum(q, self.D[a], ax) for a in range(4)], dim=ax)

    @staticmethod
    def _spread(f, w, ax):
        return torch.stack([float(w[a]) * f for a in range(4)], dim=ax)

    def rhs(self, u):
        nx, ny, nz = self.n
        q = u.reshape(5, nz, ny, nx, 4, 4, 4)
        tr, grad = [], []
        for d in range(3):
            el, ax = 3 - d, 6 - d
            tL, tR = self._sum(q, self.eL, ax), self._sum(q, self.eR, ax)
            nL, nR = torch.roll(tR, 1, el), torch.roll(tL, -1, el)
            if d == 1 and self.wall:
                refl = torch.tensor([1.0, -1, -1, -1, 1], device=q.device, dtype=q.dtype).reshape(5, 1, 1, 1, 1)
                nL[:, :, 0] = refl * tL[:, :, 0]
                nR[:, :, -1] = refl * tR[:, :, -1]
            g = self._deriv(q, ax) + self._spread(0.5 * (nL - tL), self.gL, ax) + self._spread(0.5 * (nR - tR),
                                                                                               self.gR, ax)
            grad.append(self.jac[d] * g)
            tr.append((tL, tR))
        g = [[grad[b][v] for b in range(3)] for v in range(5)]
        out = torch.zeros_like(q)
        for d in range(3):
            out -= self.jac[d] * self._deriv(_euler(q, d) - _viscous(q, g, d, self.mu, self.suth), 6 - d)
        out[1] += self.forcing
        for d in range(3):
            el, ax = 3 - d, 6 - d
            tL, tR = tr[d]
            gL = [[self._sum(g[v][b], self.eL, ax - 1) for b in range(3)] for v in range(5)]
            gR = [[self._sum(g[v][b], self.eR, ax - 1) for b in range(3)] for v in range(5)]
            vL, vR = _viscous(tL, gL, d, self.mu, self.suth), _viscous(tR, gR, d, self.mu, self.suth)
            fi = _interface(self.flux, torch.roll(tR, 1, el), tL, d)
            jL = fi - 0.5 * (vL + torch.roll(vR, 1, el)) - (_euler(tL, d) - vL)
            jR = torch.roll(fi, -1, el) - 0.5 * (vR + torch.roll(vL, -1, el)) - (_euler(tR, d) - vR)
            if d == 1 and self.wall:
                for j, t, at in ((jL, tL, 0), (jR, tR, -1)):
                    s = t[:, :, at]
                    w = -_euler(s, 1)
                    w[2] += _prim(s)[3]
                    j[:, :, at] = w
            out -= self.jac[d] * (self._spread(jL, self.gL, ax) + self._spread(jR, self.gR, ax))
        return out.reshape(u.shape)

    def steps(self, u, n, dt, more=None):
        f = self.rhs if more is None else lambda x: self.rhs(x) + more(x)
        for _ in range(n):
            a = u + dt * f(u)
            a = 0.75 * u + 0.25 * a + 0.25 * dt * f(a)
            u = u / 3.0 + 2.0 / 3.0 * a + 2.0 / 3.0 * dt * f(a)
        return u


def _features64(u, n, ext):
    """Standardised closure inputs [elements x 896] in float64."""
    nx, ny, nz = n
    D = _operators()[1]
    q = u.reshape(5, nz, ny, nx, 4, 4, 4)
    d = []
    for b in range(3):
        ax = 6 - b
        d.append(2.0 * n[b] / float(np.float32(ext[b])) * torch.stack(
            [sum(float(D[a, m]) * q.select(ax, m) for m in range(4)) for a in range(4)], dim=ax))
    ch = [q[v] for v in range(5)]
    for a in range(3):
        ch += [(d[b][1 + a] - q[1 + a] / q[0] * d[b][0]) / q[0] for b in range(3)]
    ch = torch.stack(ch).reshape(14, nx * ny * nz, 64).permute(1, 0, 2)
    m, s = (torch.tensor(x, device=u.device, dtype=u.dtype).reshape(1, 14, 1) for x in (FEAT_MEAN, FEAT_SCALE))
    return ((ch - m) / s).clamp(-8, 8).reshape(nx * ny * nz, 896)


def _layers64(seed):
    p = _net_params(seed)
    return [(torch.tensor(p[f"W{k}"], device=DEV).double(), torch.tensor(p[f"b{k}"], device=DEV).double())
            for k in (1, 2, 3, 4)]


def _net64(layers, x):
    for k, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if k < 3:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    return x


def _train64(case, seed):
    X, T, rows = _pools(case, seed)
    layers = [tuple(t.requires_grad_() for t in wb) for wb in _layers64(seed)]
    flat = [t for wb in layers for t in wb]
    m1, m2 = [torch.zeros_like(t) for t in flat], [torch.zeros_like(t) for t in flat]
    losses = []
    for k, r in enumerate(rows):
        at = torch.from_numpy(r).to(DEV)
        loss = ((_net64(layers, X[at].double())[:, :320] - T[at].double()) ** 2).mean()
        losses.append(float(loss))
        for t, g, a, b in zip(flat, torch.autograd.grad(loss, flat), m1, m2):
            a.mul_(0.9).add_(0.1 * g)
            b.mul_(0.999).add_(0.001 * g * g)
            with torch.no_grad():
                t -= 1e-3 * (a / (1 - 0.9 ** (k + 1))) / (torch.sqrt(b / (1 - 0.999 ** (k + 1))) + 1e-8)
    p = {}
    for k, (w, b) in enumerate(layers):
        p[f"W{k + 1}"], p[f"b{k + 1}"] = w.detach(), b.detach()
    return {"loss": losses, "params": p}


def _diag64(u, n, ext):
    nx, ny, nz = n
    xi, D = _operators()[:2]
    w = torch.tensor(np.polynomial.legendre.leggauss(4)[1], device=u.device)
    q = u.reshape(5, nz, ny, nx, 4, 4, 4)
    h = [float(np.float32(ext[d])) / n[d] for d in range(3)]
    d = []
    for b in range(3):
        ax = 6 - b
        d.append(2.0 / h[b] * torch.stack([sum(float(D[a, m]) * q[:4].select(ax, m) for m in range(4))
                                           for a in range(4)], dim=ax))
    vel = [q[1 + a] / q[0] for a in range(3)]
    dv = lambda a, b: (d[b][1 + a] - vel[a] * d[b][0]) / q[0]   # noqa: E731
    om = [dv(2, 1) - dv(1, 2), dv(0, 2) - dv(2, 0), dv(1, 0) - dv(0, 1)]
    wk, wj, wi = w.reshape(4, 1, 1), w.reshape(1, 4, 1), w.reshape(1, 1, 4)
    vol = wk * wj * wi * (h[0] * h[1] * h[2] / 8)
    total = lambda f: float((f * vol).sum())   # noqa: E731
    sq = lambda x: x[0] * x[0] + x[1] * x[1] + x[2] * x[2]   # noqa: E731
    rows = [q[0], *vel, vel[0] ** 2, vel[1] ** 2, vel[2] ** 2, vel[0] * vel[1]]
    plane = wk * wi * (h[0] * h[2] / 4) / (h[0] * nx * h[2] * nz)
    prof = torch.stack([(f * plane).sum(dim=(0, 2, 3, 5)).reshape(-1) for f in rows], dim=1)
    return {"mass": total(q[0]), "momentum_x": total(q[1]), "energy": total(q[4]),
            "kinetic_energy": total(0.5 * q[0] * sq(vel)), "enstrophy": total(0.5 * q[0] * sq(om)),
            "volume": total(torch.ones_like(q[0])), "profiles": prof}


def _fields64(u, n):
    nx, ny, nz = n
    q = u.reshape(5, nz, ny, nx, 4, 4, 4)
    k2 = q[1] ** 2 + q[2] ** 2 + q[3] ** 2
    r = q[0].clamp_min(1e-30)
    f = torch.stack([*q, torch.sqrt(k2) / r, (0.4 * (q[4] - 0.5 * k2 / r)).clamp_min(1e-7)])
    return f.permute(0, 3, 6, 2, 5, 1, 4).reshape(7, 4 * nx, 4 * ny, 4 * nz)


def _project64(u, nc, f):
    """L2 projection onto coarse elements f times larger per axis."""
    xi, w = np.polynomial.legendre.leggauss(4)
    P = np.zeros((4, f, 4))
    for q in range(f):
        for a in range(4):
            lag = _lagrange(xi, -1.0 + (2.0 * q + 1.0 + xi[a]) / f)
            for i in range(4):
                P[i, q, a] = w[a] * lag[i] / (f * w[i])
    P = torch.tensor(P, device=u.device)
    t = u.reshape(5, nc, f, nc, f, nc, f, 4, 4, 4)
    t = torch.einsum("vzcybxakji,lai->vzcybxkjl", t, P)
    t = torch.einsum("vzcybxkjl,mbj->vzcyxklm", t, P)
    t = torch.einsum("vzcyxklm,nck->vzyxnml", t, P)
    return t.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, seed)
    if kind == "ensemble":
        out = []
        for b, x in enumerate(_boxes(case, seed)):
            u = _flow(x.n, x.extent, x.y_wall, x.mach, seed + 1000 * b).float().double()
            e = _Exact(x.n, x.extent, x.y_wall, x.flux, x.mu, x.forcing, -1.0)
            out.append(e.steps(u, case["steps"], float(np.float32(x.dt))))
        return out
    if kind == "data":
        nc, f = case["coarse"], case["factor"]
        u = _flow((nc * f,) * 3, CHANNEL, True, 0.2, seed).float().double()
        c = _project64(u, nc, f)
        return {"coarse": c, "features": _features64(c, (nc,) * 3, CHANNEL)}
    s = _setup(case)
    u = _input(case, seed).double()
    if kind == "diag":
        return _diag64(u, s["n"], s["ext"])
    if kind == "fields":
        return _fields64(u.float().double(), s["n"])
    e = _Exact(s["n"], s["ext"], s["wall"], s["flux"], s["mu"], s["forcing"], s["suth"])
    if kind == "rhs":
        return e.rhs(u)
    more = None
    if case["closure"]:
        layers = _layers64(seed)
        sc = torch.tensor(OUT_SCALE, device=DEV).double().reshape(5, 1, 1)
        more = lambda x: (sc * _net64(layers, _features64(x, s["n"], s["ext"]))[:, :320]  # noqa: E731
                          .reshape(-1, 5, 64).permute(1, 0, 2)).reshape(-1)
    return e.steps(u, case["steps"], s["dt"], more)
