"""The workloads whose speed is measured, as a user's program runs them.

A case is one pass through the package's public calls: the resident solver
(set_flow, step, get_flow), the three kernel entry points on the reference's
buffers (U_Q, Viscous, Weno per stage, FLOW written and read by the host), the
batch of independent lattices, and the allocation-free stage.  Flows are the
Taylor-Green vortex, the isentropic vortex, the shocked slab, the wall-bounded
channel and the NACA0012 O-grid of the package's case generators, started from
a state that the seed moves about.

Results of the FP64 form are returned as the calls give them.  The reduced
forms compute in 32 bits, and a program that chooses them keeps its snapshots
in 32 bits too, so their FLOW is returned as float32.  Row 0 of every
reference array is the layout's dummy row and is left out.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from cfd_gb300 import abi, cases, runtime  # noqa: E402

PRECISION = {"fp64": 0, "mixed": 1, "split": 2}
U, V, W, P, T, RHO, MU, A, E = range(9)      # columns of FLOW


def listed():
    return [
        # the headline grid: one step between two host exchanges of FLOW
        dict(name="tgv128_fp64", path="solver", flow="tgv", precision="fp64", ni=128, nj=128, nk=128, steps=1),
        # the same grid in the two reduced forms, ten steps between exchanges
        dict(name="tgv128_split", path="solver", flow="tgv", precision="split", ni=128, nj=128, nk=128, steps=10),
        dict(name="tgv128_mixed", path="solver", flow="tgv", precision="mixed", ni=128, nj=128, nk=128, steps=10),
        # a reference host that swaps its three OpenCL launches for the drop-in calls
        dict(name="tgv96_kernels", path="kernels", flow="tgv", precision="fp64", ni=96, nj=96, nk=96, steps=1),
        # the inviscid vortex configuration (a flow that stays two-dimensional)
        dict(name="vortex64_fp64", path="solver", flow="vortex", precision="fp64", ni=64, nj=64, nk=64, steps=2),
        # airfoil O-grid with walls and far field: loc codes, ghosts, boundary routine
        dict(name="naca_split", path="solver", flow="naca", precision="split", ni=256, nj=64, nk=16, steps=10),
        # a small wall-bounded case with no round extent, in full precision
        dict(name="channel_fp64", path="solver", flow="channel", precision="fp64", ni=47, nj=33, nk=29, steps=1),
        # shocks on a curvilinear lattice with odd extents
        dict(name="shock_mixed", path="solver", flow="shock", precision="mixed", ni=161, nj=45, nk=51, steps=10),
        # many small solves advanced together, as the serving loop runs them
        dict(name="batch_split", path="batch", flow="vortex", precision="split", lo=24, hi=72, count=24, steps=5),
        dict(name="batch_fp64", path="batch", flow="vortex", precision="fp64", lo=24, hi=48, count=8, steps=1),
        # the smallest calls: a single step of a small lattice, a stage without allocations
        dict(name="tgv24_mixed", path="solver", flow="tgv", precision="mixed", ni=24, nj=24, nk=24, steps=1),
        dict(name="static17_fp64", path="static", flow="tgv", precision="fp64", ni=17, nj=17, nk=17, steps=1),
    ]


def draw(rng):
    path = rng.choices(["solver", "kernels", "batch", "static"], [6, 1, 2, 1])[0]

    def nodes(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def extents(n, least=10):
        edge = n ** (1 / 3)
        a, b = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
        return tuple(max(least, round(e)) for e in (edge * a, edge * b, edge / (a * b)))

    if path == "batch":
        precision = rng.choice(["fp64", "split", "mixed"])
        lo = rng.randint(12, 32)
        hi = rng.randint(lo + 1, 40 if precision == "fp64" else 64)
        return dict(path=path, flow="vortex", precision=precision, lo=lo, hi=hi, count=rng.randint(2, 24),
                    steps=1 if precision == "fp64" else rng.randint(1, 5))
    if path == "static":
        ni, nj, nk = extents(nodes(1000, 20000))
        return dict(path=path, flow="tgv", precision="fp64", ni=ni, nj=nj, nk=nk, steps=1)
    if path == "kernels":
        ni, nj, nk = extents(nodes(4000, 500000))
        return dict(path=path, flow="tgv", precision="fp64", ni=ni, nj=nj, nk=nk, steps=1)
    precision = rng.choice(["fp64", "split", "mixed"])
    flow = rng.choice(["tgv", "tgv", "vortex", "shock", "channel", "naca"])
    n = nodes(4000, 700000)
    if flow == "naca":
        nk = rng.randint(8, 24)
        nj = rng.randint(24, 64)
        ni, nj, nk = 4 * max(12, min(80, round(n / (4 * nj * nk)))), nj, nk
    else:
        ni, nj, nk = extents(n, 12 if flow == "channel" else 10)
    return dict(path=path, flow=flow, precision=precision, ni=ni, nj=nj, nk=nk,
                steps=rng.randint(1, 2) if precision == "fp64" else rng.randint(1, 10))


def _shapes(case):
    """Extents of every lattice of the case."""
    if case["path"] != "batch":
        return [(case["ni"], case["nj"], case["nk"])]
    q = max(1, case["count"] - 1)
    return [(round(case["lo"] * (case["hi"] / case["lo"]) ** (m / q)),) * 3 for m in range(case["count"])]


@functools.lru_cache(maxsize=40)
def _mesh(flow, shape):
    """Grid, metrics and base state of one lattice: a mesh is made once and
    serves every state that is started on it."""
    if flow == "tgv":
        return cases.taylor_green(shape=shape)
    if flow == "vortex":
        return cases.isentropic_vortex(shape=shape)
    if flow == "shock":
        return cases.shock_slab(shape=shape)
    return (cases.channel if flow == "channel" else cases.naca0012)(*shape)


def _fill(f, rho, u, v, w, p, mach):
    f[:, RHO], f[:, U], f[:, V], f[:, W], f[:, P] = rho, u, v, w, p
    f[:, T] = (1.4 * mach * mach) * (p / rho)
    f[:, A] = np.sqrt(1.4 * p / rho)
    f[:, E] = p / (0.4 * rho)
    f[:, MU] = 0.0


def _flow(flow, mesh, rng):
    """The seed's initial FLOW on a mesh."""
    out = mesh.arrays["flow"].copy()
    g, f, mach = mesh.arrays["grid"][1:], out[1:], mesh.params.mach
    x, y, z = (np.ascontiguousarray(g[k]) for k in "xyz")
    ph = rng.uniform(0.0, 2 * math.pi, 8)
    if flow == "tgv":           # the vortex shifted, with a weak three-dimensional disturbance
        X, Y, Z = x + ph[0], y + ph[1], z + ph[2]
        u = np.sin(X) * np.cos(Y) * np.cos(Z) + 0.02 * np.sin(2 * Y + ph[3])
        v = -np.cos(X) * np.sin(Y) * np.cos(Z) + 0.02 * np.sin(2 * Z + ph[4])
        w = 0.02 * np.sin(2 * X + ph[5])
        p = 1 / (1.4 * mach * mach) + (np.cos(2 * X) + np.cos(2 * Y)) * (np.cos(2 * Z) + 2.0) / 16.0
        rho = np.ones_like(u)
    elif flow == "vortex":      # centre and strength
        L, beta = 10.0, rng.uniform(4.0, 5.5)
        cx, cy = rng.uniform(0, L, 2)
        xr, yr = (x - cx + L / 2) % L - L / 2, (y - cy + L / 2) % L - L / 2
        r2 = xr * xr + yr * yr
        ex = np.exp(0.5 * (1.0 - r2))
        u, v = 0.5 - beta / (2 * math.pi) * ex * yr, beta / (2 * math.pi) * ex * xr
        w = np.zeros_like(u)
        rho = (1.0 - 0.4 * beta * beta / (8 * 1.4 * math.pi ** 2) * np.exp(1.0 - r2)) ** 2.5
        p = rho ** 1.4
    elif flow == "shock":       # place and strength of the slab, its edges a few cells wide
        p_inf, cell = 1 / (1.4 * mach * mach), 2 * math.pi / mesh.shape[0]
        d = 0.5 * math.pi - np.abs((x - ph[0]) % (2 * math.pi) - math.pi)
        inside = 0.5 * (1.0 + np.tanh(d / (1.5 * cell)))
        rho = 1.0 + rng.uniform(2.6, 3.2) * inside
        p = p_inf * (1.0 + rng.uniform(7.0, 9.0) * inside)
        u = np.full_like(rho, 1.5 / mach)
        v, w = 0.02 * np.sin(z + ph[1]), 0.02 * np.sin(y + ph[2])
    else:                       # bounded flows: one per cent disturbance of the base state
        k = 2 * math.pi / np.array([np.ptp(x), np.ptp(y), np.ptp(z)])
        rho, p = f[:, RHO].copy(), f[:, P] * (1 + 0.01 * np.sin(k[0] * x + ph[0]))
        u = f[:, U] * (1 + 0.01 * np.sin(k[1] * y + ph[1]))
        v = f[:, V] + 0.01 * np.sin(k[2] * z + ph[2])
        w = f[:, W] + 0.01 * np.sin(k[0] * x + ph[3])
    _fill(f, rho, u, v, w, p, mach)
    return out


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    meshes = [_mesh(case["flow"], s) for s in _shapes(case)]
    return [(m, _flow(case["flow"], m, rng)) for m in meshes]


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


BUFFERS = {"U0": 5, "U1": 5, "U2": 5, "Q": 5, "F": 5, "E": 5, "G": 5, "Fv": 5, "Ev": 5, "Gv": 5, "roe": 36, "L": 5,
           "flow": 9}


def _device(mesh, names):
    """Device buffers of the reference layout: geometry copied, the rest zero."""
    rows = mesh.n_rows
    d = {n: torch.zeros(rows, BUFFERS[n], dtype=torch.float64, device="cuda") for n in names}
    for n in ("det", "deter", "metric"):
        d[n] = torch.from_numpy(mesh.arrays[n]).to("cuda")
    d["grid"] = torch.from_numpy(mesh.arrays["grid"].view(np.uint8).reshape(rows, -1)).to("cuda")
    return d


def prepare(case, seed):
    inputs = _inputs(case, seed)
    s = {"case": case, "dt": 0.8 * min(m.dt for m, _ in inputs)}
    mesh, flow = inputs[0]
    if case["path"] == "static":
        s["params"] = runtime.to_params(mesh.params)
        s["buf"] = _device(mesh, ("U0", "U1", "U2", "flow", "L"))
        s["flow0"] = torch.from_numpy(flow).to("cuda")
        return s
    s["ctx"] = runtime.Context(0)
    if case["path"] == "batch":
        b = s["batch"] = runtime.Batch(s["ctx"], precision=PRECISION[case["precision"]])
        s["slots"] = [(b.add(m, flow=f, dt=s["dt"]), f) for m, f in inputs]
        b.tune()
        return s
    s["in"], s["out"], s["mesh"] = _pinned(flow), _pinned(np.zeros_like(flow)), mesh
    if case["path"] == "kernels":
        s["buf"] = _device(mesh, BUFFERS)
        s["ptr"] = {k: v.data_ptr() for k, v in s["buf"].items()}
        s["ctx"].set_rows(mesh.n_rows)
        return s
    s["solver"] = runtime.Solver(s["ctx"], mesh, precision=PRECISION[case["precision"]])
    return s


def _kept(flow, case):
    """A FLOW snapshot as the program keeps it (rows 1..)."""
    rows = torch.from_numpy(flow)[1:]
    return rows if case["precision"] == "fp64" else rows.float()


def run(state):
    case, dt = state["case"], state["dt"]
    if case["path"] == "solver":
        s = state["solver"]
        s.set_flow(state["in"])
        s.step(dt, case["steps"])
        return {"flow": _kept(s.get_flow(state["out"]), case)}
    if case["path"] == "batch":
        b = state["batch"]
        for slot, flow in state["slots"]:
            b.set_flow(slot, flow)
        b.step(case["steps"])
        return {"flow": [_kept(b.get_flow(slot), case) for slot, _ in state["slots"]]}
    if case["path"] == "kernels":
        ctx, mesh, ptr = state["ctx"], state["mesh"], state["ptr"]
        ctx.write(ptr["flow"], state["in"])
        for _ in range(case["steps"]):
            for j in range(3):
                ctx.stage(ptr, mesh.g_node, mesh.sd_node, mesh.params, j, dt)
        ctx.read(state["out"], ptr["flow"])
        return {"flow": _kept(state["out"], case), "U0": state["buf"]["U0"][1:]}
    b = state["buf"]
    b["flow"].copy_(state["flow0"])
    for _ in range(case["steps"]):
        for j in range(3):
            st = abi.load().cfd_lattice_stage_static(
                torch.cuda.current_stream().cuda_stream, case["ni"], case["nj"], case["nk"], j, dt,
                ctypes.byref(state["params"]),
                *(b[k].data_ptr() for k in ("det", "deter", "metric", "U0", "U1", "U2", "flow", "L")))
            if st != abi.OK:
                raise abi.CfdError(st, "cfd_lattice_stage_static")
    return {"flow": b["flow"][1:], "U0": b["U0"][1:], "L": b["L"][1:]}


def work(case):
    """FLOW read and written once, and per step what an ideal fused kernel
    moves: 5 state reads and 3 writes of 40 B and 22 doubles of geometry per
    stage, 848 B; about 45,000 operations per node and step (three stages of
    three faces and a viscous node)."""
    n = sum(a * b * c for a, b, c in _shapes(case))
    return {"bytes": n * (144.0 + 848.0 * case["steps"]), "flops": 45000.0 * n * case["steps"]}


# ------------------------------------------------------------- 64 bits ---
# The method written out over whole arrays: rows of the reference tables,
# neighbours by index, every formula in 64 bits.

def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    inputs = _inputs(case, seed)
    dt = 0.8 * min(m.dt for m, _ in inputs)
    got = []
    for mesh, flow in inputs:
        e = _Exact(mesh, flow, dt, dev)
        for _ in range(case["steps"]):
            for j in range(3):
                e.stage(j)
        got.append(e)
    if case["path"] == "batch":
        return {"flow": [e.f[1:] for e in got]}
    out = {"flow": got[0].f[1:]}
    if case["path"] in ("kernels", "static"):
        out["U0"] = got[0].u[0][1:]
    if case["path"] == "static":
        out["L"] = got[0].rhs[1:]
    return out


def _central(f):
    return (8.0 * (f[4] - f[2]) - (f[5] - f[1])) / 12.0


def _weno(c, eps):
    """Right-biased WENO5 value between c[2] and c[3]."""
    m, a, b, d, e = c[1], c[2], c[3], c[4], c[5]
    p = [15 / 8 * b - 5 / 4 * d + 3 / 8 * e, 3 / 8 * a + 3 / 4 * b - d / 8, -m / 8 + 3 / 4 * a + 3 / 8 * b]
    s = [13 / 12 * (b - 2 * d + e) ** 2 + 0.25 * (3 * b - 4 * d + e) ** 2,
         13 / 12 * (a - 2 * b + d) ** 2 + 0.25 * (a - d) ** 2,
         13 / 12 * (m - 2 * a + b) ** 2 + 0.25 * (m - 4 * a + 3 * b) ** 2]
    w = [k / (eps + q) ** 2 for k, q in zip((1 / 16, 5 / 8, 5 / 16), s)]
    return (w[0] * p[0] + w[1] * p[1] + w[2] * p[2]) / (w[0] + w[1] + w[2])


def _contravariant(q, m):
    """Euler flux of conservative rows q through the vector m, and U.m, c^2."""
    rho = q[:, 0]
    vel = q[:, 1:4] / rho[:, None]
    ke = 0.5 * (vel * vel).sum(1)
    e = q[:, 4] / rho - ke
    p = 0.4 * rho * e
    un = (vel * m).sum(1)
    flux = torch.cat([(rho * un)[:, None], q[:, 1:4] * un[:, None] + m * p[:, None], ((q[:, 4] + p) * un)[:, None]], 1)
    return flux, un, 0.56 * e


class _Exact:
    def __init__(self, mesh, flow, dt, dev):
        a = mesh.arrays

        def put(x):
            return torch.from_numpy(np.ascontiguousarray(x)).to(dev)

        self.prm, self.dt, self.sd = mesh.params, dt, mesh.sd_node
        self.nb = [put(a["grid"]["N%d" % s]).long() for s in range(6)]
        self.f, self.det = put(flow), put(a["det"])
        self.m = put(a["metric"][:, :9]).reshape(-1, 3, 3)
        self.fm = [put(a["metric"][:, 9 * (1 + 2 * d) + 3 * d:9 * (1 + 2 * d) + 3 * d + 3]) for d in range(3)]
        self.fdet = [put(a["deter"][:, 2 * d]) for d in range(3)]
        loc = put(a["grid"]["loc"]).long()
        rows = torch.arange(loc.numel(), device=dev)
        self.off, self.vb, self.wb = [], [], []
        for d in range(3):
            o = {0: rows}
            for k in (1, 2, 3):
                o[k], o[-k] = self.nb[(1, 0, 4)[d]][o[k - 1]], self.nb[(3, 2, 5)[d]][o[1 - k]]
            self.off.append(o)
            self.vb.append(self._branch(loc, o, True))
            self.wb.append(self._branch(loc, o, False))
        self.u, self.rhs = [None] * 3, None
        self.bc = []
        if mesh.bc is not None:
            for kind in ("outlet", "inlet", "boundary", "wall"):
                b = put(getattr(mesh.bc, kind)).long()
                for code in range(1, 7):        # face codes; these flows have no others
                    sel = b[loc[b] == code]
                    if sel.numel():
                        self.bc.append((kind, sel, self._chain(sel, (0, 2, 3, 0, 1, 4, 5)[code]),
                                        self._chain(sel, (0, 0, 1, 2, 3, 5, 4)[code])))

    def _chain(self, b, slot):
        out = []
        for _ in range(3):
            b = self.nb[slot][b]
            out.append(b)
        return out

    @staticmethod
    def _branch(loc, o, viscous):
        """Which difference formula a row takes along a direction: 1, 2
        one-sided, 3, 4 biased, 5 central, 0 none; None: central everywhere."""
        if not bool((loc != 0).any()):
            return None
        at = {k: loc[o[k]] for k in (-2, -1, 0, 1, 2)}
        edge, inner = (at[0] > 0) & (at[0] <= 52), at[0] == 0
        b = torch.full_like(loc, 0 if viscous else 5)
        b[edge & (at[1] == 100)] = 1
        b[edge & (at[-1] == 100)] = 2
        b[inner & (at[1] > 0) & (at[1] <= 52) & (at[2] == 100)] = 3
        b[inner & (at[-1] > 0) & (at[-1] <= 52) & (at[-2] == 100)] = 4
        if viscous:
            b[(at[0] != 100) & (at[-2] != 100) & (at[-1] != 100) & (at[1] != 100) & (at[2] != 100)] = 5
        return b

    def _derivative(self, x, d, branch):
        f = [x[self.off[d][k]] for k in range(-3, 4)]
        c = _central(f)
        if branch is None:
            return c
        b = branch[:, None]
        for k, v in ((1, (11 * f[3] - 18 * f[2] + 9 * f[1] - 2 * f[0]) / 6),
                     (2, (-11 * f[3] + 18 * f[4] - 9 * f[5] + 2 * f[6]) / 6),
                     (3, (2 * f[4] + 3 * f[3] - 6 * f[2] + f[1]) / 6),
                     (4, (-2 * f[2] - 3 * f[3] + 6 * f[4] - f[5]) / 6), (0, torch.zeros_like(c))):
            c = torch.where(b == k, v, c)
        return c

    def _viscous(self, u):
        """Contravariant viscous and SGS fluxes [3] of rows, and the viscosity."""
        prm, m = self.prm, self.m
        vel, rho = u[:, 1:4] / u[:, :1], u[:, 0]
        temp = 1.4 * 0.4 * prm.mach ** 2 * (u[:, 4] / rho - 0.5 * (vel * vel).sum(1))
        S = 110.4 / prm.t_inf
        mu = temp ** 1.5 * (1 + S) / (temp + S)
        if not prm.viscous:
            return None, mu
        grad, gt = 0.0, 0.0       # grad[:, a, x] = d vel_a / d x_x
        for d in range(3):
            du = self._derivative(u, d, self.vb[d])
            dv = (du[:, 1:4] - vel * du[:, :1]) / u[:, :1]
            dtemp = (du[:, 4] - u[:, 4] / rho * du[:, 0]) / rho - (vel * dv).sum(1)
            grad = grad + dv[:, :, None] * m[:, d, None, :]
            gt = gt + dtemp[:, None] * m[:, d]
        sym = grad + grad.transpose(1, 2)
        diag = torch.diagonal(grad, dim1=1, dim2=2)
        tau = sym - (2 / 3) * torch.diag_embed(diag.sum(1, keepdim=True).expand(-1, 3))
        tau = (mu / prm.reynolds)[:, None, None] * tau
        q = -(mu * 1.4 / (prm.prandtl * prm.reynolds))[:, None] * gt
        stress, heat = -tau, q - (vel[:, :, None] * tau).sum(1)
        if prm.les:
            s = 0.5 * sym
            mod = torch.sqrt(2 * (s[:, 0, 1] ** 2 + s[:, 1, 2] ** 2 + s[:, 0, 2] ** 2 + (2 / 3) * (diag ** 2).sum(1)))
            filt = self.det ** (-1 / 3)
            ed = []
            for d in range(3):
                lo, hi = self.off[d][-1], self.off[d][1]
                mean = (0.25 * u[lo, d + 1] + 0.5 * u[:, d + 1] + 0.25 * u[hi, d + 1]) / (
                    0.25 * u[lo, 0] + 0.5 * rho + 0.25 * u[hi, 0])
                k = (vel[:, d] - mean).abs()
                r = torch.where(mod != 0, filt * mod / k, torch.zeros_like(k))
                ed.append(0.03 / (1 + r / 10) * filt * k)
            x, y, z = ed
            coef = torch.stack([torch.stack([x, x, z], 1), torch.stack([x, y, y], 1), torch.stack([z, y, z], 1)], 1)
            sgs = (-2 * rho)[:, None, None] * coef * s
            qs = -1 / (1.4 * 0.4 * prm.mach ** 2) * torch.stack(ed, 1) * gt
            stress = stress + sgs
            heat = heat + 1.4 * qs + sgs.sum(2) * vel
        cart = torch.cat([torch.zeros_like(heat)[:, :, None], stress, heat[:, :, None]], 2)   # [row, x, component]
        return [self.det[:, None] * (m[:, d, :, None] * cart).sum(1) for d in range(3)], mu

    def _face(self, q, roe, d):
        """Corrected flux of every row's +1/2 face along d."""
        o, m = self.off[d], self.fm[d]
        s, vel, h = roe
        b = o[1]
        den = s + s[b]
        vel = (s[:, None] * vel + s[b, None] * vel[b]) / den[:, None]
        h, rr = (s * h + s[b] * h[b]) / den, s * s[b]
        k = m / torch.linalg.vector_norm(m, dim=1, keepdim=True)
        q2 = (vel * vel).sum(1)
        a = torch.sqrt(0.4 * (h - 0.5 * q2))
        phi, th = 0.2 * q2, (k * vel).sum(1)
        R = torch.zeros(a.numel(), 5, 5, dtype=a.dtype, device=a.device)
        L = torch.zeros_like(R)
        turn = torch.linalg.cross(vel, k, dim=1)
        g = 0.4 / (a * a)
        eye = torch.eye(3, dtype=a.dtype, device=a.device)
        for c in range(3):
            kc, e = k[:, c], eye[c].expand_as(k)
            ke = torch.linalg.cross(k, e, dim=1)
            L[:, c, 0] = kc * (1 - phi / (a * a)) - turn[:, c] / rr
            L[:, c, 1:4] = (kc * g)[:, None] * vel + ke / rr[:, None]
            L[:, c, 4] = -kc * g
            R[:, 0, c] = kc
            R[:, 1:4, c] = kc[:, None] * vel + rr[:, None] * ke
            R[:, 4, c] = kc * phi / 0.4 + rr * turn[:, c]
        beta, alpha = 1 / (math.sqrt(2) * rr * a), rr / (math.sqrt(2) * a)
        for c, sg in ((3, 1.0), (4, -1.0)):
            L[:, c, 0] = beta * (phi - sg * th * a)
            L[:, c, 1:4] = -beta[:, None] * (0.4 * vel - sg * k * a[:, None])
            L[:, c, 4] = 0.4 * beta
            R[:, 0, c] = alpha
            R[:, 1:4, c] = alpha[:, None] * (vel + sg * k * a[:, None])
            R[:, 4, c] = alpha * ((phi + a * a) / 0.4 + sg * th * a)
        c = [(L * q[o[n]][:, None, :]).sum(2) for n in range(-2, 4)]
        qp = (R * _weno(c, self.prm.weno_eps)[:, None, :]).sum(2)
        qn = (R * _weno(c[::-1], self.prm.weno_eps)[:, None, :]).sum(2)
        fp, up, cp = _contravariant(qp, m)
        fn, un, cn = _contravariant(qn, m)
        mm = (m * m).sum(1)
        lam = torch.maximum((up + torch.sqrt(cp * mm)).abs(), (un + torch.sqrt(cn * mm)).abs())
        face = 0.5 * self.fdet[d][:, None] * (fp + fn - lam[:, None] * (qp - qn))
        node = self.det[:, None] * _contravariant(q, self.m[:, d])[0]
        f = [node[o[n]] for n in range(-2, 4)]
        d2 = (-5 * f[0] + 39 * f[1] - 34 * f[2] - 34 * f[3] + 39 * f[4] - 5 * f[5]) / 48
        d4 = (f[0] - 3 * f[1] + 2 * f[2] + 2 * f[3] - 3 * f[4] + f[5]) / 2
        return face - d2 / 24 + 7 * d4 / 5760

    def stage(self, j):
        f, det, prm = self.f, self.det, self.prm
        rho, vel, p = f[:, RHO], f[:, U:W + 1], f[:, P]
        en = p / 0.4 + 0.5 * rho * (vel * vel).sum(1)
        q = torch.cat([rho[:, None], rho[:, None] * vel, en[:, None]], 1)
        self.u[j] = u = det[:, None] * q
        visc, mu = self._viscous(u)
        total = 0.0
        for d in range(3):
            face = self._face(q, (torch.sqrt(rho), vel, (en + p) / rho), d)
            total = total + (face - face[self.off[d][-1]])
            if visc is not None:
                total = total + self._derivative(visc[d], d, self.wb[d])
        self.rhs = rhs = -total
        u0, dt = self.u[0], self.dt
        new = (u0 + dt * rhs if j == 0 else 0.75 * u0 + 0.25 * u + 0.25 * dt * rhs if j == 1
               else u0 / 3 + 2 / 3 * u + 2 / 3 * dt * rhs)
        own = slice(0, self.sd + 1)
        self.u[(j + 1) % 3] = torch.cat([new[own], self.u[(j + 1) % 3][self.sd + 1:]
                                         if self.u[(j + 1) % 3] is not None else u[self.sd + 1:]])
        f = self.f = f.clone()
        f[:, MU] = mu
        c = new[own] / det[own, None]
        f[own, RHO] = c[:, 0]
        f[own, U:W + 1] = v = c[:, 1:4] / c[:, :1]
        f[own, E] = e = c[:, 4] / c[:, 0] - 0.5 * (v * v).sum(1)
        f[own, P] = 0.4 * c[:, 0] * e
        self._thermo(own)
        self._boundary()

    def _thermo(self, rows):
        f = self.f
        f[rows, T] = 1.4 * self.prm.mach ** 2 * f[rows, P] / f[rows, RHO]
        f[rows, A] = torch.sqrt(1.4 * f[rows, P] / f[rows, RHO])
        f[rows, E] = f[rows, P] / (0.4 * f[rows, RHO])

    def _boundary(self):
        f, gm2 = self.f, 1.4 * self.prm.mach ** 2
        keep = [U, V, W, P, T, RHO, A, E]
        for kind, b, inner, ghost in self.bc:
            if kind == "boundary":
                f[b[:, None], keep] = f[inner[0][:, None], keep]
            else:
                f[b, U], f[b, V], f[b, W] = (1.0 if kind == "inlet" else 0.0), 0.0, 0.0
                if kind == "outlet":
                    f[b, U:W + 1] = f[inner[0], U:W + 1]
                f[b, P] = 1 / gm2 if kind == "inlet" else f[inner[0], P]
                f[b, T] = 1.0 if kind == "inlet" else f[inner[0], T]
                f[b, RHO] = gm2 * f[b, P] / f[b, T]
                self._thermo(b)
            for s, g in zip(inner, ghost):
                src = s if kind in ("boundary", "wall") else b
                f[g[:, None], keep] = f[src[:, None], keep]
                if kind == "wall":
                    f[g, U:W + 1] = -f[s, U:W + 1]
