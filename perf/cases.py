"""Workloads of the time-advance library for timing, one pass each through its public entry points.

A case names what a program does (`kind`), its mesh, precision and options; `prepare` makes the
fields such a program holds before the call, `run` is one pass, `exact` the same result from plain
torch in 64 bits, `work` the bytes and operations the path cannot do without.

A pass of a time advance starts from the same initial state each time (the state is set by a
device-to-device copy first and read out by one afterwards), so that a pass can be repeated.
"""
import math

import torch

from novaclone_b200 import nova

DEV = "cuda"
PI2 = 2.0 * math.pi
CFL = 0.3


def listed():
    return [
        # the smallest production run: Taylor-Green at 64^3, default options (a history row per step)
        dict(name="tg64_f64_history", kind="ns", n0=64, n1=64, n2=64, prec="f64", rk="classical", steps=20, diag=1),
        # the headline run: Taylor-Green at 256^3, FP64, the state kept on the device
        dict(name="tg256_f64", kind="ns", n0=256, n1=256, n2=256, prec="f64", rk="classical", steps=5, diag=0),
        # the same in FP32-split with the monitored history a production run keeps
        dict(name="tg256_split_history", kind="ns", n0=256, n1=256, n2=256, prec="split", rk="classical", steps=5,
             diag=1),
        # a mesh that divides into no tile: channel-like box with odd and non power-of-two extents
        dict(name="ns_ragged_f64_history", kind="ns", n0=120, n1=75, n2=100, prec="f64", rk="classical", steps=10,
             diag=1),
        # 3-D Orszag-Tang MHD at 128^3 with its energy and max|div B| history
        dict(name="ot128_f64_history", kind="mhd", n0=128, n1=128, n2=128, prec="f64", rk="classical", steps=5,
             diag=1),
        # the MHD jet, 192 x 192 x 384, FP32-split, the reference app's (literal) loop
        dict(name="jet_split", kind="mhd", n0=192, n1=192, n2=384, prec="split", rk="literal", steps=2, diag=0),
        # temporal shear layer between walls in y, DCT pressure, a projection per stage
        dict(name="shear_walls_f64", kind="shear", n0=256, n1=256, n2=128, prec="f64", steps=2, diag=0),
        # weakly-compressible stratified shear layer at 256^3
        dict(name="wc_shear256", kind="wc", n0=256, n1=256, n2=256, steps=2, diag=0),
        # gradient of the final kinetic energy: forward, checkpoints, recomputation and reverse sweep
        dict(name="adjoint_tg256_f64", kind="adjoint", model="ns", n0=256, n1=256, n2=256, prec="f64", steps=4,
             every=2),
        # the explicit operators called one by one, as the reference's programs do
        dict(name="operators_128", kind="ops", n0=128, n1=128, n2=128, m=6),
        # the same on a small odd mesh, where the cost of a call counts
        dict(name="operators_small_odd", kind="ops", n0=33, n1=47, n2=29, m=6),
        # an implicit diffusion step: matrix assembly and line relaxation to a tolerance
        dict(name="implicit_128", kind="im", n0=128, n1=128, n2=128),
    ]


def _extent(rng, lo, hi):
    """half the time an extent that FFTs and tiles like, else any (odd ones among them), log-uniform"""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.5:
        return min((32, 48, 64, 96, 128, 160, 192, 256), key=lambda v: abs(math.log(v / x)))
    return max(lo, min(hi, int(round(x))))


def draw(rng):
    kind = rng.choice(["ns"] * 4 + ["mhd"] * 2 + ["shear", "wc", "adjoint"] + ["ops"] * 2 + ["im"])
    lo, hi = {"ns": (32, 256), "mhd": (32, 192), "shear": (32, 256), "wc": (32, 192), "adjoint": (32, 128),
              "ops": (24, 160), "im": (24, 160)}[kind]
    n = [_extent(rng, lo, hi) for _ in range(3)]
    if rng.random() < 0.35:
        n = [n[0]] * 3
    c = dict(kind=kind, n0=n[0], n1=n[1], n2=n[2])
    pts = n[0] * n[1] * n[2]
    if kind == "ns":
        c.update(prec=rng.choice(["f64", "split"]), rk=rng.choice(["classical", "classical", "literal"]),
                 steps=20 if pts < 500000 else (8 if pts < 4000000 else 4), diag=rng.choice([0, 1, 4]))
    elif kind == "mhd":
        c.update(prec=rng.choice(["f64", "split"]), rk=rng.choice(["classical", "literal"]),
                 steps=10 if pts < 500000 else (4 if pts < 3000000 else 2), diag=rng.choice([0, 1]))
    elif kind == "shear":
        c.update(prec=rng.choice(["f64", "split"]), steps=3 if pts < 1000000 else 1, diag=0)
    elif kind == "wc":
        c.update(steps=4 if pts < 1000000 else 1, diag=0)
    elif kind == "adjoint":
        c.update(model=rng.choice(["ns", "mhd"]), prec=rng.choice(["f64", "split"]), steps=4, every=rng.choice([2, 4]))
    elif kind == "ops":
        c.update(m=rng.choice([2, 4, 6, 6, 6, 8]))
    return c


# ------------------------------------------------------------------------------ initial fields --
def _shape(c):
    return c["n0"], c["n1"], c["n2"]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(shape, g):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _axes(N, L, org=(0.0, 0.0, 0.0)):
    x = [org[a] + torch.arange(N[a], device=DEV, dtype=torch.float64) * (L[a] / N[a]) for a in range(3)]
    return torch.meshgrid(*x, indexing="ij")


def _phase(g):
    return [float(v) for v in torch.rand(3, generator=g, device=DEV, dtype=torch.float64) * PI2]


def _box(c):
    if c["kind"] == "shear":
        return (PI2, PI2, math.pi), (0.0, 0.0, 0.0)
    if c["kind"] == "wc":
        return (2.8, 0.34, 3.0), (0.0, 0.0, 0.0)
    if c["kind"] == "mhd" and c["n2"] > 1.5 * c["n0"]:
        return (8.0, 8.0, 16.0), (-4.0, -4.0, 0.0)
    return (PI2, PI2, PI2), (0.0, 0.0, 0.0)


def _tg(N, g):
    """Taylor-Green vortex with seeded phases, and noise of amplitude 1e-3"""
    X, Y, Z = _axes(N, (PI2,) * 3)
    a, b, c = _phase(g)
    U = torch.stack([torch.sin(X + a) * torch.cos(Y + b) * torch.cos(Z + c),
                     -torch.cos(X + a) * torch.sin(Y + b) * torch.cos(Z + c), torch.zeros_like(X)])
    return U + 1e-3 * _randn(U.shape, g)


def _ot(N, g):
    """Orszag-Tang fields with seeded phases, and noise of amplitude 1e-3"""
    X, Y, Z = _axes(N, (PI2,) * 3)
    a, b, c = _phase(g)
    X, Y, Z = X + a, Y + b, Z + c
    U = torch.stack([-2.0 * torch.sin(Y), 2.0 * torch.sin(X), torch.zeros_like(X)])
    B = torch.stack([-2.0 * torch.sin(2.0 * Y) + torch.sin(Z), 2.0 * torch.sin(X) + torch.sin(Z),
                     torch.zeros_like(X)])
    return U + 1e-3 * _randn(U.shape, g), B


def _jet(N, L, org, g):
    X, Y, _ = _axes(N, L, org)
    r = torch.sqrt(X * X + Y * Y)
    z = torch.zeros_like(X)
    U = torch.stack([z, z, 0.5 * (1.0 - torch.tanh((r - 1.0) / 0.1))])
    e = 0.2 * torch.exp(-r * r)
    return U + 1e-3 * _randn(U.shape, g), torch.stack([-e * Y, e * X, torch.full_like(X, 0.5)])


def _shear(N, L, g):
    y = torch.arange(N[1] + 1, device=DEV, dtype=torch.float64) * (L[1] / N[1])
    u = torch.tanh(28.0 * (y - math.pi))[None, :, None].expand(N[0], N[1] + 1, N[2])
    U = torch.stack([u, torch.zeros_like(u), torch.zeros_like(u)])
    return U + 1e-3 * _randn(U.shape, g)


def _wc(N, L, g):
    """weakly-compressible shear layer, Mach 0.1: constants, U, T"""
    Re0, Ri0, Pr, rho0, cs, h0, t0 = 1967.0, 0.08, 7.0, 999.57, 0.0417, 0.2, 0.1
    u0 = 0.1 * cs
    mu = rho0 * u0 * h0 / Re0
    prm = dict(rho0=rho0, mu=mu, ka=mu / Pr, gz=-Ri0 * u0 * u0 / t0 / h0, K=cs * cs / 2.0 / rho0,
               dt=CFL * min(L[a] / N[a] for a in range(3)) / (cs + u0 / 2.0))
    X, _, Z = _axes(N, L)
    Z = Z - 7.5 * h0
    k0 = 2.0 * math.pi / (14.0 * h0 / 2.0)
    a, b = 0.005, 0.4177
    th, ch = torch.tanh(2.0 * Z / h0), torch.cosh(2.0 * Z / h0)

    def noise():
        return 2.0 * torch.rand(N, generator=g, device=DEV, dtype=torch.float64) - 1.0
    U = torch.stack([u0 / 2.0 * th + a * u0 / 2.0 / k0 * (-torch.cos(2 * k0 * X) + 2.0 * b * torch.cos(k0 * X)) * th / ch,
                     a * u0 / 2.0 * noise() / ch / ch, a * u0 / 2.0 * noise() / ch / ch])
    return prm, U, (t0 / 2.0 * th + a * t0 / 2.0 * noise() / ch / ch)[None]


def _fields(c, seed):
    """the case's initial fields and parameters, from the seed alone"""
    N, g = _shape(c), _gen(seed)
    L, org = _box(c)
    d = [L[a] / N[a] for a in range(3)]
    k = c["kind"]
    f = dict(N=N, L=L, org=org)
    if k == "ns" or (k == "adjoint" and c["model"] == "ns"):
        f.update(U=_tg(N, g), nu=1.0 / 1600.0)
    elif k in ("mhd", "adjoint"):
        f["U"], f["B"] = _jet(N, L, org, g) if L[2] > 10.0 else _ot(N, g)
        f["nu"] = f["eta"] = 1.0 / 1500.0 if L[2] > 10.0 else 1.0 / 1000.0
    elif k == "shear":
        f.update(U=_shear(N, L, g), nu=1.0 / 2000.0)
    elif k == "wc":
        f["prm"], f["U"], f["T"] = _wc(N, L, g)
        f["dt"] = f["prm"]["dt"]
        return f
    elif k == "ops":
        U = _tg(N, g)
        f.update(U=U, s=(torch.cos(2.0 * U[:1]) + 0.1 * _randn((1,) + N, g)), nu=1.0 / 1600.0)
        return f
    else:  # an implicit diffusion step (1/dt - nu laplacian) x = x_old / dt, written as mu laplacian(x) - x = f
        f.update(x=_tg(N, g)[:1].contiguous() + 0.1 * _randn((1,) + N, g), f=_randn((1,) + N, g), mu=1e-3, c=1.0)
        return f
    # a speed bound that does not depend on the noise's largest value
    top = {"ns": 2.0, "shear": 1.1, "mhd": 7.5}["mhd" if "B" in f else ("shear" if k == "shear" else "ns")]
    if "B" in f and L[2] > 10.0:
        top = 1.7
    f["dt"] = CFL * min(d) / top
    return f


# ------------------------------------------------------------------------------ the timed pass --
def _out(mesh, nc):
    return torch.empty((nc,) + mesh.shape, device=DEV, dtype=torch.float64)


def prepare(case, seed):
    c = case
    f = _fields(c, seed)
    k = c["kind"]
    M = nova.Mesh(f["N"], L=f["L"], origin=f["org"], m=c.get("m", 6), walls=(0, 1, 0) if k == "shear" else (0, 0, 0))
    M.set_stream(torch.cuda.current_stream().cuda_stream)
    prec = nova.F32SPLIT if c.get("prec") == "split" else nova.F64
    s = dict(kind=k, case=c, mesh=M, f=f)
    if k in ("ns", "mhd", "shear", "adjoint"):
        s["U"], s["p"] = nova.Field(M, 3, prec), nova.Field(M, 1)
        s["oU"], s["op"] = _out(M, 3), _out(M, 1)
        if "B" in f:
            s["B"], s["pB"] = nova.Field(M, 3, prec), nova.Field(M, 1)
            s["oB"] = _out(M, 3)
        if k == "shear":
            # u, w Neumann 0, v Dirichlet 0 on both walls; pressure Neumann 0
            ubc = [0] * 18
            for q in range(3):
                ubc[6 * q] = ubc[1 + 6 * q] = 2 if q == 1 else 1
            s["U"].set_bc(ubc)
            s["p"].set_bc([1, 1] + [0] * 16)
        s["rd"] = nova.run_desc(model="mhd" if "B" in f else "ns",
                                rk_mode="shear" if k == "shear" else c.get("rk", "classical"), precision=prec,
                                dt=f["dt"], nu=f["nu"], eta=f.get("eta", 0.0), diag_every=c.get("diag", 0),
                                poisson="dct" if k == "shear" else "fft")
    elif k == "wc":
        prm = f["prm"]
        s["wd"] = nova.wc_desc("shear", dt=prm["dt"], mu=prm["mu"], ka=prm["ka"], eos_k=prm["K"],
                               g=(0.0, 0.0, prm["gz"]), diag_every=c["diag"])
        s["U"], s["rho"], s["p"], s["T"] = nova.Field(M, 3), nova.Field(M, 1), nova.Field(M, 1), nova.Field(M, 1)
        s["T"].copy_from_device(f["T"].data_ptr())
        nova.wc_hydrostatic(M, s["wd"], prm["rho0"], s["T"], s["p"], s["rho"])
        f["p"], f["rho"] = _out(M, 1), _out(M, 1)
        s["p"].copy_to_device(f["p"].data_ptr())
        s["rho"].copy_to_device(f["rho"].data_ptr())
        s["out"] = {q: _out(M, 3 if q == "U" else 1) for q in ("U", "rho", "p", "T")}
    elif k == "ops":
        s["U"], s["s"] = nova.Field(M, 3), nova.Field(M, 1)
        s["U"].copy_from_device(f["U"].contiguous().data_ptr())
        s["s"].copy_from_device(f["s"].contiguous().data_ptr())
        s["p"] = nova.Field(M, 1)
        s["out"] = {q: _out(M, n) for q, n in (("grad", 3), ("gradv", 9), ("div", 1), ("curl", 3), ("lap", 3),
                                               ("adv", 3), ("p", 1))}
    else:
        s["x"], s["fld"], s["out"] = nova.Field(M, 1), nova.Field(M, 1), _out(M, 1)
        s["fld"].copy_from_device(f["f"].contiguous().data_ptr())
    torch.cuda.synchronize()
    return s


def run(s):
    return {"ns": _run_advance, "mhd": _run_advance, "shear": _run_advance, "adjoint": _run_adjoint, "wc": _run_wc,
            "ops": _run_ops, "im": _run_im}[s["kind"]](s)


def _run_advance(s):
    c, f, M = s["case"], s["f"], s["mesh"]
    B, pB = s.get("B"), s.get("pB")
    s["U"].copy_from_device(f["U"].data_ptr())
    if B is not None:
        B.copy_from_device(f["B"].data_ptr())
    hist = nova.advance(M, s["rd"], s["U"], s["p"], B, pB, nsteps=c["steps"], history=c["diag"] > 0)
    s["U"].copy_to_device(s["oU"].data_ptr())
    s["p"].copy_to_device(s["op"].data_ptr())
    if B is not None:
        B.copy_to_device(s["oB"].data_ptr())
        return {"U": s["oU"], "p": s["op"], "B": s["oB"], "hist": hist}
    return {"U": s["oU"], "p": s["op"], "hist": hist}


def _run_adjoint(s):
    c, f = s["case"], s["f"]
    s["U"].copy_from_device(f["U"].data_ptr())
    if "B" in f:
        s["B"].copy_from_device(f["B"].data_ptr())
        J, g, gB = nova.adjoint_grad(s["mesh"], s["rd"], s["U"], c["steps"], c["every"], B0=s["B"], total_energy=True)
        gB.copy_to_device(s["oB"].data_ptr())
        g.copy_to_device(s["oU"].data_ptr())
        return {"J": J, "gU": s["oU"], "gB": s["oB"]}
    J, g = nova.adjoint_grad(s["mesh"], s["rd"], s["U"], c["steps"], c["every"])
    g.copy_to_device(s["oU"].data_ptr())
    return {"J": J, "gU": s["oU"]}


def _run_wc(s):
    f, o = s["f"], s["out"]
    for q in ("U", "rho", "p", "T"):
        s[q].copy_from_device(f[q].data_ptr())
    nova.advance_wc(s["mesh"], s["wd"], s["U"], s["rho"], s["p"], s["T"], nsteps=s["case"]["steps"])
    for q in ("U", "rho", "p", "T"):
        s[q].copy_to_device(o[q].data_ptr())
    return o


def _run_ops(s):
    ex, U, o = nova.ex, s["U"], s["out"]
    got = {"grad": ex.grad(s["s"]), "gradv": ex.grad(U), "div": ex.div(U), "curl": ex.curl(U),
           "lap": ex.laplacian(s["f"]["nu"], U), "adv": ex.div(U, U)}
    top = nova.tools.maximum(got["div"])
    eq = nova.poisson(s["p"])
    eq.rhs(got["div"])
    eq.solve()
    got["p"] = s["p"]
    for q, x in got.items():
        x.copy_to_device(o[q].data_ptr())
    return {"max": top, **o}


def _run_im(s):
    f = s["f"]
    s["x"].copy_from_device(f["x"].data_ptr())
    A = nova.im.laplacian(f["mu"], s["x"])
    A.add_diagonal(-f["c"])
    A.eq(s["fld"])
    its, _ = A.solve(1e-12, 80)
    s["x"].copy_to_device(s["out"].data_ptr())
    A.close()
    return {"x": s["out"], "iterations": its}


# ------------------------------------------------------------ the same results in plain 64 bits --
COEF = {2: (1.0,), 4: (4.0 / 3.0, -1.0 / 3.0), 6: (6.0 / 4.0, -12.0 / 20.0, 1.0 / 10.0),
        8: (8.0 / 5.0, -4.0 / 5.0, 24.0 / 105.0, -8.0 / 280.0)}


class _Grid:
    """Central differences on a periodic box, or with walls at both ends of y (axis 1).
    A field is a list of (values, wall parity) with parity +1 for a mirrored (Neumann 0) and -1
    for an antimirrored (Dirichlet 0) component."""

    def __init__(self, N, L, m=6, walls=False):
        self.N, self.L, self.walls = N, L, walls
        self.d = [L[a] / N[a] for a in range(3)]
        cf = COEF[m]
        self.cf = cf
        self.a = [[cf[i] / 2.0 / (i + 1) / self.d[x] for i in range(len(cf))] for x in range(3)]
        self.b = [[cf[i] / ((i + 1) * self.d[x]) ** 2 for i in range(len(cf))] for x in range(3)]

    def sh(self, f, ax, s, par=1):
        if not (self.walls and ax == 1):
            return torch.roll(f, -s, ax)
        n, h = f.shape[1], abs(s)
        if s > 0:
            return torch.cat([f[:, s:], par * f[:, n - 1 - h:n - 1].flip(1)], 1)
        return torch.cat([par * f[:, 1:h + 1].flip(1), f[:, :n - h]], 1)

    def D(self, f, ax, par=1):
        return sum(w * (self.sh(f, ax, i + 1, par) - self.sh(f, ax, -i - 1, par)) for i, w in enumerate(self.a[ax]))

    def Q(self, f, ax):
        return sum(2.0 * w * (self.sh(f, ax, i) - self.sh(f, ax, -i - 1)) for i, w in enumerate(self.a[ax]))

    def lap(self, f, par=1):
        r = 0.0
        for ax in range(3):
            for i, w in enumerate(self.b[ax]):
                r = r + w * ((self.sh(f, ax, i + 1, par) - f) + (self.sh(f, ax, -i - 1, par) - f))
        return r

    def div(self, U, par=(1, 1, 1)):
        return sum(self.D(U[x], x, par[x]) for x in range(3))

    def grad(self, p):
        return torch.stack([self.D(p, x) for x in range(3)])

    def curl(self, U, D):
        return torch.stack([D(U[2], 1) - D(U[1], 2), D(U[0], 2) - D(U[2], 0), D(U[1], 0) - D(U[0], 1)])

    def skew(self, V, f, par=(1, 1, 1), fp=1):
        """div(V, f) = ( f div V + sum_d [ D_d(V_d f) + V_d D_d f ] ) / 2"""
        r = f * self.div(V, par)
        for x in range(3):
            r = r + self.D(V[x] * f, x, par[x] * fp) + V[x] * self.D(f, x, fp)
        return 0.5 * r

    def _k2(self, n, L, x, fold):
        i = torch.arange(n, device=DEV, dtype=torch.float64)
        kk = torch.where(2 * i < n, i, n - i) * (PI2 / L)
        kp = sum(c / (j + 1) * torch.sin((j + 1) * kk * self.d[x]) / self.d[x] for j, c in enumerate(self.cf))
        return (kp * kp)[: (n if fold else n // 2 + 1)]

    def solve(self, f):
        """p with div grad p = f in the discrete operators, its null space left out"""
        N, L = list(self.N), list(self.L)
        n1 = f.shape[1]
        if self.walls:
            f = torch.cat([f, f[:, 1:n1 - 1].flip(1)], 1)
            N[1], L[1] = 2 * N[1], 2.0 * L[1]
        k2 = (self._k2(N[0], L[0], 0, True)[:, None, None] + self._k2(N[1], L[1], 1, True)[None, :, None]
              + self._k2(N[2], L[2], 2, False)[None, None, :])
        h = torch.fft.rfftn(f)
        h = torch.where(k2 < 1e-16, torch.zeros_like(h), -h / torch.where(k2 < 1e-16, torch.ones_like(k2), k2))
        return torch.fft.irfftn(h, s=N)[:, :n1]

    def project(self, U, div, scale, par=(1, 1, 1)):
        p = self.solve(self.div(U, par) / div)
        return U - scale * self.grad(p), p


RKA, RKW = (0.5, 0.5, 1.0), (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)


def _rk(rhs, Y, dt, rk):
    if rk == "literal":  # one increment of the old state under all four weights
        return Y + dt * rhs(Y)
    s, acc = Y, Y
    for i in range(4):
        k = dt * rhs(s)
        acc = acc + RKW[i] * k
        if i < 3:
            s = Y + RKA[i] * k
    return acc


def _vec(fn):
    return torch.stack([fn(q) for q in range(3)])


def _rhs_ns(G, U, nu):
    return _vec(lambda q: nu * G.lap(U[q]) - G.skew(U, U[q]))


def _rhs_mhd_u(G, U, B, nu):
    e = 0.5 * (B * B).sum(0)
    return _vec(lambda q: nu * G.lap(U[q]) - G.skew(U, U[q]) + G.skew(B, B[q]) - G.D(e, q))


def _rhs_mhd_b(G, B, U, eta):
    return _vec(lambda q: eta * G.lap(B[q]) - G.skew(U, B[q]) + G.skew(B, U[q]))


def _row(G, f, U, B, n):
    dt = f["dt"]
    w, J = G.curl(U, G.Q).square().sum(0).sqrt(), None
    r = [float(n), n * dt, float(0.5 * U.square().sum(0).mean()), 0.0, float(G.div(U).abs().max()), 0.0,
         float(w.mean()), 0.0, 0.0, 0.0, float(U.square().sum(0).sqrt().max())]
    if B is not None:
        J = G.curl(B, G.Q).square().sum(0).sqrt()
        r[3], r[5], r[7], r[8] = (float(0.5 * B.square().sum(0).mean()), float(G.div(B).abs().max()), float(J.mean()),
                                  float(J.max()))
    r[9] = -f["nu"] * r[6] ** 2 - f.get("eta", 0.0) * r[7] ** 2
    cx = max(0.0, float(U[0].max())) * dt / G.d[0]
    r += [cx, max(cx, float(U[1][0, 0, 0]) * dt / G.d[1]), max(cx, float(U[2][0, 0, 0]) * dt / G.d[2])]
    r.append(float(0.5 * G.curl(U, G.D).square().sum(0).mean()))
    r.append(0.0 if B is None else float(0.5 * G.curl(B, G.D).square().sum(0).mean()))
    return r


def _step(G, c, f, U, B):
    dt, rk = f["dt"], c.get("rk", "classical")
    if B is None:
        U, p = G.project(_rk(lambda s: _rhs_ns(G, s, f["nu"]), U, dt, rk), dt, dt)
    else:
        U, p = G.project(_rk(lambda s: _rhs_mhd_u(G, s, B, f["nu"]), U, dt, rk), dt, dt)
        B, _ = G.project(_rk(lambda s: _rhs_mhd_b(G, s, U, f["eta"]), B, dt, "classical"), 1.0, 1.0)
    return U, B, p


def _exact_shear(c, f):
    G, nu, dt = _Grid(f["N"], f["L"], walls=True), f["nu"], f["dt"]
    par = (1, -1, 1)

    def fix(U):
        U = U.clone()
        for q in (0, 2):
            U[q][:, 0], U[q][:, -1] = U[q][:, 1], U[q][:, -2]
        U[1][:, 0] = 0.0
        U[1][:, -1] = 0.0
        return U
    U = f["U"]
    for _ in range(c["steps"]):
        U = fix(U)
        old = U
        for w, s in zip(RKW, (0.5, 0.5, 1.0, 1.0)):
            F = _vec(lambda q: nu * G.lap(U[q], par[q]) - G.skew(U, U[q], par, par[q]))
            U, p = G.project(fix(old + w * dt * F), dt * s, dt * s, par)
            U = fix(U)
    return {"U": U, "p": p[None], "hist": None}


def _exact_wc(c, f):
    G, prm, dt = _Grid(f["N"], f["L"]), f["prm"], f["dt"]
    U, T = f["U"], f["T"][0]
    col = T * G.d[2] * prm["gz"] * prm["rho0"]
    p = prm["K"] * prm["rho0"] ** 2 + torch.flip(torch.cumsum(torch.flip(col, [2]), 2), [2])
    rho = torch.sqrt(p / prm["K"])
    for _ in range(c["steps"]):
        mom0, acc = rho * U, rho * U
        gp = G.grad(p)
        for i in range(4):
            V = rho * U
            F = _vec(lambda q: prm["mu"] * G.lap(U[q]) - G.skew(V, U[q])) - gp
            F[2] -= rho * T * prm["gz"]
            acc = acc + RKW[i] * dt * F
            U = (mom0 + RKA[i] * dt * F) / rho if i < 3 else acc / rho
        rho = _rk(lambda r: -G.div(r * U), rho, dt, "classical")
        p = prm["K"] * rho * rho
        V = rho * U
        T = _rk(lambda y: prm["ka"] * G.lap(y / rho) - G.skew(V, y / rho), rho * T, dt, "classical") / rho
    return {"U": U, "rho": rho[None], "p": p[None], "T": T[None]}


def _exact_adjoint(c, f):
    from torch.utils.checkpoint import checkpoint
    G = _Grid(f["N"], f["L"])
    U0 = f["U"].clone().requires_grad_(True)
    B0 = f["B"].clone().requires_grad_(True) if "B" in f else None

    def ck(fn, *a):
        return checkpoint(fn, *a, use_reentrant=False)

    def one(q, E, F, visc, kind):
        if kind == "ns":
            return visc * G.lap(E[q]) - ck(G.skew, E, E[q])
        if kind == "u":
            return visc * G.lap(E[q]) - ck(G.skew, E, E[q]) + ck(G.skew, F, F[q]) - G.D(0.5 * (F * F).sum(0), q)
        return visc * G.lap(E[q]) - ck(G.skew, F, E[q]) + ck(G.skew, E, F[q])

    def rk(E, F, visc, kind):
        return _rk(lambda s: torch.stack([ck(one, q, s, F, visc, kind) for q in range(3)]), E, f["dt"], "classical")

    def step(U, B):
        U = ck(lambda y: G.project(y, f["dt"], f["dt"])[0], rk(U, B, f["nu"], "ns" if B is None else "u"))
        if B is not None:
            B = ck(lambda y: G.project(y, 1.0, 1.0)[0], rk(B, U, f["eta"], "b"))
        return (U,) if B is None else (U, B)
    U, B = U0, B0
    for _ in range(c["steps"]):
        r = step(U, B)
        U, B = r[0], (r[1] if len(r) > 1 else None)
    n = U[0].numel()
    J = 0.5 * U.square().sum() / n + (0.0 if B is None else 0.5 * B.square().sum() / n)
    J.backward()
    o = {"J": float(J.detach()), "gU": U0.grad}
    if B0 is not None:
        o["gB"] = B0.grad
    return o


def _exact_ops(c, f):
    G, U, s = _Grid(f["N"], f["L"], c["m"]), f["U"], f["s"][0]
    div = G.div(U)
    return {"max": float(div.abs().max()), "grad": G.grad(s),
            "gradv": torch.stack([G.Q(U[q], x) for q in range(3) for x in range(3)]), "div": div[None],
            "curl": G.curl(U, G.Q), "lap": f["nu"] * _vec(lambda q: G.lap(U[q])),
            "adv": _vec(lambda q: G.skew(U, U[q])), "p": G.solve(div)[None]}


def _exact_im(c, f):
    G, x, mu = _Grid(f["N"], f["L"]), f["x"][0], f["mu"]
    w = [mu / G.d[a] ** 2 for a in range(3)]
    low = sum(w[a] * (torch.roll(x, 1, a) + torch.roll(x, -1, a) - 2.0 * x) for a in range(3))
    rhs = low - mu * G.lap(x) + f["f"][0]
    sym = -f["c"]
    for a in range(3):
        k = torch.arange(f["N"][a], device=DEV, dtype=torch.float64) * (PI2 / f["N"][a])
        sym = sym + (w[a] * (2.0 * torch.cos(k) - 2.0)).reshape([-1 if b == a else 1 for b in range(3)])
    return {"x": torch.fft.ifftn(torch.fft.fftn(rhs) / sym).real[None], "iterations": None}


def exact(case, seed):
    c, f = case, _fields(case, seed)
    k = c["kind"]
    if k in ("shear", "wc", "adjoint", "ops", "im"):
        return {"shear": _exact_shear, "wc": _exact_wc, "adjoint": _exact_adjoint, "ops": _exact_ops,
                "im": _exact_im}[k](c, f)
    G, U, B = _Grid(f["N"], f["L"]), f["U"], f.get("B")
    rows = []
    for n in range(1, c["steps"] + 1):
        U, B, p = _step(G, c, f, U, B)
        if c["diag"]:
            rows.append(_row(G, f, U, B, n) if n % c["diag"] == 0 or n == c["steps"] else [0.0] * nova.HIST_COLS)
    out = {"U": U, "p": p[None], "hist": torch.tensor(rows, dtype=torch.float64) if rows else None}
    if B is not None:
        out["B"] = B
    return out


# ------------------------------------------------------------------------- what cannot be left out --
def work(case):
    """Bytes: each sweep over the mesh that the method's data dependences ask for reads its inputs
    and writes its outputs once.  A stage reads the stage state and (after the first) the base state
    and writes the next one; a projection reads U*, transforms along three directions there and
    back, and writes U and p.  Operations: the stencil sums, 5 N log2 N per complex transform."""
    c = case
    n = c["n0"] * c["n1"] * c["n2"]
    lg = math.log2(max(n, 2))
    w = 4 if c.get("prec") == "split" else 8
    k = c["kind"]
    fft = 2.5 * lg * 2
    proj_b, proj_f = 24 + 8 + 5 * 16 + 8 + 24 + 3 * 8, fft + 60
    stage_b, stage_f = (24 + 3 * 48 + 24) / 8 * w + 24, 4 * 140
    if k == "ns":
        if c["rk"] == "literal":
            stage_b, stage_f = 6 * w + 24, 150
        rows = c["steps"] // c["diag"] if c["diag"] else 0
        return {"bytes": n * (c["steps"] * (stage_b + proj_b) + rows * 24), "flops": n * (c["steps"] * (stage_f + proj_f) + rows * 110)}
    if k == "mhd":
        rows = c["steps"] if c["diag"] else 0
        loop_b = stage_b + 4 * 3 * w
        u_b = loop_b if c["rk"] == "classical" else 9 * w + 24
        u_f = 4 * 310 if c["rk"] == "classical" else 310
        return {"bytes": n * (c["steps"] * (u_b + loop_b + 2 * proj_b) + rows * 48),
                "flops": n * (c["steps"] * (u_f + 4 * 290 + 2 * proj_f) + rows * 220)}
    if k == "shear":
        return {"bytes": n * c["steps"] * 4 * (9 * w + proj_b), "flops": n * c["steps"] * 4 * (150 + proj_f)}
    if k == "wc":
        # U loop: U, rho, p, T and the old momentum; rho loop: rho, U; T loop: T, rho, U
        return {"bytes": n * c["steps"] * (4 * (6 * 8 + 24) + 72 + 4 * (4 * 8 + 8) + 24 + 4 * (5 * 8 + 8) + 24),
                "flops": n * c["steps"] * (4 * 220 + 4 * 40 + 4 * 110)}
    if k == "adjoint":
        loops = 2 if c["model"] == "mhd" else 1
        rec = 2.0 - c["every"] / c["steps"]
        rev_b, rev_f = 4 * 12 * w + proj_b, 4 * 260 + proj_f
        if loops == 2:
            rev_b, rev_f = rev_b + 4 * 9 * w, rev_f + 4 * 170
        return {"bytes": n * c["steps"] * loops * (rec * (stage_b + proj_b) + rev_b),
                "flops": n * c["steps"] * loops * (rec * (stage_f + proj_f) + rev_f)}
    if k == "ops":
        return {"bytes": n * 8 * ((1 + 3) + (3 + 9) + (3 + 1) + (3 + 3) + (3 + 3) + (3 + 3) + 1 + (1 + 10 + 1)),
                "flops": n * c["m"] / 6 * (18 + 54 + 18 + 39 + 60 + 160) + n * fft}
    # implicit: assembly and about 25 iterations of a residual and three line sweeps
    return {"bytes": n * (8 * 10 + 25 * (72 + 3 * 80)), "flops": n * 25 * (16 + 3 * 20)}
