"""The calls whose speed is measured, with what they need and what they should return.

The work of this package is a time step: a pressure solve, Darcy fluxes and the small
passes around them, one solve per species and one for heat, in the reference's FP64
arithmetic ("fp64", the default of a config) or with FP32 sweeps under an FP64 residual
("fp32dc").  Most cases are one of these calls through ``transportse_b200.kernels.Model``
as the driver makes it; two are whole runs (``Simulation``, ``Ensemble``).  Sizes and
fields are those of ``transportse_b200.workloads`` (a 60 x 1 x 30 slice, ensemble members
of 32 to 128 cells an axis, served cubes of 16 to 192, the 256 x 256 x 128 reservoir) and
odd ones of the same ranges.

``exact`` evaluates the same equations (tse.py:170-1494) in plain torch, 64 bits.
"""
import math

import numpy
import torch

from transportse_b200 import workloads
from transportse_b200.driver import Simulation
from transportse_b200.ensemble import Ensemble
from transportse_b200.kernels import Model

G = 9.81
EOS = dict(rho0=1000.0, species=200.0, tcoef=0.3, T0=20.0)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a config as users start with: the 2-D density-driven slice, default precision,
        # from the config module to the fields after eight steps
        dict(name="run slice fp64", kind="run", nx=60, ny=1, nz=30, steps=8, precision="fp64"),
        # a small served request's pressure solve (cubes from 16 a side), alone
        dict(name="P fp32dc 33x29x31", kind="P", nx=33, ny=29, nz=31, precision="fp32dc", style="member"),
        # a mid-size model in the default precision
        dict(name="P fp64 63x57x41", kind="P", nx=63, ny=57, nz=41, precision="fp64", style="reservoir"),
        # an upper-range ensemble member
        dict(name="P fp32dc 100x90x81", kind="P", nx=100, ny=90, nz=81, precision="fp32dc", style="member"),
        # the headline reservoir's pressure solve
        dict(name="P fp32dc 256x256x128", kind="P", nx=256, ny=256, nz=128, precision="fp32dc",
             style="reservoir"),
        # a large model in the default precision, sloped (buoyancy along x and z), odd height
        dict(name="P fp64 192x160x101", kind="P", nx=192, ny=160, nz=101, precision="fp64", style="sloped"),
        # the reservoir's species solve (imbalance term on)
        dict(name="C fp32dc 256x256x128", kind="C", nx=256, ny=256, nz=128, precision="fp32dc",
             style="reservoir", omega=1.0),
        # a sloped model's species solve with dispersion
        dict(name="C fp32dc disp 129x127x63", kind="C", nx=129, ny=127, nz=63, precision="fp32dc",
             style="sloped", omega=1.0),
        # the reservoir's heat solve
        dict(name="T fp32dc 256x256x128", kind="T", nx=256, ny=256, nz=128, precision="fp32dc",
             style="reservoir", omega=1.0),
        # a small Crank-Nicolson species solve with dispersion, default precision
        dict(name="C fp64 half 48x40x37", kind="C", nx=48, ny=40, nz=37, precision="fp64",
             style="sloped", omega=0.5),
        # what a step does around its solves: fluxes, flow error, CFL limit, Smolarkiewicz
        # velocities, EOS, Picard norm, skip-test sums, mass totals
        dict(name="flow 255x256x127", kind="flow", nx=255, ny=256, nz=127, precision="fp64",
             style="sloped"),
        # a parameter study: five uneven models through six steps, solves batched
        dict(name="ensemble 5 x 6 steps", kind="ensemble", models=5, n_min=32, n_max=72, steps=6,
             precision="fp32dc"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "P", "P", "P", "P", "C", "C", "T", "T", "flow", "ensemble"))
    if kind == "run":
        return dict(kind="run", nx=_log_uniform(rng, 24, 90), ny=1, nz=_log_uniform(rng, 12, 40),
                    steps=rng.randint(3, 8), precision=rng.choice(("fp64", "fp64", "fp32dc")))
    if kind == "ensemble":
        return dict(kind="ensemble", models=rng.randint(3, 5), n_min=rng.randint(24, 36),
                    n_max=rng.randint(50, 72), steps=rng.randint(2, 6), precision="fp32dc")
    # cells log-uniform from a small served cube to the reservoir, axes uneven
    precision = "fp64" if kind == "flow" else rng.choice(("fp32dc", "fp64"))
    top = 8.0e6 if kind in ("C", "T", "flow") else 8.0e6 if precision == "fp32dc" else 3.0e6
    cells = math.exp(rng.uniform(math.log(16 ** 3), math.log(top)))
    a = math.exp(rng.uniform(-0.35, 0.35))
    b = math.exp(rng.uniform(-0.35, 0.35))
    side = (cells / (a * b)) ** (1.0 / 3.0)
    c = dict(kind=kind, nx=max(5, int(round(side * a))), ny=max(5, int(round(side * b))),
             nz=max(5, int(round(side))), precision=precision,
             style=rng.choice(("member", "reservoir", "sloped")))
    if c["nx"] * c["ny"] * c["nz"] > top:
        c["nx"] = int(top / (c["ny"] * c["nz"]))
    if kind in ("C", "T"):
        c["omega"] = rng.choice((1.0, 1.0, 0.5))
    return c


def work(case):
    """Bytes and operations of one pass: each input field read once, each output written
    once; operations from the iterations such a solve takes."""
    k = case["kind"]
    if k == "run":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=8.0 * n * 46, flops=case["steps"] * n * (110 * 30.0 + 4 * 30.0))
    if k == "ensemble":
        n = case["models"] * math.sqrt(case["n_min"] * case["n_max"]) ** 3
        return dict(bytes=8.0 * n * 46, flops=case["steps"] * n * (600 * 15.0 + 8 * 15.0))
    n = case["nx"] * case["ny"] * case["nz"]
    if k == "P":
        # SOR iterations grow with the longest side; 14 operations an update
        return dict(bytes=8.0 * n * 13, flops=14.0 * n * (250 + 4.0 * max(case["nx"], case["ny"], case["nz"])))
    if k == "C":
        return dict(bytes=8.0 * n * 16, flops=n * (120 + 4 * 14.0))
    if k == "T":
        return dict(bytes=8.0 * n * 17, flops=n * (200 + 4 * 14.0))
    # flow: P Pn BP K(3) nue rho phi c_f c_r WP C(2) WC(2) T R cp_f rho_r cp_r WT in; q(3) e rho v(3) out
    return dict(bytes=8.0 * n * (22 + 8), flops=n * 150.0)


# ----------------------------------------------------------------- the inputs
def _spacing(style, n, d0):
    if style == "reservoir":
        return workloads.geometric_spacing(n, d0)
    return numpy.full(n, {"member": 1.0, "sloped": 2.0 * d0}[style])


def _beta(style):
    return 5.0 if style == "sloped" else 0.0


def _inputs(case, seed):
    """The fields of one model some steps into its run, as torch tensors on the GPU."""
    nx, ny, nz, style = case["nx"], case["ny"], case["nz"], case["style"]
    shape = (nx, ny, nz)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 7919 + 17)
    f64 = dict(dtype=torch.float64, device=dev)
    rnd = lambda: torch.rand(shape, generator=g, **f64)      # noqa: E731
    rndn = lambda: torch.randn(shape, generator=g, **f64)    # noqa: E731
    full = lambda v: torch.full(shape, float(v), **f64)      # noqa: E731
    I = dict(shape=shape, beta=_beta(style))
    I["dx"], I["dy"], I["dz"] = (_spacing(style, nx, 1.0), _spacing(style, ny, 1.0),
                                 _spacing(style, nz, 0.5))
    if style == "reservoir":
        # log10 K: a Gaussian random field of correlation length 8 cells
        k2 = sum((torch.fft.fftfreq(n, **f64) ** 2).reshape([-1 if a == q else 1 for a in range(3)])
                 for q, n in enumerate(shape))
        fld = torch.fft.ifftn(torch.fft.fftn(rndn()) * torch.exp(-2.0 * math.pi ** 2 * 64.0 * k2)).real
        fld = fld - fld.mean()
        K = 10.0 ** (-12.0 + 0.5 * fld / fld.std())
        I["Kx"], I["Ky"], I["Kz"] = K, K.clone(), K.clone()
        I["phi"] = 0.05 + 0.2 * rnd()
    else:
        sd = 0.7
        K = 1e-12 * torch.exp(sd * rndn() - 0.5 * sd * sd)
        I["Kx"], I["Ky"] = K, K.clone()
        I["Kz"] = K * (0.1 if style == "sloped" else 1.0)
        I["phi"] = full(0.15 if style == "sloped" else 0.2)
    I["c_f"], I["c_r"], I["nue"] = full(4.5e-10), full(1e-10), full(1e-3)
    I["cp_f"], I["cp_r"], I["l_f"], I["l_r"] = full(4180.0), full(900.0), full(0.6), full(2.5)
    I["rho_r"] = full(2650.0)
    # a plume from the top and a warm bottom
    ax = lambda n, q: torch.linspace(0, 1, n, **f64).reshape([-1 if a == q else 1 for a in range(3)])  # noqa: E731
    x, y, z = ax(nx, 0), ax(ny, 1), ax(nz, 2)
    plume = torch.exp(-((x - 0.5) ** 2 + (y - 0.5) ** 2) / 0.05 - (1 - z) ** 2 / 0.1)
    I["C"] = (plume * (0.8 + 0.2 * rnd())).contiguous()
    I["C1"] = (torch.exp(-((x - 0.3) ** 2 + (z - 0.3) ** 2) / 0.04) * (0.9 + 0.1 * rnd())).contiguous()
    I["T"] = (20.0 + 60.0 * (1 - z) + 2.0 * rnd()).contiguous()
    I["rho_f"] = EOS["rho0"] + EOS["species"] * I["C"] - EOS["tcoef"] * (I["T"] - EOS["T0"])
    # pressure: hydrostatic head and what the last steps left on it
    dz = torch.as_tensor(I["dz"], **f64)
    head = torch.zeros(nz, **f64)
    if nz > 1:
        head[:-1] = torch.flip(torch.cumsum(torch.flip(0.5 * (dz[:-1] + dz[1:]), (0,)), 0), (0,))
    cb = math.cos(math.radians(I["beta"]))
    I["P"] = (1.0e5 + 1000.0 * G * cb * head.reshape(1, 1, -1) + 50.0 * rndn()).contiguous()
    top = torch.zeros(shape, **f64)
    top[:, :, -1] = 1.0
    I["BP"] = top
    I["P"][:, :, -1] = 1.0e5
    I["BC"] = torch.zeros(shape, **f64)
    I["BC"][nx // 3:max(nx // 3 + 1, 2 * nx // 3), ny // 3:max(ny // 3 + 1, 2 * ny // 3), -1] = 1.0
    I["BT"] = top.clone()
    I["BT"][:, :, 0] = 1.0
    # one injecting and one producing cell
    I["WP"], I["WC"], I["WC1"], I["WT"] = full(0), full(0), full(0), full(0)
    for sign in (1.0, -1.0):
        at = tuple(int(torch.randint(0, max(1, n - 1), (1,), generator=g, device=dev)) for n in shape)
        V = float(I["dx"][at[0]] * I["dy"][at[1]] * I["dz"][at[2]])
        I["WP"][at] += sign * 1e-5 * 1000.0 / V
        if sign > 0:
            I["WC"][at] = 1e-5 / V
            I["WT"][at] = 1e-5 * 1000.0 * 4180.0 * 40.0 / V
    I["R"] = full(1.0)
    I["D_fx"], I["D_fy"], I["D_fz"] = full(1e-9), full(1e-9), full(1e-9)
    I["l_l"] = full(10.0 if style == "sloped" else 0.0)
    I["l_t"] = full(1.0 if style == "sloped" else 0.0)
    I["imblflo"] = style == "reservoir"
    I["dt"] = 3600.0 if style == "reservoir" else 600.0
    I["Pn"] = I["P"] - 20.0 * rnd()
    if case["kind"] in ("C", "T"):
        # the fluxes and flow error of a smooth pressure state
        P = 1.0e5 + 1000.0 * G * cb * head.reshape(1, 1, -1) + 2000.0 * torch.sin(3 * x) * torch.cos(2 * y) * (1 - z)
        P = P.contiguous()
        I["qx"], I["qy"], I["qz"] = _darcy(I, P)
        I["e"] = 1e-3 * _flow_error(I, P, P - 1.0, I["qx"], I["qy"], I["qz"], I["dt"])
    return I


def _run_config(case, seed):
    """The config module of a whole run: the slice, its permeability disturbed."""
    cfg = workloads.slice_2d(case["nx"], case["ny"], case["nz"], case["steps"])
    rng = numpy.random.default_rng(seed)
    K = 1e-12 * numpy.exp(0.3 * rng.standard_normal((case["nx"], case["ny"], case["nz"])))
    cfg.Kx[:], cfg.Ky[:], cfg.Kz[:] = K, K, K
    return cfg


def _members(case, seed):
    # the sizes are the case's, the fields and source cells the seed's
    sizes = numpy.random.default_rng(case["models"] + 100 * case["n_min"] + 10000 * case["n_max"])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [workloads.ensemble_member(int(seed) * 64 + q,
                                      shape=tuple(int(round(math.exp(v))) for v in sizes.uniform(lo, hi, 3)))
            for q in range(case["models"])]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "run":
        s.cfg = _run_config(case, seed)
        return s
    if case["kind"] == "ensemble":
        s.cfgs = _members(case, seed)
        return s
    I = s.I = _inputs(case, seed)
    m = s.m = Model(*I["shape"], I["dx"], I["dy"], I["dz"], G, I["beta"], device="cuda",
                    precision=case["precision"])
    m.freeze(I["c_r"], I["l_r"], I["rho_r"], I["cp_r"], I["l_l"], I["l_t"], I["l_l"], I["l_t"],
             I["imblflo"], I["imblflo"])
    I["zero"] = torch.zeros_like(I["P"])
    s.x = torch.empty_like(I["P"])       # the field a solve updates in place
    if case["kind"] == "flow":
        s.q = [torch.zeros_like(I["P"]) for _ in range(3)]
        s.v = [torch.zeros_like(I["P"]) for _ in range(3)]
        s.e = torch.empty_like(I["P"])
        s.rho = torch.empty_like(I["P"])
    return s


# ------------------------------------------------------------------- one pass
def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "run":
        sim = Simulation(s.cfg, device="cuda", precision=case["precision"]).run(max_steps=case["steps"])
        return dict(P=sim.field("P"), C=sim.field("C"), qz=sim.field("qz"), t=float(sim.t_sim),
                    its=[sim.counters["P"], sim.counters["C"]])
    if kind == "ensemble":
        res, _ = Ensemble(s.cfgs, device="cuda", precision=case["precision"]).run(case["steps"])
        return [dict(P=r["P"], C=r["C"], T=r["T"], t=float(r["t_sim"])) for r in res]
    I, m = s.I, s.m
    if kind == "P":
        # a Picard iteration starts again from the step's first pressure
        s.x.copy_(I["P"])
        t, dt, P, Pn, conv, it = m.compute_P(
            s.x, I["c_f"], I["nue"], I["rho_f"], I["phi"], I["Kx"], I["Ky"], I["Kz"], I["zero"],
            I["zero"], I["zero"], I["dt"], I["BP"], I["WP"], SOR=SOR_P, max_it=20000, inc_it=1.25,
            max_dt=864000.0, P_conv=1e-10)
        return dict(P=P, Pn=Pn, t=float(t), dt=float(dt), converged=conv, it=it)
    if kind == "C":
        s.x.copy_(I["C"])
        t, dt, C, conv, it = m.compute_C(
            s.x, I["D_fx"], I["D_fy"], I["D_fz"], I["phi"], I["rho_f"], I["qx"], I["qy"], I["qz"],
            I["dt"], I["BC"], I["WC"], I["R"], I["e"], omega=case["omega"], SOR=1.0, max_it=100,
            max_dt=864000.0, C_conv=1e-10)
        return dict(C=C, t=float(t), dt=float(dt), converged=conv, it=it)
    if kind == "T":
        s.x.copy_(I["T"])
        t, dt, T, conv, it = m.compute_T(
            s.x, I["l_f"], I["cp_f"], I["rho_f"], I["phi"], I["qx"], I["qy"], I["qz"], I["dt"],
            I["BT"], I["WT"], I["e"], omega=case["omega"], SOR=1.0, max_it=100, max_dt=864000.0,
            T_conv=1e-10)
        return dict(T=T, t=float(t), dt=float(dt), converged=conv, it=it)
    q, v = s.q, s.v
    m.compute_q(I["P"], I["BP"], I["Kx"], I["Ky"], I["Kz"], *q, I["nue"], I["rho_f"])
    e = m.flow_error(I["P"], I["Pn"], *q, I["WP"], I["phi"], I["c_f"], I["c_r"], I["rho_f"], I["dt"],
                     out=s.e)
    dt_cfl = m.dt_cfl(*q, I["phi"])
    sums = m.sums([I["C"], I["C1"], I["WC"], I["WC1"]])
    m.smolarkiewicz(I["C"], *q, *v, I["dt"])
    m.eos_linear([I["C"], I["C1"]], I["T"], s.rho, EOS["rho0"], [(0, EOS["species"])], EOS["tcoef"],
                 EOS["T0"])
    l2 = m.l2_norm(s.rho, I["R"])
    mass = m.mass_totals(I["phi"], s.rho, I["R"], [I["C"], I["C1"]], [I["WC"], I["WC1"]], I["T"],
                         I["cp_f"], I["rho_r"], I["cp_r"], I["WP"], I["WT"])
    return dict(q=list(q), e=e, dt_cfl=dt_cfl, sums=sums, v=list(v), rho=s.rho, l2=l2, mass=mass)


SOR_P = 1.9   # the factor of the 3-D workloads


# ------------------------------------------------- the same in plain torch, 64 bits
def _ax(a, q, dev):
    return torch.as_tensor(numpy.asarray(a), dtype=torch.float64, device=dev).reshape(
        [-1 if p == q else 1 for p in range(3)])


def _lo(x, q):
    return x.narrow(q, 0, x.shape[q] - 1)


def _hi(x, q):
    return x.narrow(q, 1, x.shape[q] - 1)


def _harm(a, b, d1, d2):
    ok = (a != 0) & (b != 0)
    one = torch.ones_like(a)
    return torch.where(ok, (d1 + d2) / (d1 / torch.where(ok, a, one) + d2 / torch.where(ok, b, one)),
                       torch.zeros_like(a))


def _face(f, x, d, q):
    """f of the two cells of every face along axis q."""
    return f(_hi(x, q), _lo(x, q), _hi(d, q), _lo(d, q))


def _amean(a, b, d1, d2):
    return (a * d1 + b * d2) / (d1 + d2)


def _grid(I):
    return [_ax(I[n], q, I["phi"].device) for q, n in enumerate(("dx", "dy", "dz"))]


def _grav(I):
    b = float(numpy.radians(I["beta"]))
    return (math.sin(b), 0.0, math.cos(b))


def _darcy(I, P):
    out = []
    for q, (d, K, s) in enumerate(zip(_grid(I), ("Kx", "Ky", "Kz"), _grav(I))):
        v = torch.zeros_like(P)
        if P.shape[q] > 1:
            k = _face(_harm, I[K], d, q) / _face(_harm, I["nue"], d, q)
            dist = 0.5 * (_hi(d, q) + _lo(d, q))
            w = -k * ((_hi(P, q) - _lo(P, q)) / dist + _face(_amean, I["rho_f"], d, q) * G * s)
            shut = (_hi(I["BP"], q) != 0) & (_lo(I["BP"], q) != 0)
            _lo(v, q).copy_(torch.where(shut, torch.zeros_like(w), w))
        out.append(v)
    return out


def _flow_error(I, P, Pn, qx, qy, qz, dt):
    e = torch.zeros_like(P)
    for q, (d, f) in enumerate(zip(_grid(I), (qx, qy, qz))):
        if P.shape[q] > 1:
            r = _lo(f, q) * _face(_harm, I["rho_f"], d, q)
            _lo(e, q).sub_(r / _lo(d, q))
            _hi(e, q).add_(r / _hi(d, q))
    return e + (I["WP"] + ((1 - I["phi"]) * I["c_r"] + I["phi"] * I["c_f"]) * (P - Pn) * I["rho_f"] / dt)


def _checker(shape, dev):
    i, j, k = (torch.arange(n, device=dev).reshape([-1 if p == q else 1 for p in range(3)])
               for q, n in enumerate(shape))
    return (i + j + k) % 2 == 0


def _red_black(X, co, const, den, free, sor, conv, schedule, most, once=False):
    """The red-black iteration until the relative change is below conv; co: the neighbour
    coefficients [(plus, minus) per axis]; returns (X, iterations)."""
    red = _checker(X.shape, X.device)
    w = sor / den
    wc = [torch.where(red & free, w, torch.zeros_like(w)), torch.where(~red & free, w, torch.zeros_like(w))]
    keep = [1.0 - sor * (red & free).double(), 1.0 - sor * (~red & free).double()]
    X = X.clone()
    old = torch.empty_like(X)
    s = torch.empty_like(X)
    it = 0
    while True:
        it += 1
        check = not schedule or it < 50 or it % 10 == 0
        if check:
            old.copy_(X)
        for c in range(2):
            s.copy_(const)
            for q, (p, m) in enumerate(co):
                if X.shape[q] > 1:
                    _lo(s, q).addcmul_(_lo(p, q), _hi(X, q))
                    _hi(s, q).addcmul_(_hi(m, q), _lo(X, q))
            X.mul_(keep[c]).addcmul_(wc[c], s)
        if once:
            return X, it
        if check:
            diff = float(torch.linalg.vector_norm(X - old) / math.sqrt(float((old * old).sum()) + 1e-200))
            if diff < conv:
                return X, it
        if it >= most:
            raise RuntimeError("exact: no convergence in %d iterations" % it)


def _pressure(I, P, dt, sor, max_dt):
    co, const = [], I["WP"].clone()
    M = torch.zeros_like(P)
    for q, (d, K, g) in enumerate(zip(_grid(I), ("Kx", "Ky", "Kz"), _grav(I))):
        p, m = torch.zeros_like(P), torch.zeros_like(P)
        if P.shape[q] > 1:
            f = (_face(_harm, I[K], d, q) / _face(_harm, I["nue"], d, q)) * _face(_harm, I["rho_f"], d, q)
            tot = 0.5 * (_hi(d, q) + _lo(d, q))
            _lo(p, q).copy_(f / (_lo(d, q) * tot))
            _hi(m, q).copy_(f / (_hi(d, q) * tot))
            b = _face(_amean, I["rho_f"], d, q) * G * tot * g
            _lo(const, q).addcmul_(_lo(p, q), b)
            _hi(const, q).addcmul_(_hi(m, q), b, value=-1.0)
        co.append((p, m))
        M = M + p + m
    R = I["rho_f"] * ((1 - I["phi"]) * I["c_r"] + I["phi"] * I["c_f"]) / dt
    const = const + R * P
    X, it = _red_black(P, co, const, R + M, I["BP"] == 0, sor, 1e-10, True, 20000)
    return X, dt, min(dt * 1.25, max_dt) if it < 10000 else dt, it


def _shift(x, q, by):
    """x at the next (by = 1) or previous (by = -1) cell of axis q, 0 outside."""
    v = torch.zeros_like(x)
    if x.shape[q] > 1:
        if by > 0:
            _lo(v, q).copy_(_hi(x, q))
        else:
            _hi(v, q).copy_(_lo(x, q))
    return v


def _inside(shape, q, by, dev):
    v = torch.ones(shape, dtype=torch.float64, device=dev)
    v.select(q, shape[q] - 1 if by > 0 else 0).zero_()
    return v


def _dispersion(I, B, flux, q, by):
    """Dispersion of the face toward the next / previous cell of axis q (tse.py:460-644)."""
    dev, shape = B.device, tuple(B.shape)
    here = _inside(shape, q, by, dev)
    along = flux[q] * here if by > 0 else _shift(flux[q], q, -1)
    open_ = here * (_shift(B, q, by) == 0).double()
    across = torch.zeros_like(B)
    for v in range(3):
        if v == q:
            continue
        four = flux[v] + _shift(flux[v], q, by)
        four = four + _shift(four, v, -1)
        cnt = 0.5 - 0.25 * _inside(shape, v, -1, dev)
        across = across + (four * cnt * open_).abs()
    return I["l_l"] * along.abs() + I["l_t"] * across


def _transport(I, X0, flux, dt, omega, heat, B, W, e, max_dt, imblflo):
    d3 = _grid(I)
    co, M, oldsum = [], torch.zeros_like(X0), torch.zeros_like(X0)
    disp = bool((I["l_l"] != 0).any() or (I["l_t"] != 0).any())
    for q, d in enumerate(d3):
        p, m = torch.zeros_like(X0), torch.zeros_like(X0)
        if X0.shape[q] > 1:
            if heat:
                por = _face(_amean, I["phi"], d, q)
                rc = _face(_harm, I["rho_f"], d, q) * _face(_harm, I["cp_f"], d, q)
                f = (1 - por) * _face(_harm, I["l_r"], d, q) + por * _face(_harm, I["l_f"], d, q)
            else:
                f = _face(_harm, I[("D_fx", "D_fy", "D_fz")[q]], d, q) * _face(_amean, I["phi"], d, q)
                rc = torch.ones_like(f)
            tot = 0.5 * (_hi(d, q) + _lo(d, q))
            qf = _lo(flux[q], q)
            dp = _lo(_dispersion(I, B, flux, q, 1), q) if disp else 0.0
            dm = _hi(_dispersion(I, B, flux, q, -1), q) if disp else 0.0
            dP = (f + dp * rc) / (tot * _lo(d, q))
            dM = (f + dm * rc) / (tot * _hi(d, q))
            lo, hi = qf.clamp(max=0) * rc, qf.clamp(min=0) * rc
            _lo(p, q).copy_(dP - lo / _lo(d, q))
            _hi(m, q).copy_(dM + hi / _hi(d, q))
            _lo(M, q).sub_(dP + hi / _lo(d, q))
            _hi(M, q).sub_(dM - lo / _hi(d, q))
            _lo(oldsum, q).addcmul_(_lo(p, q), _hi(X0, q))
            _hi(oldsum, q).addcmul_(_hi(m, q), _lo(X0, q))
        co.append((omega * p, omega * m))
    if heat:
        num = I["phi"] * I["rho_f"] * I["cp_f"] + (1 - I["phi"]) * I["rho_r"] * I["cp_r"]
        ex = I["cp_f"] * X0 * e if imblflo else 0.0
    else:
        num = I["R"] * I["phi"]
        ex = X0 / I["rho_f"] * e if imblflo else 0.0
    R = num / dt
    const = (1 - omega) * (X0 * M + oldsum) + R * X0 + W - ex
    X, it = _red_black(X0, co, const, R - omega * M, B == 0, 1.0, 1e-10, False, 100, once=omega == 0)
    return X, dt, min(dt * 1.05, max_dt) if it < 50 else dt, it


def _steps(cfg, steps):
    """tse.py's step loop without SIA for a config of these runs, fields on the GPU."""
    dev = torch.device("cuda")
    T_ = lambda a: torch.as_tensor(numpy.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    I = {n: T_(getattr(cfg, n)) for n in ("phi", "Kx", "Ky", "Kz", "c_r", "cp_r", "l_r", "rho_r", "c_f",
                                          "cp_f", "l_f", "nue", "P", "BP", "BC", "BT", "WP", "WT", "T", "R")}
    I["beta"], I["dx"], I["dy"], I["dz"] = cfg.beta, cfg.dx, cfg.dy, cfg.dz
    C, WC = T_(cfg.C[..., 0]), T_(cfg.WC[..., 0])
    I["D_fx"], I["D_fy"], I["D_fz"] = (T_(a[..., 0]) for a in (cfg.D_fx, cfg.D_fy, cfg.D_fz))
    rho = cfg.GPU_EOS["rho"]
    density = lambda C, T: rho["rho0"] + rho["species"][0][1] * C - rho["tcoef"] * (T - rho["T0"])  # noqa: E731
    P, T = I["P"], I["T"]
    I["rho_f"] = density(C, T)
    flux = [torch.zeros_like(P) for _ in range(3)]
    t_sim, dt, dt_max = 0.0, cfg.dt, cfg.dt_max
    for _ in range(steps):
        # the step advances by the dt the solve used; dt_P is its proposal for the next
        P, dt, dt_P, _ = _pressure(I, P, dt, cfg.SOR_P, dt_max)
        I["P"] = P
        flux = _darcy(I, P)
        cfl = 1e10
        if t_sim > 0:
            cfl = _cfl(I, flux)
        dt_max = min(cfl, cfg.dt_max)
        if dt > dt_max:
            dt = dt_max
        lz = torch.zeros_like(P)
        I["l_l"], I["l_t"] = T_(cfg.lf_l), T_(cfg.lf_t)
        C, dt, dt_C, _ = _transport(I, C, flux, dt, 1.0, False, I["BC"], WC, lz, cfg.dt_max, False)
        nxt = min(dt_P, dt_C)
        if cfg.HEATTRANS:
            I["l_l"], I["l_t"] = T_(cfg.lt_l), T_(cfg.lt_t)
            T, dt, dt_T, _ = _transport(I, T, flux, dt, 1.0, True, I["BT"], I["WT"], lz, cfg.dt_max, False)
            nxt = min(nxt, dt_T)
        I["rho_f"] = density(C, T)
        t_sim += dt
        dt = min(nxt, cfg.t - t_sim)
    return P, C, T, flux, t_sim


def _cfl(I, flux):
    v = 0.0
    for f, d in zip(flux, (I["dx"], I["dy"], I["dz"])):
        n = f.numel()
        dd = torch.as_tensor(numpy.asarray(d), dtype=torch.float64, device=f.device)
        v += float(((f.abs() / I["phi"]).reshape(-1) / dd[torch.arange(n, device=f.device) % len(d)]).max())
    return 0.9 / v


def exact(case, seed):
    kind = case["kind"]
    host = lambda t: t.cpu().numpy()  # noqa: E731
    if kind == "run":
        P, C, _, flux, t = _steps(_run_config(case, seed), case["steps"])
        return dict(P=host(P), C=host(C)[..., None], qz=host(flux[2]), t=float(t), its=[None, None])
    if kind == "ensemble":
        out = []
        for cfg in _members(case, seed):
            P, C, T, _, t = _steps(cfg, case["steps"])
            out.append(dict(P=host(P), C=host(C)[..., None], T=host(T), t=float(t)))
        return out
    I = _inputs(case, seed)
    if kind == "P":
        X, t, dt, it = _pressure(I, I["P"], I["dt"], SOR_P, 864000.0)
        return dict(P=X, Pn=I["P"], t=float(t), dt=float(dt), converged=True, it=it)
    if kind in ("C", "T"):
        heat = kind == "T"
        flux = [I["qx"], I["qy"], I["qz"]]
        X, t, dt, it = _transport(I, I[kind], flux, I["dt"], case["omega"], heat, I["BT" if heat else "BC"],
                                  I["WT" if heat else "WC"], I["e"], 864000.0, I["imblflo"])
        return {kind: X, "t": float(t), "dt": float(dt), "converged": True, "it": it}
    q = _darcy(I, I["P"])
    e = _flow_error(I, I["P"], I["Pn"], *q, I["dt"])
    sums = [float(I[n].sum()) for n in ("C", "C1", "WC", "WC1")]
    v = []
    c = I["C"]
    for a, (d, f) in enumerate(zip(_grid(I), q)):
        w = torch.zeros_like(c)
        dist = 0.5 * (_hi(d, a) + _lo(d, a))
        fl, c0, c1 = _lo(f, a), _lo(c, a), _hi(c, a)
        y = 1.08 * (fl.abs() * dist - I["dt"] * (fl * fl)) * (c1 - c0) / ((c0 + c1 + 1e-15) * dist)
        _lo(w, a).copy_(torch.where(c0 > 0, y, torch.zeros_like(y)))
        v.append(w)
    rho = EOS["rho0"] + EOS["species"] * I["C"] - EOS["tcoef"] * (I["T"] - EOS["T0"])
    l2 = float(torch.linalg.vector_norm(rho - I["R"]) / torch.linalg.vector_norm(I["R"]))
    dx, dy, dz = _grid(I)
    V = dx * dy * dz
    tot = lambda a: float((a * V).sum())  # noqa: E731
    mass = [tot(I["phi"] * rho), tot(I["R"] * I["phi"] * I["C"]), tot(I["R"] * I["phi"] * I["C1"]),
            tot((I["phi"] * rho * I["cp_f"] + (1 - I["phi"]) * I["rho_r"] * I["cp_r"]) * I["T"]),
            tot(I["WP"]), tot(I["WC"]), tot(I["WC1"]), tot(I["WT"])]
    return dict(q=q, e=e, dt_cfl=_cfl(I, q), sums=sums, v=v, rho=rho, l2=l2, mass=numpy.array(mass))
