"""The work this package is timed on: what a user's program has it do, each case through the entry
points such a program calls, over the sizes of the analytic basins and of generic ones.

A case is a dict: `kind` (one of KINDS), the basin (`Lm` x `Mm` interior points, `N` levels) or the
number of rows, the precision ("fp32", "fp64") and the options of its kind.  Initial states are
smooth random flows (sums of plane waves) over the shelf-and-seamount depth; they are made in 64
bits on the device and rounded to the case's precision, so `exact` starts from the same values.
"""
import ctypes
import math
import os

import numpy as np
import torch

from sailfish_b200 import closure, configs, ensemble, host
from sailfish_b200._lib import check, lib
from sailfish_b200.model import Grid, Model, stream_handle

F64 = torch.float64
DTYPE = {"fp32": torch.float32, "fp64": F64}
WEIGHTS = os.path.join(os.path.dirname(closure.__file__), "weights")
G, RHO0, ALPHA, DRAG = 10.0, 1025.0, 1.7e-4, 3e-3


def listed():
    return [
        # the smallest calls: a 2D run (main2d) of the flat 130 x 66 basin, 16 steps of 15 s
        dict(name="main2d_130x66_fp64", kind="main2d", Lm=128, Mm=64, dx=5e3, steps=16, dt=15.0,
             prec="fp64", flat=True),
        # the barotropic loop of one baroclinic step: the 512 x 256 basin in FP32 ...
        dict(name="loop_514x258_fp32", kind="loop", Lm=512, Mm=256, dx=2e3, dt=240.0, nd=37,
             prec="fp32"),
        # ... and an odd-sized one in FP64, the plain form that errors are stated against
        dict(name="loop_771x387_fp64", kind="loop", Lm=769, Mm=385, dx=2e3, dt=240.0, nd=37,
             prec="fp64"),
        # the explicit 3D part of a step: fluxes, vertical velocity, right-hand side, stresses
        dict(name="rhs_1026x514x50_fp32", kind="rhs", Lm=1024, Mm=512, N=50, dx=2e3, prec="fp32"),
        # the implicit 3D part: column solves, barotropic restart, walls; an odd row length
        dict(name="column_1003x501x50_fp32", kind="column", Lm=1001, Mm=499, N=50, dx=2e3,
             dt=120.0, prec="fp32"),
        # vertical mixing by plain GLS on every column: k-epsilon in FP32 ...
        dict(name="gls_1026x514x50_fp32", kind="gls", Lm=1024, Mm=512, N=50, dx=2e3, dt=120.0,
             model="k-epsilon", prec="fp32"),
        # ... and the generic k-psi model in FP64 on the 512 x 256 x 32 basin
        dict(name="gls_514x258x32_fp64", kind="gls", Lm=512, Mm=256, N=32, dx=2e3, dt=240.0,
             model="gen", prec="fp64"),
        # vertical mixing by the learned closure (the shipped network)
        dict(name="closure_1026x514x50_fp32", kind="closure", Lm=1024, Mm=512, N=50, dx=2e3,
             dt=120.0, net="closure_basin4.npz", prec="fp32"),
        # one optimizer step of the closure's training (batch of the shipped networks' training)
        dict(name="train_8192", kind="train", rows=8192, N=50, act="relu"),
        # whole steps: the benchmark's default (the reference's semantics from rest, 2050 x 1026 x 50,
        # learned closure) ...
        dict(name="ref_step_2050x1026x50_fp32", kind="step", Lm=2048, Mm=1024, N=50, dx=1e3,
             dt=120.0, nd=40, semantics="reference", net="closure_basin4.npz", prec="fp32"),
        # ... the same basin in the ROMS form, a flow under wind and drag ...
        dict(name="roms_step_2050x1026x50_fp32", kind="step", Lm=2048, Mm=1024, N=50, dx=1e3,
             dt=120.0, nd=40, semantics="roms", net="closure_basin4.npz", prec="fp32"),
        # ... and an ensemble of uneven basins in the ROMS form
        dict(name="ensemble_64_fp32", kind="ensemble", members=64, sizes=0, dt=240.0, nd=37,
             prec="fp32"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(KINDS)
    prec = rng.choice(("fp32", "fp32", "fp64"))
    if kind == "main2d":
        return dict(kind=kind, Lm=size(24, 700), Mm=size(16, 400), dx=5e3, steps=size(4, 64),
                    dt=15.0, prec=prec, flat=True)
    if kind == "loop":
        return dict(kind=kind, Lm=size(48, 2048), Mm=size(32, 1024), dx=2e3, dt=240.0,
                    nd=rng.choice((37, 40, 50)), prec=prec)
    if kind == "train":
        return dict(kind=kind, rows=16 * size(32, 2048), N=rng.choice((32, 50)),
                    act=rng.choice(("relu", "gelu")))
    if kind == "ensemble":
        return dict(kind=kind, members=size(4, 64), sizes=rng.randrange(1 << 16), dt=240.0,
                    nd=37, prec=rng.choice(("fp32", "fp64")))
    N = rng.choice((16, 20, 30, 32, 40, 50))
    c = dict(kind=kind, Lm=size(64, 1024), Mm=size(48, 512), N=N, dx=2e3, prec=prec)
    if kind in ("column", "gls"):
        c["dt"] = rng.choice((60.0, 120.0, 240.0))
    if kind == "gls":
        c["model"] = rng.choice(("k-epsilon", "gen"))
    if kind in ("closure", "step"):
        c["N"], c["dt"] = rng.choice(((32, 240.0), (50, 120.0)))
        c["net"] = rng.choice({32: ("closure_basin1.npz", "closure_basin1_relu.npz"),
                               50: ("closure_basin4.npz", "closure_basin4_gelu.npz")}[c["N"]])
        c["prec"] = "fp32"
    if kind == "step":
        c["nd"] = 40
        c["semantics"] = rng.choice(("roms", "roms", "reference"))
    return c


# -- inputs ---------------------------------------------------------------------------------
class Basin:
    """Metrics, depth and vertical coordinate of a case on the device, in 64 bits: the package's
    analytic basin (tanh shelf across y, Gaussian seamounts, beta plane, Vtransform 2, Vstretching 4,
    theta_s 5, theta_b 0.4, hc 100 m)."""

    def __init__(self, c):
        self.I, self.J, self.N = c["Lm"] + 2, c["Mm"] + 2, c.get("N", 5)
        dx = c["dx"]
        j, i = torch.meshgrid(torch.arange(self.J, device="cuda", dtype=F64),
                              torch.arange(self.I, device="cuda", dtype=F64), indexing="ij")
        x, y, Lx, Ly = (i - 0.5) * dx, (j - 0.5) * dx, c["Lm"] * dx, c["Mm"] * dx
        h = 50.0 + 3950.0 * 0.5 * (1.0 + torch.tanh((y / Ly - 0.25) / 0.1))
        for f in (1 / 3, 2 / 3):
            h = h - 2000.0 * torch.exp(-((x - f * Lx) ** 2 + (y - 0.6 * Ly) ** 2) / 20e3 ** 2)
        self.h = torch.full_like(x, 4000.0) if c.get("flat") else h.clamp(min=50.0)
        self.f = 1e-4 + 2e-11 * (y - 0.5 * Ly)
        self.x, self.y, self.Ly, self.dx = x, y, Ly, dx
        self.xs, self.ys = x / Lx, y / Ly

    def package(self, c):
        """The package's grid and boundary on this basin."""
        g = Grid.analytic(self.I - 2, self.J - 2, self.N, self.h.cpu().numpy(), self.dx, self.dx,
                          self.f.cpu().numpy())
        return g, host.Boundary(g.L, g.M, configs.CLOSED)

    def depths(self, zeta):
        """z_w (N+1), z_r (N), Hz (N) of the free surface zeta."""
        def z(s):
            C = (1 - torch.cosh(5.0 * s)) / (math.cosh(5.0) - 1)
            C = (torch.exp(0.4 * C) - 1) / (1 - math.exp(-0.4))
            s, C = s[:, None, None], C[:, None, None]
            return zeta + (zeta + self.h) * (100.0 * s + self.h * C) / (100.0 + self.h)
        k = torch.arange(self.N + 1, device="cuda", dtype=F64)
        zw = z((k - self.N) / self.N)
        return zw, z((k[1:] - 0.5 - self.N) / self.N), zw[1:] - zw[:-1]


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def waves(b, gen, amp, n=12):
    """A smooth random field: n plane waves of 1 to 8 periods a basin, RMS about amp."""
    r = torch.rand(n, 4, generator=gen, device="cuda", dtype=F64).cpu()
    out = torch.zeros_like(b.h)
    for kx, ky, ph, a in r.tolist():
        out += (0.5 + a) * torch.cos(2 * math.pi * ((8 * kx - 4) * b.xs + (8 * ky - 4) * b.ys + ph))
    return out * (amp * math.sqrt(2.0 / n))


def faces(b, a, dim):
    """`a` on the interior U (dim -1) or V (dim -2) faces, 0 on walls and the ring."""
    out = torch.zeros_like(a)
    s = (slice(1, -1), slice(2, -1)) if dim == -1 else (slice(2, -1), slice(1, -1))
    out[(...,) + s] = a[(...,) + s]
    return out


def state2d(b, gen):
    """zeta (ring = nearest interior node), ubar, vbar and the zonal wind stress."""
    z = waves(b, gen, 0.2)
    for d in (0, 1):
        z = z.index_select(d, torch.arange(z.shape[d], device="cuda").clamp(1, z.shape[d] - 2))
    u, v = faces(b, waves(b, gen, 0.05), -1), faces(b, waves(b, gen, 0.05), -2)
    tau = float(torch.rand(1, generator=gen, device="cuda", dtype=F64)) * 0.1 + 0.05
    return dict(zeta=z, ubar=u, vbar=v, sustr=tau / RHO0 * torch.cos(math.pi * b.ys),
                svstr=torch.zeros_like(z))


def flow3d(b, gen, zeta, real):
    """Depths and a surface-intensified velocity, rounded to `real` (u, v have N+1 levels)."""
    zw, zr, Hz = (a.to(real) for a in b.depths(zeta))
    out = dict(z_w=zw, z_r=zr, Hz=Hz)
    for n, dim in (("u", -1), ("v", -2)):
        a = torch.zeros((b.N + 1, b.J, b.I), device="cuda", dtype=real)
        top, deep = faces(b, waves(b, gen, 0.2), dim), faces(b, waves(b, gen, 0.05), dim)
        for k in range(b.N):
            a[k] = (top * torch.exp(zr[k].double() / 60.0) + deep * torch.exp(zr[k].double() / 1500.0)).to(real)
        out[n] = a
    return out


def inputs(c, seed):
    """The arrays of a case that prepare and exact share."""
    b, gen, real = Basin(c), generator(seed), DTYPE[c["prec"]]
    d = state2d(b, gen)
    kind = c["kind"]
    if kind in ("main2d", "loop"):
        return b, {k: a.to(real) for k, a in d.items()}
    d.update(flow3d(b, gen, d["zeta"], real))
    if kind == "column":
        area = b.dx * b.dx
        for n, dim in (("ru", -1), ("rv", -2)):
            base = faces(b, waves(b, gen, 0.05), dim)
            for s in range(3):   # right-hand sides of three steps: Hz f u / (pm pn), drifting slowly
                a = torch.zeros((b.N + 1, b.J, b.I), device="cuda", dtype=real)
                w = base + faces(b, waves(b, gen, 0.005), dim)
                for k in range(b.N):
                    a[k] = (1e-4 * area * w * d["Hz"][k]).to(real)
                d["%s%d" % (n, s)] = a
        W = torch.zeros((b.N + 1, b.J, b.I), device="cuda", dtype=real)
        AKv = torch.zeros_like(W)
        w, lg = waves(b, gen, 1e-5) * area, waves(b, gen, 0.7)
        for k in range(b.N + 1):
            s = k / b.N
            W[k] = (w * math.sin(math.pi * s)).to(real)
            AKv[k] = (10.0 ** (lg - 4.0 + 2.0 * s * s)).to(real)
        D = b.h + d["zeta"]
        d.update(W=W, AKv=AKv,
                 DU=d["ubar"] * 0.5 * (D + D.roll(1, -1)) * b.dx, DV=d["vbar"] * 0.5 * (D + D.roll(1, -2)) * b.dx)
    if kind in ("gls", "closure", "step"):
        r = torch.rand(2, generator=gen, device="cuda", dtype=F64)
        zs = 300.0 + 400.0 * float(r[0])
        d["zscale"] = zs
        bvf = torch.empty((b.N + 1, b.J, b.I), device="cuda", dtype=real)
        for k in range(b.N + 1):
            bvf[k] = (G * ALPHA * 20.0 / zs * torch.exp(d["z_w"][k].double() / zs)).to(real)
        d["bvf"] = bvf
        d["sustr"] = (0.05 + 0.1 * float(r[1])) / RHO0 * torch.cos(math.pi * b.ys)
    if kind == "gls":   # a turbulent surface layer over a quiet interior, columns differing
        P = closure.GLS_PRESETS[c["model"]]
        lg = waves(b, gen, 0.3)
        new = {n: torch.empty((b.N + 1, b.J, b.I), device="cuda", dtype=real)
               for n in ("tke", "gls", "AKv", "Akt", "Akk", "Akp", "Lscale")}
        for k in range(b.N + 1):
            zk = d["z_w"][k].double()
            t = 1e-3 * 10.0 ** lg * torch.exp(zk / 25.0) + 1e-5
            le = 0.4 * ((-zk).clamp(min=0.05) / (1 + (-zk).clamp(min=0.05) / 10.0))
            e = 0.3 * le * t.sqrt()
            vals = dict(tke=t, gls=P["cmu0"] ** P["p"] * t ** P["m"] * le ** P["n"], AKv=e + 1e-5,
                        Akt=0.8 * e + 1e-6, Akk=e / P["sigk"] + 5e-6, Akp=e / P["sigp"] + 5e-6, Lscale=le)
            for n, a in vals.items():
                new[n][k] = a.to(real)
        d.update(new)
    for n in ("zeta", "ubar", "vbar", "sustr", "svstr"):
        d[n] = d[n].to(real)
    return b, d


def training_rows(c, seed):
    gen = generator(seed)
    nf = 2 * (c["N"] - 1) + 3
    X = torch.zeros((c["rows"], 128), device="cuda")
    X[:, :nf] = torch.randn(c["rows"], nf, generator=gen, device="cuda")
    A = torch.randn(nf, 128, generator=gen, device="cuda") / math.sqrt(nf)
    return X, torch.tanh(X[:, :nf] @ A) - 4.0


# -- what a user's program holds --------------------------------------------------------------
def _fill(m, d, names):
    for n in names:
        getattr(m, n).copy_(d[n].reshape(getattr(m, n).shape))


def _mixing(m, c, d, mode):
    net = closure.Network.load(os.path.join(WEIGHTS, c["net"])) if mode == "mlp" else None
    mix = closure.Closure(m, mode, net, gls_model=c.get("model"))
    for n in ("bvf", "sustr", "svstr"):
        getattr(mix.cols, n).copy_(d[n].reshape(getattr(mix.cols, n).shape))
    return mix


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "train":
        X, T = training_rows(c, seed)
        n, L, W = c["rows"], closure.LAYERS, closure.WIDTH
        z = lambda *s: torch.zeros(*s, device="cuda")
        s = dict(c=c, net=closure.Network(c["N"], seed=seed, act=c["act"]), X=X, T=T,
                 acts=z(L - 1, n, W), pre=z(L, n, W), Y=z(n, W), dY=z(n, W), work=z(2, n, W),
                 dW=[z(W, W) for _ in range(L)], db=[z(W) for _ in range(L)], loss=z(1))
        return s
    if kind == "ensemble":
        members = ensemble.ensemble_members(seed=c["sizes"], n=c["members"])
        r = np.random.default_rng(seed)
        new = []
        for g, bd, _ in members:   # this seed's surface bumps on the case's basins
            x0, y0, a = r.uniform(0, g.x.max()), r.uniform(0, g.y.max()), r.uniform(0.05, 0.1)
            new.append((g, bd, a * np.exp(-((g.x - x0) ** 2 + (g.y - y0) ** 2) / 50e3 ** 2)))
        e = ensemble.make(new, c["prec"], c["dt"], c["nd"], semantics="roms")
        ensemble.roms_forcing(e, tau0=0.05)
        e.AKv.fill_(1e-2)
        e.start()
        return dict(c=c, m=e)
    b, d = inputs(c, seed)
    g, bd = b.package(c)
    if kind == "main2d":
        m = Model(g, bd, c["dt"], 1, precision=c["prec"], semantics="roms")
    else:
        m = Model(g, bd, c.get("dt", 120.0), c.get("nd", 1), precision=c["prec"],
                  semantics=c.get("semantics", "roms"))
    s = dict(c=c, m=m)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    at_rest = kind == "step" and c["semantics"] == "reference"
    if m.semantics == "roms":
        m.rdrag2 = DRAG
        _fill(m, d, ("sustr", "svstr"))
    if kind in ("main2d", "loop", "step") and not at_rest:
        for k in range(3):
            for n in ("zeta", "ubar", "vbar"):
                getattr(m, n)[k].copy_(d[n])
    if kind in ("rhs", "column", "gls", "closure"):
        _fill(m, d, ("u", "v", "z_w", "z_r", "Hz"))
    if kind == "column":
        _fill(m, d, ("W", "AKv"))
        m.DU_avg1.copy_(d["DU"].reshape(-1))
        m.DV_avg1.copy_(d["DV"].reshape(-1))
        s["rs"] = [d["%s%d" % (n, k)] for n in ("ru", "rv") for k in range(3)]
    if kind == "gls":
        s["mix"] = _mixing(m, c, d, "gls")
        m.AKv.copy_(d["AKv"])
        for n in ("tke", "gls", "Akt", "Akk", "Akp", "Lscale"):
            getattr(s["mix"].cols, n).copy_(d[n])
    if kind == "closure":
        s["mix"] = _mixing(m, c, d, "mlp")
    if kind == "step":
        m.mixing = _mixing(m, c, d, "mlp")
        if not at_rest:
            _fill(m, d, ("u", "v"))
            m.Zt_avg1.copy_(d["zeta"].reshape(-1))
        m.start()
    s["p"] = p
    return s


# -- one pass ---------------------------------------------------------------------------------
def run(state):
    return RUN[state["c"]["kind"]](state)


def run_main2d(s):
    m = s["m"]
    m.step2d(s["c"]["steps"])
    return levels(m)


def levels(m):
    """zeta, ubar, vbar at the newest time level and at the one before (ROMS form)."""
    return {n + t: getattr(m, n)[m.slots[k]] for n in ("zeta", "ubar", "vbar") for t, k in (("", 1), ("_old", 0))}


def run_loop(s):
    m, p = s["m"], s["p"]
    st = m.state2d()
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    check(lib.sf_roms_barotropic_loop(
        m.ctx.ptr, ctypes.byref(st), p(m.DU_avg2), p(m.DV_avg2), p(m.sustr), p(m.svstr), m.rdrag2,
        m.nfast, ptr(m.W1), ptr(m.W2), m.dtfast, stream_handle()), "sf_roms_barotropic_loop")
    m._sync_slots(st)
    return dict(levels(m), **{n: getattr(m, n) for n in ("Zt_avg1", "DU_avg1", "DV_avg1", "DU_avg2", "DV_avg2")})


def run_rhs(s):
    m, p, st = s["m"], s["p"], stream_handle()
    check(lib.sf_maxflux_omega(m.ctx.ptr, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.W),
                               p(m.z_w), None, None, None, st), "sf_maxflux_omega")
    check(lib.sf_roms_rhs3d(m.ctx.ptr, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.ru),
                            p(m.rv), st), "sf_roms_rhs3d")
    check(lib.sf_roms_stress3d(m.ctx.ptr, p(m.u), p(m.v), p(m.ru), p(m.rv), p(m.sustr), p(m.svstr),
                               m.rdrag2, st), "sf_roms_stress3d")
    return {n: getattr(m, n) for n in ("Huon", "Hvom", "W", "ru", "rv")}


def run_column(s):
    m, p, st = s["m"], s["p"], stream_handle()
    ub, vb, us, vs = m.ubar[1], m.vbar[1], m.ubar[2], m.vbar[2]
    check(lib.sf_roms_step3d_uv(
        m.ctx.ptr, p(m.u), p(m.v), *[p(t) for t in s["rs"]], p(ub), p(vb), p(us), p(vs), p(m.Hz),
        p(m.AKv), p(m.z_r), p(m.W), p(m.DU_avg1), p(m.DV_avg1), 5, 0, m.lam, m.dt, st),
        "sf_roms_step3d_uv")
    check(lib.sf_lateral_uv_bc(m.ctx.ptr, 0.0, p(m.u), p(m.v), st), "sf_lateral_uv_bc")
    check(lib.sf_roms_closed_walls(m.ctx.ptr, p(m.u), p(m.v), st), "sf_roms_closed_walls")
    return dict(u=m.u, v=m.v, ubar=ub, vbar=vb)


def run_gls(s):
    s["mix"]()
    q = s["mix"].cols
    return dict({n: getattr(q, n) for n in ("tke", "gls", "Akt", "Akk", "Akp", "Lscale")}, AKv=s["m"].AKv)


def run_closure(s):
    s["mix"]()
    return dict(AKv=s["m"].AKv, Akt=s["mix"].cols.Akt)


def run_train(s):
    """One iteration of closure.Network.train on a batch in hand."""
    net, n, st = s["net"], s["c"]["rows"], stream_handle()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    P = net.params()
    ptrs = lambda ts: (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
    s["loss"].zero_()
    check(lib.sf_mlp_forward(ctypes.byref(P), n, p(s["X"]), p(s["Y"]), p(s["acts"]), p(s["pre"]),
                             p(net.err), st), "sf_mlp_forward")
    check(lib.sf_mlp_mse(n, closure.nout(net.N), p(s["Y"]), p(s["T"]), p(s["dY"]), p(s["loss"]), st),
          "sf_mlp_mse")
    check(lib.sf_mlp_backward(ctypes.byref(P), n, p(s["X"]), p(s["acts"]), p(s["pre"]), p(s["dY"]),
                              ptrs(s["dW"]), ptrs(s["db"]), p(s["work"]), p(net.err), st),
          "sf_mlp_backward")
    net.step_count += 1
    f = ctypes.c_float
    for l in range(closure.LAYERS):
        for k, w, dw, mm, v, wb in ((128 * 128, net.W, s["dW"], net.mW, net.vW, p(net.Wb[l])),
                                    (128, net.b, s["db"], net.mb, net.vb, None)):
            check(lib.sf_mlp_adam(k, p(w[l]), p(dw[l]), p(mm[l]), p(v[l]), wb, f(2e-3), f(0.9),
                                  f(0.999), net.step_count, f(1e-8), st), "sf_mlp_adam")
    return dict(loss=s["loss"], Y=s["Y"], dW=s["dW"], db=s["db"], W=net.W, b=net.b)


def run_step(s):
    m = s["m"]
    m.step(1)
    k = 1 if m.semantics == "roms" else 2
    out = {n: getattr(m, n)[m.slots[k]] for n in ("zeta", "ubar", "vbar")}
    out.update({n: getattr(m, n) for n in ("Zt_avg1", "DU_avg1", "DV_avg1", "u", "v", "W")})
    if m.mixing is not None:
        out["AKv"] = m.AKv
    return out


RUN = dict(main2d=run_main2d, loop=run_loop, rhs=run_rhs, column=run_column, gls=run_gls,
           closure=run_closure, train=run_train, step=run_step, ensemble=run_step)
KINDS = tuple(RUN)


# -- what a pass cannot do without --------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "train":   # X, T in; hidden states kept for the backward pass are not counted
        n = c["rows"]
        return dict(bytes=4.0 * n * 128 * 3 + 5 * 128 * 129 * 4 * 7, flops=2.0 * n * 128 * 128 * 14)
    e = 4 if c["prec"] == "fp32" else 8

    def loop(s2, nsub, ee):   # per substep: two levels in, one out, metrics, tendencies; averages in 64 bits
        return s2 * nsub * (23.0 * ee + 80.0), s2 * nsub * 250.0

    def columns(n3, ee):      # fluxes + rhs (u, v, Hz, z_w -> Huon, Hvom, W, ru, rv), solve, depths
        return n3 * ee * (9.0 + 14.0 + 3.0), n3 * 180.0

    if kind == "ensemble":
        B = F = 0.0
        nf = host.set_weights(c["nd"])[0]
        rng = np.random.default_rng(c["sizes"])
        for _ in range(c["members"]):   # the sizes that ensemble.ensemble_members draws
            Lm, Mm = int(rng.integers(64, 513)), int(rng.integers(32, 257))
            N = int(rng.choice((16, 32)))
            rng.uniform(size=3)
            s2 = (Lm + 2) * (Mm + 2)
            for b, f in (loop(s2, nf, e), columns(s2 * N, e)):
                B, F = B + b, F + f
        return dict(bytes=B, flops=F)
    s2 = (c["Lm"] + 2) * (c["Mm"] + 2)
    n3 = s2 * c.get("N", 1)
    if kind == "main2d":
        return dict(bytes=s2 * c["steps"] * 23.0 * e, flops=s2 * c["steps"] * 230.0)
    if kind == "loop":
        b, f = loop(s2, host.set_weights(c["nd"])[0], e)
        return dict(bytes=b, flops=f)
    if kind == "rhs":
        return dict(bytes=n3 * e * 9.0, flops=n3 * 80.0)
    if kind == "column":
        return dict(bytes=n3 * e * 14.0, flops=n3 * 100.0)
    if kind == "gls":
        return dict(bytes=n3 * e * 19.0, flops=n3 * 300.0)
    mlp = (n3 * e * 6.0, s2 * 2.0 * 5 * 128 * 128)
    if kind == "closure":
        return dict(bytes=mlp[0], flops=mlp[1])
    nf = host.set_weights(c["nd"])[0]
    b, f = loop(s2, nf, e) if c["semantics"] == "roms" else (s2 * (nf + 1) * 132.0, s2 * nf * 150.0)
    cb, cf = columns(n3, e)
    return dict(bytes=b + cb + mlp[0], flops=f + cf + mlp[1])


# -- the same in 64 bits --------------------------------------------------------------------------
def exact(case, seed):
    f = EXACT.get(case["kind"])
    return f(case, seed) if f else None


def _avg(a, dim):
    """Mean of a point and its west (dim -1) or south (dim -2) neighbour."""
    return 0.5 * (a + a.roll(1, dim))


class Shallow:
    """One phase after another of the free-surface and depth-mean momentum scheme (LF-AM3)."""

    def __init__(self, c, b, d):
        real = DTYPE[c["prec"]]
        self.h = b.h.to(real).double()
        self.fomn = (b.f * b.dx * b.dx).to(real).double()
        self.dx, self.b = b.dx, b
        self.tau = d["sustr"].double(), d["svstr"].double()
        self.z, self.u, self.v = ([d[n].double()] * 2 for n in ("zeta", "ubar", "vbar"))
        self.r = [None, None]

    def flux(self, z, u, v):
        D = z + self.h
        return u * _avg(D, -1) * self.dx, v * _avg(D, -2) * self.dx

    def phase(self, z, u, v, zs, us, vs, dtz, dtm, zwrk, fz, fm):
        """New level from the old one (zs, us, vs) and the fluxes and forces at (z, u, v)."""
        DU, DV = self.flux(z, u, v)
        rz = (DU - DU.roll(-1, -1)) + (DV - DV.roll(-1, -2))
        zn = zs + dtz / self.dx ** 2 * fz(rz)
        for dim in (0, 1):
            k = torch.arange(zn.shape[dim], device="cuda").clamp(1, zn.shape[dim] - 2)
            zn = zn.index_select(dim, k)
        w, h = zwrk(zn), self.h
        out, rr = [], []
        for dim, q, o, qs, sgn, tau in ((-1, u, v, us, 1.0, self.tau[0]), (-2, v, u, vs, -1.0, self.tau[1])):
            od = -3 - dim
            pg = 0.5 * G * self.dx * ((h.roll(1, dim) + h) * (w.roll(1, dim) - w) + (w.roll(1, dim) ** 2 - w ** 2))
            cor = sgn * _avg(0.5 * (z + h) * self.fomn * (o + o.roll(-1, od)), dim)
            o4 = 0.5 * _avg(o + o.roll(-1, od), dim)
            r = pg + cor + (tau - DRAG * q * torch.sqrt(q * q + o4 * o4)) * self.dx ** 2
            r = faces(self.b, r, dim)
            new = (qs * 2 * _avg(zs + h, dim) + 4 / self.dx ** 2 * dtm * fm(r, dim)) / (2 * _avg(zn + h, dim))
            out.append(faces(self.b, new, dim))
            rr.append(r)
        return zn, out[0], out[1], (rz, rr[0], rr[1])

    def step(self, dt, first, acc=lambda *a: None):
        z, u, v = self.z, self.u, self.v
        same = lambda r, *a: r
        o = 1 if first else 0
        acc(0, z[1], *self.flux(z[1], u[1], v[1]))
        if first:
            zw = lambda zn: 0.5 * (z[1] + zn)
        else:
            zw = lambda zn: 0.68 * z[1] + 0.16 * (z[0] + zn)
        zp, up, vp, rn = self.phase(z[1], u[1], v[1], z[o], u[o], v[o], dt if first else 2 * dt,
                                    0.5 * dt if first else dt, zw, same, same)
        acc(1, zp, *self.flux(zp, up, vp))
        rb = self.r[1]
        if first:
            zc, fz, fm = (lambda zn: 0.5 * (z[1] + zn)), same, same
        else:
            am3 = lambda r, k: 5 / 12 * r + 8 / 12 * rn[k] - 1 / 12 * rb[k]
            zc = lambda zn: 0.6 * zn + 0.4 * zp
            fz, fm = (lambda r: am3(r, 0)), (lambda r, dim: am3(r, 1 if dim == -1 else 2))
        zn, un, vn, _ = self.phase(zp, up, vp, z[1], u[1], v[1], dt, 0.5 * dt, zc, fz, fm)
        self.z, self.u, self.v = [z[1], zn], [u[1], un], [v[1], vn]
        self.r = [rb, rn]

    def levels(self):
        return {n + t: a[k] for n, a in (("zeta", self.z), ("ubar", self.u), ("vbar", self.v))
                for t, k in (("", 1), ("_old", 0))}


def exact_main2d(c, seed):
    b, d = inputs(c, seed)
    s = Shallow(c, b, d)
    for k in range(c["steps"]):
        s.step(c["dt"], k == 0)
    return s.levels()


def exact_loop(c, seed):
    b, d = inputs(c, seed)
    s = Shallow(c, b, d)
    nf, w1, _ = host.set_weights(c["nd"])   # host tables, not the path under test
    W1 = np.concatenate([[0.0], w1])
    W2 = np.array([0.0] + [W1[i:nf + 1].sum() for i in range(1, nf + 1)] + [0.0, 0.0])
    W2 /= W2.sum()
    A = {n: torch.zeros_like(b.h) for n in ("Zt_avg1", "DU_avg1", "DV_avg1", "DU_avg2", "DV_avg2")}

    def add(c1, c2, z, DU, DV):
        A["Zt_avg1"] += c1 * z
        A["DU_avg1"] += c1 * DU
        A["DV_avg1"] += c1 * DV
        A["DU_avg2"] += c2 * DU
        A["DV_avg2"] += c2 * DV

    for m in range(1, nf + 2):
        def acc(ph, z, DU, DV):
            if ph:
                add(0.0, W2[1] if m == 1 else 5 / 12 * W2[m], z, DU, DV)
            elif m == 1:
                add(0.0, -1 / 12 * W2[2], z, DU, DV)
            else:
                add(W1[m - 1], 8 / 12 * W2[m] - 1 / 12 * W2[m + 1], z, DU, DV)
        if m <= nf:
            s.step(c["dt"] / c["nd"], m == 1, acc)
        else:
            acc(0, s.z[1], *s.flux(s.z[1], s.u[1], s.v[1]))
    return dict(s.levels(), **{n: a.reshape(-1) for n, a in A.items()})


def exact_rhs(c, seed):
    b, d = inputs(c, seed)
    N, dx = b.N, b.dx
    fomn = (b.f * dx * dx).to(DTYPE[c["prec"]]).double()
    out = {n: torch.zeros((N + 1, b.J, b.I), device="cuda", dtype=F64) for n in ("Huon", "Hvom", "W", "ru", "rv")}
    sus, svs = d["sustr"].double(), d["svstr"].double()
    run_w = torch.zeros_like(b.h)
    for k in range(N):
        u, v, H = d["u"][k].double(), d["v"][k].double(), d["Hz"][k].double()
        hu, hv = _avg(H, -1) * u * dx, _avg(H, -2) * v * dx
        out["Huon"][k], out["Hvom"][k] = hu, hv
        if k > 0:
            run_w = run_w - ((hu.roll(-1, -1) - hu) + (hv.roll(-1, -2) - hv))
            out["W"][k] = run_w
        for n, q, o, hq, ho, dim, sgn, tau in (("ru", u, v, hu, hv, -1, 1, sus), ("rv", v, u, hv, hu, -2, -1, svs)):
            od = -3 - dim
            cor = sgn * _avg(H * fomn * 0.5 * (o + o.roll(-1, od)), dim)
            X = 0.25 * (hq + hq.roll(-1, dim)) * (q + q.roll(-1, dim))        # at rho points
            E = 0.25 * (ho + ho.roll(1, dim)) * (q + q.roll(1, od))          # at psi points
            r = cor - ((X - X.roll(1, dim)) + (E.roll(-1, od) - E))
            if k == N - 1:
                r = r + tau * dx * dx
            if k == 0:
                o4 = 0.5 * _avg(o + o.roll(-1, od), dim)
                r = r - DRAG * q * torch.sqrt(q * q + o4 * o4) * dx * dx
            out[n][k] = faces(b, r, dim)
    zw = d["z_w"].double()
    for k in range(1, N):
        out["W"][k] -= run_w * (zw[k] - zw[0]) / (zw[N - 1] - zw[0])
    ring = torch.ones_like(b.h, dtype=torch.bool)
    ring[1:-1, 1:-1] = False
    out["W"][:, ring] = 0.0
    return out


def exact_column(c, seed):
    b, d = inputs(c, seed)
    N, dt = b.N, c["dt"]
    fac = dt / b.dx ** 2
    coef = (23 / 12, -16 / 12, 5 / 12)
    out = {}
    for n, r, bar, dim, avg in (("u", "ru", "ubar", -1, "DU"), ("v", "rv", "vbar", -2, "DV")):
        f = lambda a: _avg(a.double(), dim)
        hz = [f(d["Hz"][k]) for k in range(N)]
        zero = torch.zeros_like(b.h)
        FC, Wf = [], [zero]
        for k in range(N - 1):
            FC.append(-dt * f(d["AKv"][k + 1]) / f(d["z_r"][k + 1].double() - d["z_r"][k].double()))
            Wf.append(fac * f(d["W"][k + 1]))
        FC.append(zero)
        Wf.append(zero)
        B, U, R = [], [], []
        for k in range(N):
            fm = FC[k - 1] if k else zero
            x = hz[k] * d[n][k].double() + fac * sum(a * d["%s%d" % (r, s)][k].double() for s, a in enumerate(coef))
            dg = hz[k] - FC[k] - fm + Wf[k + 1].clamp(min=0) - Wf[k].clamp(max=0)
            if k:
                w = (fm - Wf[k].clamp(min=0)) / B[-1]
                dg, x = dg - w * U[-1], x - w * R[-1]
            B.append(dg)
            U.append(FC[k] + Wf[k + 1].clamp(max=0))
            R.append(x)
        X = [None] * N
        X[-1] = R[-1] / B[-1]
        for k in range(N - 2, -1, -1):
            X[k] = (R[k] - U[k] * X[k + 1]) / B[k]
        H = sum(hz)
        target = d[avg].double() / b.dx
        du = (sum(h * x for h, x in zip(hz, X)) - target) / H
        q = torch.zeros((N + 1, b.J, b.I), device="cuda", dtype=F64)
        for k in range(N):
            q[k] = faces(b, X[k] - du, dim)
        out[n], out[bar] = q, faces(b, target / H, dim)
    return out


def _gls(c, model, d, N, dt):
    """The GLS corrector's column physics on every interior column (rows and columns 1..-2)."""
    P = dict(Kmin=7.6e-6, Pmin=1e-12, Akv_bak=1e-5, Akt_bak=1e-6, Akk_bak=5e-6, Akp_bak=5e-6,
             **closure.GLS_PRESETS[model])
    p, m, n, cmu0, sk, sp = (P[k] for k in ("p", "m", "n", "cmu0", "sigk", "sigp"))
    Zos, Zob, kap, eps = 0.02, 0.02, 0.41, 1e-10
    C = lambda a: a.double()[1:-1, 1:-1]
    at = {k: [C(d[k][l]) for l in range(N + 1)] for k in ("tke", "gls", "AKv", "Akt", "Akk", "Akp", "Lscale", "bvf")}
    Hz, zr = [C(d["Hz"][k]) for k in range(N)], [C(d["z_r"][k]) for k in range(N)]
    zero = torch.zeros_like(Hz[0])
    FK, FP = [zero] * (N + 1), [zero] * (N + 1)
    for k in range(2, N):
        FK[k] = -0.5 * dt * (at["Akk"][k] + at["Akk"][k - 1]) / Hz[k - 1]
        FP[k] = -0.5 * dt * (at["Akp"][k] + at["Akp"][k - 1]) / Hz[k - 1]
    tk, gl, BK, BP = ([None] * (N + 1) for _ in range(4))
    sh = lambda a: a[1:-1, 1:-1] + a[1:-1, 2:]
    sv = lambda a: a[1:-1, 1:-1] + a[2:, 1:-1]
    for k in range(1, N):
        cff = 0.5 / (zr[k] - zr[k - 1])
        du, dv = sh(d["u"][k].double() - d["u"][k - 1].double()), sv(d["v"][k].double() - d["v"][k - 1].double())
        s2, hz = (cff * du) ** 2 + (cff * dv) ** 2, 0.5 * (Hz[k - 1] + Hz[k])
        t0, g0, n2 = at["tke"][k], at["gls"][k], at["bvf"][k]
        c3 = torch.where(n2 > 0, zero + P["c3m"], zero + P["c3p"])
        bt, bv = n2 * (at["Akt"][k] - P["Akt_bak"]), at["AKv"][k] - P["Akv_bak"]
        kp, pp = s2 * bv - bt, P["c1"] * s2 * bv - c3 * bt
        neg, negp = kp < 0, pp < 0
        kp, pp = torch.where(neg, kp + bt, kp), torch.where(negp, pp + c3 * bt, pp)
        tk[k], gl[k] = hz * t0 + dt * hz * kp, hz * g0 + dt * hz * pp * g0 / t0.clamp(min=P["Kmin"])
        diss = g0 ** (-1 / n) * cmu0 ** (3 + p / n) * t0 ** (0.5 + m / n)
        BK[k] = hz * (1 + dt * diss + dt * neg * bt / t0) - FK[k] - FK[k + 1]
        BP[k] = hz * (1 + dt * P["c2"] * diss + dt * negp * c3 * bt / t0) - FP[k] - FP[k + 1]
    ub, vb = d["u"][0].double(), d["v"][0].double()
    bu = DRAG * ub * torch.sqrt(ub ** 2 + (0.5 * _avg(vb + vb.roll(-1, -2), -1)) ** 2)
    bv = DRAG * vb * torch.sqrt(vb ** 2 + (0.5 * _avg(ub + ub.roll(-1, -1), -2)) ** 2)
    tk[N] = (0.5 / cmu0 ** 2 * torch.hypot(sh(d["sustr"].double()), sv(d["svstr"].double()))).clamp(min=P["Kmin"])
    tk[0] = (0.5 / cmu0 ** 2 * torch.hypot(sh(bu), sv(bv))).clamp(min=P["Kmin"])
    gl[N] = (cmu0 ** p * tk[N] ** m * (kap * Zos) ** n).clamp(min=P["Pmin"])
    gl[0] = (cmu0 ** p * (kap * Zob) ** n * tk[0] ** m).clamp(min=P["Pmin"])
    CF = [None] * (N + 1)

    def down(F, B, x):
        for k in range(N - 1, 0, -1):
            cf = 1 / (B[k] - CF[k + 1] * F[k + 1]) if k < N - 1 else 1 / B[k]
            x[k] = cf * (x[k] - F[k + 1] * x[k + 1]) if k < N - 1 else cf * x[k]
            CF[k] = cf * F[k]
        return cf

    down(FK, BK, tk)
    tk[1] = tk[1].clamp(min=P["Kmin"])
    for k in range(2, N):
        tk[k] = (tk[k] - CF[k] * tk[k - 1]).clamp(min=P["Kmin"])
    ft = dt * cmu0 ** p * n * (0.5 * (tk[N] + tk[N - 1])) ** m * kap ** n * (Zos + 0.5 * Hz[N - 1]) ** (n - 1) * \
        0.5 * (at["Akp"][N] + at["Akp"][N - 1])
    fb = dt * cmu0 ** p * n * kap ** n * (0.5 * (tk[0] + tk[1])) ** m * (0.5 * Hz[0] + Zob) ** (n - 1) * \
        0.5 * (at["Akp"][0] + at["Akp"][1])
    gl[N - 1] = gl[N - 1] - ft
    cf = down(FP, BP, gl)
    gl[1] = gl[1] - cf * fb
    for k in range(2, N):
        gl[k] = gl[k] - CF[k] * gl[k - 1]
    A1, A2, B1, B2, C1 = 0.92, 0.74, 16.6, 10.1, 0.08
    new = {q: [None] * (N + 1) for q in ("tke", "gls", "AKv", "Akt", "Akk", "Akp", "Lscale")}
    for k in range(1, N):
        b2 = at["bvf"][k]
        b2p = b2.clamp(min=0)
        t, g = tk[k].clamp(min=P["Kmin"]), gl[k].clamp(min=P["Pmin"])
        lim = 0.56 ** (0.5 * n) * cmu0 ** p * t ** (m + 0.5 * n) * (b2p.sqrt() + eps) ** (-n)
        g = torch.minimum(g, lim) if n >= 0 else torch.maximum(g, lim)
        Ls = (g ** (1 / n) * cmu0 ** (-p / n) * t ** (-m / n)).clamp(min=eps)
        Ls = torch.where(b2 > 0, torch.minimum(Ls, torch.sqrt(0.56 * t / (b2p + eps))), Ls)
        g = (cmu0 ** p * t ** m * Ls ** n).clamp(min=P["Pmin"])
        Gh = (-b2 * Ls * Ls / (2 * t)).clamp(max=0.0233)
        Gh = torch.minimum(Gh, Gh - (Gh - 0.02) ** 2 / (Gh + 0.0233 - 0.04)).clamp(min=-0.28)
        Sh = A2 * (1 - 6 * A1 / B1) / (1 - 3 * A2 * (6 * A1 + B2) * Gh)
        Sm = (A1 * (1 - 3 * C1 - 6 * A1 / B1) + Sh * Gh * (18 * A1 * A1 + 9 * A1 * A2)) / (1 - 9 * A1 * A2 * Gh)
        ql = math.sqrt(2.0) * 0.5 * (Ls * t.sqrt() + at["Lscale"][k] * at["tke"][k].sqrt())
        for q, a in dict(tke=t, gls=g, AKv=P["Akv_bak"] + Sm * ql, Akt=P["Akt_bak"] + Sh * ql, Lscale=Ls,
                         Akk=P["Akk_bak"] + Sm * ql / sk, Akp=P["Akp_bak"] + Sm * ql / sp).items():
            new[q][k] = a
    for k, z in ((N, Zos), (0, Zob)):
        a = P["Akv_bak"] + kap * z * cmu0 * tk[k].sqrt()
        for q, x in dict(tke=tk[k], gls=gl[k], AKv=a, Akt=zero + P["Akt_bak"], Akk=P["Akk_bak"] + a / sk,
                         Akp=P["Akp_bak"] + a / sp, Lscale=at["Lscale"][k]).items():
            new[q][k] = x
    return new


def exact_gls(c, seed):
    b, d = inputs(c, seed)
    new = _gls(c, c["model"], d, b.N, c["dt"])
    out = {q: d[q].double() for q in new}
    for q, a in new.items():
        for k in range(b.N + 1):
            out[q][k, 1:-1, 1:-1] = a[k]
    return out


def _network(c, d, b):
    """log10 of Akv and Akt at levels 1..N-1 (N-1, J, I) and whether a column is in range."""
    w = np.load(os.path.join(WEIGHTS, c["net"]))
    t = lambda a: torch.tensor(np.asarray(a, np.float64), device="cuda")
    N = b.N
    X = torch.zeros((b.J, b.I, 128), device="cuda", dtype=F64)
    for k in range(1, N):
        cff = 0.5 / (d["z_r"][k].double() - d["z_r"][k - 1].double())
        du, dv = (d[q][k].double() - d[q][k - 1].double() for q in ("u", "v"))
        X[..., k - 1] = torch.log10((cff * (du + du.roll(-1, -1))) ** 2 + (cff * (dv + dv.roll(-1, -2))) ** 2 + 1e-12)
        n2 = d["bvf"][k].double()
        X[..., N - 2 + k] = torch.copysign(torch.log10(1 + n2.abs() * 1e8), n2)
    su = d["sustr"].double()
    sv = d["svstr"].double()
    X[..., 2 * N - 2] = torch.log10(0.5 * torch.hypot(su + su.roll(-1, -1), sv + sv.roll(-1, -2)) + 1e-10)
    X[..., 2 * N] = torch.log10(b.h)
    nf = 2 * (N - 1) + 3
    ok = ((X >= t(w["lo"])) & (X <= t(w["hi"])))[..., :nf].all(-1)
    X = ((X - t(w["mu"])) * t(w["isd"])).reshape(-1, 128)
    gelu = "act" not in w or str(w["act"]) == "gelu"
    for l in range(5):
        X = X @ t(w["W"][l]).T + t(w["b"][l])
        if l < 4:
            X = torch.nn.functional.gelu(X, approximate="tanh") if gelu else X.relu()
    Y = X.clamp(-6.0, -1.0).T.reshape(128, b.J, b.I)
    return Y[:N - 1], Y[N - 1:2 * N - 2], ok, str(w["gls_model"]) if "gls_model" in w else "k-epsilon"


def exact_closure(c, seed, d=None, b=None, dt=None):
    if d is None:
        b, d = inputs(c, seed)
    N = b.N
    kv, kt, ok, model = _network(c, d, b)
    full = lambda a: torch.full((N + 1, b.J, b.I), a, device="cuda", dtype=DTYPE[c["prec"]])
    d = dict(d, AKv=full(1e-3), Akt=full(1e-6), Akk=full(5e-6), Akp=full(5e-6), tke=full(7.6e-6),
             gls=full(1e-12), Lscale=full(0.0))
    AKv, Akt = d["AKv"].double(), d["Akt"].double()
    inside = ok[1:-1, 1:-1]
    new = _gls(c, model, d, N, c["dt"]) if not bool(inside.all()) else None
    for k in range(N + 1):
        for a, y, q in ((AKv, kv, "AKv"), (Akt, kt, "Akt")):
            v = a[k, 1:-1, 1:-1]
            if 1 <= k < N:
                v[inside] = (10.0 ** y[k - 1])[1:-1, 1:-1][inside]
            if new is not None:
                v[~inside] = new[q][k][~inside]
    return dict(AKv=AKv, Akt=Akt)


def exact_train(c, seed):
    X, T = (a.double() for a in training_rows(c, seed))
    net = closure.Network(c["N"], seed=seed, act=c["act"])   # the initial weights
    W = [w.double().requires_grad_() for w in net.W]
    b = [w.double().requires_grad_() for w in net.b]
    Y = X
    for l in range(5):
        Y = Y @ W[l].to(torch.bfloat16).double().detach().T + b[l] + Y @ (W[l] - W[l].detach()).T
        if l < 4:
            Y = torch.nn.functional.gelu(Y, approximate="tanh") if c["act"] == "gelu" else Y.relu()
    no = 2 * (c["N"] - 1)
    loss = ((Y - T)[:, :no] ** 2).mean()
    grads = torch.autograd.grad(loss, W + b)
    new = [(w - 2e-3 * g / (g.abs() + 1e-8)).detach() for w, g in zip(W + b, grads)]
    return dict(loss=loss.detach().reshape(1), Y=Y.detach(), dW=list(grads[:5]), db=list(grads[5:]),
                W=new[:5], b=new[5:])


def exact_step(c, seed):
    """The reference's semantics from rest stay at rest; the mixing is the closure's at rest."""
    if c["semantics"] != "reference":
        return None
    b, d = inputs(c, seed)
    z = torch.zeros_like(b.h)
    real = DTYPE[c["prec"]]
    d["z_w"], d["z_r"], d["Hz"] = (a.to(real) for a in b.depths(z))
    z3 = torch.zeros((b.N + 1, b.J, b.I), device="cuda", dtype=F64)
    d["u"] = d["v"] = z3.to(real)
    out = {n: z for n in ("zeta", "ubar", "vbar")}
    out.update({n: z.reshape(-1) for n in ("Zt_avg1", "DU_avg1", "DV_avg1")})
    return dict(out, u=z3, v=z3, W=z3, AKv=exact_closure(c, seed, d, b)["AKv"])


EXACT = dict(main2d=exact_main2d, loop=exact_loop, rhs=exact_rhs, column=exact_column, gls=exact_gls,
             closure=exact_closure, train=exact_train, step=exact_step)
