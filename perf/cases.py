"""The work that programs have this framework do, as cases that can be timed and compared.

A case is a dict of plain values. `prepare` makes what a program has in hand
before the call (inputs from a seed, on the GPU or, for the host binding, in
numpy), `run` is one pass through the public entry points, `work` the bytes
and operations the pass cannot do without, and `exact` the same outputs in
plain FP64 torch.

Scenes (the geometry of the benchmark configurations, on grids of any size):
  feed   Gaussian feed plane +-50 mm (w0 10 mm, lambda 3 mm; J and M) onto an
         f 300, D 300 paraboloid that faces it
  dish   illuminated paraboloid (D 1000, f 500, lambda 1 mm; M = 0) onto its
         focal plane +-50 mm
  far    illuminated paraboloid (D 2000, f 800, lambda 1 mm; M = 0) into the
         far field +-0.5 deg
"""
import math

import numpy as np
import torch

from pypo_gb300 import BindGPU, PyPOTypes, autograd, beams, efficiencies, engine, fitgauss, surfaces

FLOAT_PI = float(np.float32(3.14159265359))   # the reference's float-literal pi
LAM = {"feed": 3.0, "dish": 1.0, "far": 1.0}
ROWS_OUT = {"JM": 12, "EH": 12, "JMEH": 24, "EHP": 15, "FF": 12, "scalar": 2}


def listed():
    return [
        # a small propagation inside a larger loop: the call's own cost counts
        dict(name="feed_small", kind="forward", scene="feed", mode="JM", sx=31, sy=33, tx=29, ty=31, precision="mixed"),
        # runPO on a small grid through PyPO's own binding, numpy in and out
        dict(name="binding_small", kind="binding", scene="feed", mode="EH", sx=31, sy=31, tx=31, ty=31),
        # one optimisation step on a feed and its dish: outputs and every gradient
        dict(name="feed_dish_step", kind="step", scene="feed", mode="JM", sx=101, sy=101, tx=101, ty=101,
             precision="mixed"),
        # the focal field of a large dish
        dict(name="dish_focal", kind="forward", scene="dish", mode="EH", sx=501, sy=501, tx=301, ty=301,
             precision="mixed"),
        # sensitivities of the focal field of a mid-size dish, odd sizes
        dict(name="dish_focal_adjoint", kind="adjoint", scene="dish", mode="EH", sx=251, sy=249, tx=151, ty=149,
             precision="mixed"),
        # the beam of a large dish
        dict(name="dish_far", kind="forward", scene="far", mode="FF", sx=1001, sy=1001, tx=401, ty=401,
             precision="mixed"),
        # sensitivities of the beam
        dict(name="dish_far_adjoint", kind="adjoint", scene="far", mode="FF", sx=501, sy=499, tx=201, ty=203,
             precision="mixed"),
        # one draw of a surface-error study: grids, feed and error made on the
        # device, feed -> dish -> far field, gradient with respect to the error
        dict(name="surface_error_chain", kind="chain", feed=101, dish=301, far=101),
        # runPO onto a reflector through PyPO's own binding
        dict(name="binding_reflector", kind="binding", scene="feed", mode="JM", sx=101, sy=101, tx=201, ty=201),
        # one trial of a grid-size search (scalar propagation)
        dict(name="scalar_trial", kind="forward", scene="feed", mode="scalar", sx=101, sy=103, tx=121, ty=119,
             precision="mixed"),
        # the plain FP64 sum, taken where a scene is too large for the mixed path: outputs and gradients
        dict(name="fp64_step", kind="step", scene="dish", mode="EH", sx=101, sy=99, tx=41, ty=43, precision="fp64"),
        # a beam's figures of merit: spillover, taper, cross-polar, Gaussian fit and main beam
        dict(name="beam_figures", kind="figures", nx=201, ny=201),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "adjoint", "step", "step64", "binding", "chain", "figures"])
    if kind == "chain":
        return dict(kind="chain", feed=_logint(rng, 21, 101), dish=_logint(rng, 61, 301), far=_logint(rng, 21, 101))
    if kind == "figures":
        return dict(kind="figures", nx=_logint(rng, 61, 301), ny=_logint(rng, 61, 301))
    if kind == "binding":
        s, t = _logint(rng, 13, 201), _logint(rng, 13, 201)
        return dict(kind="binding", scene="feed", mode=rng.choice(["JM", "EH", "JMEH", "scalar"]), sx=s,
                    sy=s + rng.randint(0, 3), tx=t, ty=t + rng.randint(0, 3))
    if kind == "step64":
        s, t = _logint(rng, 13, 101), _logint(rng, 13, 51)
        scene = rng.choice(["feed", "dish", "far"])
        return dict(kind="step", scene=scene, mode="FF" if scene == "far" else rng.choice(["EH", "JM"]), sx=s,
                    sy=s + rng.randint(0, 3), tx=t, ty=t + rng.randint(0, 3), precision="fp64")
    scene = rng.choice(["feed", "dish", "far"])
    mode = "FF" if scene == "far" else rng.choice(["JM", "EH", "JMEH", "EHP", "scalar"] if kind == "forward" else
                                                  ["JM", "EH", "JMEH", "scalar"])
    s, t = _logint(rng, 17, 351 if kind == "forward" else 201), _logint(rng, 17, 201 if kind == "forward" else 151)
    return dict(kind=kind, scene=scene, mode=mode, sx=s, sy=s + rng.randint(0, 3), tx=t, ty=t + rng.randint(0, 3),
                precision="mixed")


# ------------------------------------------------------------------- scenes

def _facing(f, D, n, m):
    return surfaces.translate(surfaces.rotate_x(surfaces.paraboloid(f, [n, m], gmode=1, lims_a=[0.0, D / 2]), 180.0),
                              dz=f)


def _reflectors(scene, sx, sy, tx, ty):
    if scene == "feed":
        return surfaces.plane([sx, sy], gmode=0, lims_a=[-50.0, 50.0]), _facing(300.0, 300.0, tx, ty)
    if scene == "dish":
        return (surfaces.paraboloid(500.0, [sx, sy], gmode=1, lims_a=[0.0, 500.0]),
                surfaces.translate(surfaces.plane([tx, ty], gmode=0, lims_a=[-50.0, 50.0]), dz=500.0))
    return (surfaces.paraboloid(800.0, [sx, sy], gmode=1, lims_a=[0.0, 1000.0]),
            surfaces.farfield([tx, ty], [-0.5, 0.5], [-0.5, 0.5]))


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _currents(scene, s7, g):
    """Source currents (12, ns): the feed's J and M, or a dish's tapered
    tangential J, each point with a small random amplitude and phase."""
    n = s7.shape[1]
    c = (1.0 + 0.05 * _randn(g, n)) * torch.exp(0.05j * _randn(g, n))
    if scene == "feed":
        _, cur = beams.gauss_beam_dev(s7, LAM[scene], 10.0, 0.0, 4 * math.pi)
        v = torch.complex(cur.view(2, 2, 3, n)[:, 0], cur.view(2, 2, 3, n)[:, 1]) * c
        return torch.stack([v.real, v.imag], dim=1).reshape(12, n).contiguous()
    r = torch.hypot(s7[0], s7[1])
    taper = torch.exp(-0.5 * math.log(10.0) * (r / r.max()) ** 2)
    nrm = s7[3:6]
    pol = torch.zeros_like(nrm)
    pol[0] = 1.0
    jt = (pol - nrm[0] * nrm) * (taper * c)
    cur = torch.zeros((12, n), dtype=torch.float64, device="cuda")
    cur[0:3], cur[3:6] = jt.real, jt.imag
    return cur


def _inputs(case, seed):
    g = _gen(seed)
    src, tgt = _reflectors(case["scene"], case["sx"], case["sy"], case["tx"], case["ty"])
    s7, t7 = engine.generate_grid_dev(src), engine.generate_grid_dev(tgt)
    cur = _currents(case["scene"], s7, g)
    if case["mode"] == "scalar":
        cur = cur[[0, 3]].contiguous()
    return dict(case=case, s7=s7, t7=t7, cur=cur, grid=(src["gmode"], case["sx"], case["sy"]),
                k=2 * math.pi / LAM[case["scene"]], m_zero=case["scene"] != "feed",
                cot=_randn(g, ROWS_OUT[case["mode"]], t7.shape[1]), src=src, tgt=tgt, g=g)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        return dict(case=case, seed=int(seed) % (1 << 31), cot=_randn(_gen(seed), 12, case["far"] ** 2))
    if kind == "figures":
        return _prepare_figures(case, seed)
    st = _inputs(case, seed)
    if kind == "step":
        near = case["mode"] != "FF"
        st["cur"].requires_grad_(True)
        st["ds"] = (1e-3 * _randn(st["g"], st["s7"].shape[1])).requires_grad_(True)
        st["dt"] = (1e-3 * _randn(st["g"], st["t7"].shape[1])).requires_grad_(True) if near else None
    if kind == "adjoint":
        ns, nt = st["s7"].shape[1], st["t7"].shape[1]
        new = lambda *shape: torch.empty(shape, dtype=torch.float64, device="cuda")
        st["grads"] = (new(*st["cur"].shape), new(ns), None if case["mode"] == "FF" else new(nt))
    if kind == "binding":
        host = st["cur"].cpu().numpy()
        shape = (case["sx"], case["sy"])
        run_dict = dict(mode=case["mode"], exp="fwd", epsilon=1.0, k=st["k"])
        if case["mode"] == "scalar":
            run_dict["s_scalarfield"] = PyPOTypes.scalarfield((host[0] + 1j * host[1]).reshape(shape))
        else:
            c = [(host[6 * a + i] + 1j * host[6 * a + 3 + i]).reshape(shape) for a in range(2) for i in range(3)]
            run_dict["s_current"] = PyPOTypes.currents(*c)
        return dict(case=case, src=st["src"], tgt=st["tgt"], run_dict=run_dict)
    return st


# ---------------------------------------------------------------------- run

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "chain":
        return _run_chain(state)
    if kind == "figures":
        return _run_figures(state)
    if kind == "binding":
        out = BindGPU.PyPO_GPUf(state["src"], state["tgt"], state["run_dict"])
        if case["mode"] == "scalar":
            return out.S
        parts = out if isinstance(out, list) else [out]
        return [p[i] for p in parts for i in range(6)]
    mode, prec = case["mode"], case["precision"]
    if kind == "forward":
        return engine.propagate_dev(mode, state["s7"], state["cur"], *state["grid"], state["t7"], state["k"],
                                    precision=prec, m_zero=state["m_zero"])
    if kind == "adjoint":
        gc, gs, gt = state["grads"]
        engine.adjoint_dev(mode, state["s7"], state["cur"], *state["grid"], state["t7"], state["k"], state["cot"],
                           precision=prec, m_zero=state["m_zero"], grad_cur=gc, grad_ds=gs, grad_dt=gt)
        return [gc, gs] if gt is None else [gc, gs, gt]
    out = autograd.propagate(mode, state["s7"], state["cur"], *state["grid"], state["t7"], state["k"],
                             ds=state["ds"], dt=state["dt"], precision=prec)
    wrt = [v for v in (state["cur"], state["ds"], state["dt"]) if v is not None]
    return [out.detach(), *torch.autograd.grad(out, wrt, grad_outputs=state["cot"])]


CHAIN_LAM = 2.0


def _run_chain(state):
    """Feed (w0 10 mm, +-50 mm) -> D 600, f 400 dish with a correlated error
    (rms lambda / 40 over 30 mm) -> far field +-1 deg, and the gradient of a
    linear loss with respect to the error."""
    c, k = state["case"], 2 * math.pi / CHAIN_LAM
    feed = surfaces.plane([c["feed"], c["feed"]], gmode=0, lims_a=[-50.0, 50.0])
    f7 = engine.generate_grid_dev(feed)
    d7 = engine.generate_grid_dev(_facing(400.0, 600.0, c["dish"], c["dish"]))
    ff7 = engine.generate_grid_dev(surfaces.farfield([c["far"], c["far"]], [-1.0, 1.0], [-1.0, 1.0]))
    ff7[0] = math.pi - ff7[0]
    _, cur = beams.gauss_beam_dev(f7, CHAIN_LAM, 10.0, 0.0, 4 * math.pi)
    delta = engine.correlated_error_dev(d7, CHAIN_LAM / 40.0, 30.0, state["seed"]).requires_grad_(True)
    on_dish = autograd.propagate("JM", f7, cur, 0, c["feed"], c["feed"], d7, k, dt=delta)
    far = autograd.propagate("FF", d7, on_dish, 1, c["dish"], c["dish"], ff7, k, ds=delta)
    grad, = torch.autograd.grad(far, [delta], grad_outputs=state["cot"])
    return [far.detach(), grad, delta.detach()]


def _prepare_figures(case, seed):
    """An Airy-like beam on a +-0.5 deg far-field grid with a weak
    cross-polar part, its width and pointing drawn from the seed."""
    g = _gen(seed)
    refl = surfaces.farfield([case["nx"], case["ny"]], [-0.5, 0.5], [-0.5, 0.5])
    plain = engine.generate_grid_dev(refl, transform=False, spheric=False)
    n = plain.shape[1]
    off = 0.02 * torch.rand(3, generator=g, dtype=torch.float64, device="cuda")
    r = torch.hypot(1.1 * (plain[0] - off[0]), plain[1] - off[1]) * (1.0 + off[2])
    z = r * (3.8317059702075125 / 0.25) + 1e-12
    beam = 2.0 * torch.special.bessel_j1(z) / z
    f = torch.zeros((12, n), dtype=torch.float64, device="cuda")
    f[0], f[3] = beam * torch.cos(0.3 * r), beam * torch.sin(0.3 * r)
    f[1] = 1e-3 * plain[0] * plain[1] * beam
    f[4] = 1e-4 * _randn(g, n)
    return dict(case=case, plain=plain, spheric=engine.generate_grid_dev(refl, transform=False), f=f,
                aper=dict(shape="ell", center=np.zeros(2), outer=np.array([0.004, 0.004])))


def _run_figures(st):
    case = st["case"]
    popt = fitgauss.fit_gauss_abs_dev(st["plain"], case["nx"], case["ny"], st["f"], 0)
    return [efficiencies.spillover_dev(st["spheric"], st["f"], 0, st["aper"]),
            efficiencies.taper_dev(st["spheric"], st["f"], 0),
            efficiencies.xpol_dev(st["spheric"], st["f"], 0, 1),
            fitgauss.calc_main_beam_dev(st["plain"], case["nx"], case["ny"], st["f"], 0), popt]


# --------------------------------------------------------------------- work

def _prop_work(mode, ns, nt, has_m, forward=True, adjoint=False):
    """Operations per pair (FMA = 2): the counts of the kernel formulas."""
    ncur, nout = (2 if mode == "scalar" else 12), ROWS_OUT[mode]
    if mode == "scalar":
        f, b = 25, 40
    elif mode == "FF":
        f, b = (61, 147) if has_m else (37, 99)
    else:
        f, b = (234, 608) if has_m else (140, 466)
    nbytes, flops = 0, 0
    if forward:
        nbytes += 8 * (ns * (7 + ncur) + nt * (7 + nout))
        flops += f * ns * nt
    if adjoint:
        nbytes += 8 * (ns * (7 + 2 * ncur + 1) + nt * (7 + nout + 1))
        flops += b * ns * nt
    return dict(bytes=nbytes, flops=flops)


def work(case):
    kind = case["kind"]
    if kind == "figures":   # each field row once per figure, the region's Gaussian once
        n = case["nx"] * case["ny"]
        return dict(bytes=8 * n * (5 + 5 + 4 + 4 + 4), flops=60 * n)
    if kind == "chain":
        nf, nd, na = case["feed"] ** 2, case["dish"] ** 2, case["far"] ** 2
        a = _prop_work("JM", nf, nd, True, adjoint=True)
        b = _prop_work("FF", nd, na, False, adjoint=True)
        return dict(bytes=a["bytes"] + b["bytes"], flops=a["flops"] + b["flops"])
    return _prop_work(case["mode"], case["sx"] * case["sy"], case["tx"] * case["ty"], case["scene"] == "feed",
                      forward=kind != "adjoint", adjoint=kind in ("adjoint", "step"))


# -------------------------------------------------------------------- exact
#
# The same sums in FP64 torch, written from the physical-optics formulas:
# every source's currents times trapezoid weight, area and prefactor, the
# dyadic Green's function in e^{jwt}, unlit sources left out.

def _weights(ns, gmode, ncx, ncy):
    w = torch.ones((ncx, ncy), dtype=torch.float64, device="cuda")
    w[0] *= 0.5
    w[-1] *= 0.5
    if gmode != 1:
        w[:, 0] *= 0.5
        w[:, -1] *= 0.5
    return w.reshape(ns)


def _cross(a, b):
    """a x b over the first axis (three entries each)."""
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _rows(*vs):
    return torch.cat([p for v in vs for p in (v.real, v.imag)])


def _sum_over_sources(mode, s, ns_, cur, wa, t7, tp, k, t=-1.0):
    """Output rows at targets tp (3, m) of sources s (3, n)."""
    pref = k * k / (4.0 * FLOAT_PI)
    if mode == "FF":
        th, ph = t7[0], t7[1]
        r = torch.stack([torch.cos(ph) * torch.sin(th), torch.sin(ph) * torch.sin(th), torch.cos(th)])
        lit = (ns_.T @ r >= 0).double()
        G = torch.polar(lit, -t * k * (s.T @ r))                        # n x m
        c = torch.complex(cur.view(2, 2, 3, -1)[:, 0], cur.view(2, 2, 3, -1)[:, 1]) * (-1j * pref * wa)
        S = c.reshape(6, -1) @ G
        SJ, SM = S[:3], S[3:]
        dot = lambda v: (v * r).sum(0)
        return _rows(SJ - dot(SJ) * r + t * _cross(r, SM), SM - dot(SM) * r - t * _cross(r, SJ))
    d = [tp[c][None, :] - s[c][:, None] for c in range(3)]              # n x m each
    R = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    if mode == "scalar":
        f = torch.complex(cur[0], cur[1]) * (-pref * wa)
        o = f[None] @ (torch.polar(1.0 / R, -t * k * R))
        return torch.cat([o.real, o.imag])
    e = [v / R for v in d]
    lit = (ns_[0][:, None] * e[0] + ns_[1][:, None] * e[1] + ns_[2][:, None] * e[2] >= 0).double()
    u = 1.0 / (k * R)
    Gu = torch.polar(u * lit, t * k * R)
    c1 = Gu * torch.complex(t * u, u * u - 1.0)
    c2 = -3.0 * c1 - 2j * Gu
    c3 = Gu * torch.complex(-u, torch.full_like(u, t))
    c = torch.complex(cur.view(2, 2, 3, -1)[:, 0], cur.view(2, 2, 3, -1)[:, 1]) * (pref * wa)
    out = []
    for a, b, sign in ((c[0], c[1], 1.0), (c[1], c[0], -1.0)):          # E from J (M), H from M (J)
        p = c2 * (a[0][:, None] * e[0] + a[1][:, None] * e[1] + a[2][:, None] * e[2])
        q = [sign * c3 * (b[(i + 1) % 3][:, None] * e[(i + 2) % 3] - b[(i + 2) % 3][:, None] * e[(i + 1) % 3])
             for i in range(3)]
        out.append(torch.stack([a[i] @ c1 + (p * e[i] + q[i]).sum(0) for i in range(3)]))
    E, H = out
    if mode == "EH":
        return _rows(E, H)
    J = 2.0 * _cross(t7[3:6], H)
    jm = _rows(J, torch.zeros_like(J))
    return jm if mode == "JM" else torch.cat([jm, _rows(E, H)])


def _exact_run(mode, s7, cur, grid, t7, k, ds=None, dt=None, cot=None, wants=()):
    """Output rows and, with cot, the gradients of sum(cot * rows) with respect to `wants` ("cur", "ds", "dt")."""
    ns, nt = s7.shape[1], t7.shape[1]
    wa = _weights(ns, *grid) * s7[6]
    zero = lambda v, n: torch.zeros(n, dtype=torch.float64, device="cuda") if v is None else v.detach()
    cur, ds, dt = cur.detach().clone(), zero(ds, ns).clone(), zero(dt, nt).clone()
    leaves = {"cur": cur, "ds": ds, "dt": dt}
    for w in wants:
        leaves[w].requires_grad_(True)
    total = {w: torch.zeros_like(leaves[w]) for w in wants}
    rows = torch.empty((ROWS_OUT[mode], nt), dtype=torch.float64, device="cuda")
    step = max(1, (40_000_000 if mode in ("FF", "scalar") else 12_000_000) // ns)
    for a in range(0, nt, step):
        b = min(nt, a + step)
        with torch.set_grad_enabled(bool(wants)):
            s = s7[0:3] + ds * s7[3:6]
            tc = t7[:, a:b]
            tp = tc[0:3] + dt[a:b] * tc[3:6]
            o = _sum_over_sources(mode, s, s7[3:6], cur, wa, tc, tp, k)
        rows[:, a:b] = o.detach()
        if wants:
            got = torch.autograd.grad(o, [leaves[w] for w in wants], grad_outputs=cot[:, a:b], allow_unused=True)
            for w, v in zip(wants, got):
                if v is not None:
                    total[w] += v
    return rows, [total[w] for w in wants]


def _plain_plane(n, m, half):
    x, y = np.meshgrid(np.linspace(-half, half, n), np.linspace(-half, half, m), indexing="ij")
    g = np.zeros((7, n * m))
    g[0], g[1], g[5] = x.ravel(), y.ravel(), 1.0
    g[6] = (2 * half / (n - 1)) * (2 * half / (m - 1))
    return g


def _plain_facing_dish(f, D, n, m, f32=False):
    """z = r^2 / a^2 (a = 2 sqrt f) on (u, v) = (radius, angle), turned by 180 deg about x and moved to z = f."""
    a = 2.0 * math.sqrt(f)
    a = float(np.float32(a)) if f32 else a
    du, dv = D / 2 / (n - 1), 2 * math.pi / m
    u, v = np.meshgrid(np.arange(n) * du, np.arange(m) * dv, indexing="ij")
    u, v = u.ravel(), v.ravel()
    x, y, z = u * np.cos(v), u * np.sin(v), u * u / a**2
    nx, ny = -2 * x / a**2, -2 * y / a**2
    nrm = np.sqrt(nx * nx + ny * ny + 1.0)
    turn = math.pi
    sn = float(np.float32(math.sin(turn))) if f32 else math.sin(turn)
    g = np.empty((7, n * m))
    g[0], g[1], g[2] = x, -y - sn * z, sn * y - z + f
    g[3], g[4], g[5] = nx / nrm, (-ny - sn) / nrm, (sn * ny - 1.0) / nrm
    g[6] = u * nrm * du * dv
    return g


def _exact_error(d7, rms, corr_len, seed, modes=512):
    """Sum of plane waves: wave vectors and phases from mt19937 deviates, one of each polar pair."""
    raw = np.frombuffer(np.random.RandomState(seed).bytes(4 * 16 * 4 * modes), dtype="<u4").astype(np.float64)
    uni = (raw[0::2] + raw[1::2] * 2.0**32) * 2.0**-64
    x, y = 2 * uni[0::2] - 1, 2 * uni[1::2] - 1
    r2 = x * x + y * y
    ok = (r2 <= 1.0) & (r2 > 0.0)
    g = (y[ok] * np.sqrt(-2 * np.log(r2[ok]) / r2[ok]))[:4 * modes].reshape(modes, 4)
    kx, ky, ph = g[:, 0] / corr_len, g[:, 1] / corr_len, np.arctan2(g[:, 2], g[:, 3])
    kx, ky, ph = (torch.from_numpy(v).cuda() for v in (kx, ky, ph))
    arg = kx[:, None] * d7[0][None] + ky[:, None] * d7[1][None] + ph[:, None]
    return rms * math.sqrt(2.0 / modes) * torch.cos(arg).sum(0)


def _exact_chain(case, seed):
    st = prepare(case, seed)
    k = 2 * math.pi / CHAIN_LAM
    nf, nd, na = case["feed"], case["dish"], case["far"]
    f7 = torch.from_numpy(_plain_plane(nf, nf, 50.0)).cuda()
    d7 = torch.from_numpy(_plain_facing_dish(400.0, 600.0, nd, nd)).cuda()
    az, el = np.meshgrid(np.linspace(-1, 1, na), np.linspace(-1, 1, na), indexing="ij")
    az, el = az.ravel(), el.ravel()
    ff7 = torch.zeros((7, na * na), dtype=torch.float64, device="cuda")
    ff7[0] = torch.from_numpy(math.pi - np.hypot(az, el) * math.pi / 180)
    ff7[1] = torch.from_numpy(np.arctan2(el, az))
    _, cur = beams.gauss_beam(f7.cpu().numpy(), CHAIN_LAM, 10.0, 0.0, 4 * math.pi)
    cur = torch.from_numpy(np.ascontiguousarray(cur)).cuda()
    delta = _exact_error(d7, CHAIN_LAM / 40.0, 30.0, st["seed"])
    on_dish, _ = _exact_run("JM", f7, cur, (0, nf, nf), d7, k, dt=delta)
    far, (g_cur, g_far) = _exact_run("FF", d7, on_dish, (1, nd, nd), ff7, k, ds=delta, cot=st["cot"],
                                     wants=("cur", "ds"))
    _, (g_dish,) = _exact_run("JM", f7, cur, (0, nf, nf), d7, k, dt=delta, cot=g_cur, wants=("dt",))
    return [far, g_far + g_dish, delta]


def _exact_binding(case, seed):
    """The float ABI's numbers: parameters, wavenumber and currents rounded to float32, the sums in FP64."""
    st = prepare(case, seed)
    s7 = torch.from_numpy(_plain_plane(case["sx"], case["sy"], 50.0)).cuda()
    t7 = torch.from_numpy(_plain_facing_dish(300.0, 300.0, case["tx"], case["ty"], f32=True)).cuda()
    rd = st["run_dict"]
    src = [rd["s_scalarfield"].S] if case["mode"] == "scalar" else [rd["s_current"][i] for i in range(6)]
    c = torch.stack([torch.from_numpy(np.ascontiguousarray(v.ravel())) for v in src]).cuda()
    c = torch.complex(c.real.float().double(), c.imag.float().double())
    cur = _rows(c) if case["mode"] == "scalar" else _rows(c[:3], c[3:])
    rows, _ = _exact_run(case["mode"], s7, cur, (0, case["sx"], case["sy"]), t7, float(np.float32(rd["k"])))
    shape = (case["tx"], case["ty"])
    if case["mode"] == "scalar":
        return torch.complex(rows[0], rows[1]).reshape(shape)
    return [torch.complex(rows[6 * a + i], rows[6 * a + 3 + i]).reshape(shape)
            for a in range(rows.shape[0] // 6) for i in range(3)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "figures" or case.get("mode") == "EHP":
        return None
    if kind == "chain":
        return _exact_chain(case, seed)
    if kind == "binding":
        return _exact_binding(case, seed)
    pairs = case["sx"] * case["sy"] * case["tx"] * case["ty"]
    if pairs > (1.2e10 if case["mode"] == "FF" else 4e9):
        return None
    st = prepare(case, seed)
    args = (case["mode"], st["s7"], st["cur"], st["grid"], st["t7"], st["k"])
    if kind == "forward":
        return _exact_run(*args)[0]
    wants = ("cur", "ds") if case["mode"] == "FF" else ("cur", "ds", "dt")
    rows, grads = _exact_run(*args, ds=st.get("ds"), dt=st.get("dt"), cot=st["cot"], wants=wants)
    return grads if kind == "adjoint" else [rows, *grads]
