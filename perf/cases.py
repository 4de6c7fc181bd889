"""The work that a user of this framework has it do, as cases that can be timed and checked.

A case is one whole use of a public entry point: the initial state goes in, a number of steps are
taken, the final state and the step info come out.  Single domains go through `capi.Solver` (FP64 or
mixed precision), many independent problems through `capi.Batch`, request streams through
`capi.Server`.  `exact` restates the scheme in plain 64-bit torch.
"""
import math

import numpy as np
import torch

from turbostructred_gb300 import capi

RECON = {"pwc": capi.RECON_PWC, "eno2": capi.RECON_ENO2, "bj": capi.RECON_LINEAR2_LIM, "vk": capi.RECON_LINEAR2_LIM}
RIEMANN = {"roe": capi.RS_ROE, "hllc": capi.RS_HLLC}
BC = {"natural": capi.BC_NATURAL, "symmetry": capi.BC_SYMMETRY, "wall": capi.BC_WALL}


def _one(name, prec, scen, nx, ny=1, nz=1, recon="bj", riemann="roe", bc="natural", steps=10, cfl=0.4, eps=0.0,
         t_end=0.0, gravity=0.0, p_in=10.0, host=False):
    """A single domain through Solver; t_end > 0: Solver.run to that time, else `steps` steps."""
    return dict(name=name, kind="solver", prec=prec, scen=scen, nx=nx, ny=ny, nz=nz, recon=recon, riemann=riemann,
                bc=bc, steps=steps, cfl=cfl, eps=eps, t_end=t_end, gravity=gravity, p_in=p_in, host=host)


def listed():
    return [
        # the shock tube every user starts with (the drop-in's own first run): FP64, from host arrays, to t = 0.2
        _one("sod1d_fp64_run", "fp64", "tube", 1000, recon="pwc", cfl=0.5, t_end=0.2, host=True),
        # a short odd-sized tube at second order: the smallest FP64 call
        _one("tube1d_fp64_small", "fp64", "tube", 397, riemann="hllc", steps=64, host=True),
        # a small ragged 2D box with walls and the entropy fix, FP64: many launches of little work
        _one("box2d_fp64_ragged", "fp64", "quadrants", 203, 157, recon="eno2", bc="wall", eps=0.05, steps=40, host=True),
        # the 2D shear layer on the plain FP64 path
        _one("shear2d_fp64_1024", "fp64", "shear", 1024, 1024, riemann="hllc", bc="periodic", steps=16),
        # the 3D blast on the plain FP64 path: what every mixed-precision figure is compared with
        _one("blast3d_fp64_192", "fp64", "blast", 192, 192, 192, bc="symmetry", steps=4),
        # the same tube in mixed precision: latency of a stage
        _one("tube1d_mixed", "mixed", "tube", 1000, steps=256, cfl=0.5, host=True),
        # a small 2D problem of the served sizes, alone
        _one("quad2d_mixed_128", "mixed", "quadrants", 128, 128, steps=200),
        # the 2D shear layer in mixed precision
        _one("shear2d_mixed_1024", "mixed", "shear", 1024, 1024, riemann="hllc", bc="periodic", steps=100),
        # the headline: the 3D blast with reflective walls in mixed precision
        _one("blast3d_mixed_256", "mixed", "blast", 256, 256, 256, bc="symmetry", steps=20),
        # a ragged 3D box under gravity, HLLC
        _one("box3d_mixed_ragged", "mixed", "blast", 97, 61, 83, riemann="hllc", bc="symmetry", steps=40, gravity=-0.3, p_in=1.0),
        # a batch of shock tubes of many sizes, both equations of state, first and second order
        dict(name="batch_tubes", kind="batch", count=192, lo=64, hi=4096, steps=300),
        # a burst of served 2D Riemann problems
        dict(name="served_burst", kind="served", count=24, lo=64, hi=512, steps=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.randrange(8)
    riemann = rng.choice(["roe", "hllc"])
    recon = rng.choice(["pwc", "eno2", "bj", "bj", "bj"])
    prec = rng.choice(["fp64", "mixed"])
    if k <= 1:
        n = _log(rng, 64, 8000)
        c = _one("", prec, "tube", n, recon=recon, riemann=riemann, steps=rng.randrange(32, 257), host=rng.random() < 0.5)
    elif k <= 3:
        top = 1024 if prec == "mixed" else 512
        scen, bc = rng.choice([("shear", "periodic"), ("quadrants", "natural"), ("quadrants", "wall")])
        if scen == "shear":
            recon = rng.choice([recon, "vk"])
        c = _one("", prec, scen, _log(rng, 33, top), _log(rng, 33, top), recon=recon, riemann=riemann, bc=bc,
                 steps=rng.randrange(8, 40), eps=rng.choice([0.0, 0.05]), gravity=rng.choice([0.0, -0.2]))
    elif k <= 5:
        top = 200 if prec == "mixed" else 96
        c = _one("", prec, "blast", _log(rng, 17, top), _log(rng, 17, top), _log(rng, 17, top), recon=recon, riemann=riemann,
                 bc=rng.choice(["symmetry", "periodic"]), steps=rng.randrange(3, 16), p_in=1.0)
    elif k == 6:
        c = dict(kind="batch", count=rng.randrange(8, 193), lo=64, hi=_log(rng, 128, 4096), steps=rng.randrange(50, 301))
    else:
        c = dict(kind="served", count=rng.randrange(4, 25), lo=64, hi=rng.choice([128, 256, 512]), steps=rng.randrange(20, 101))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
def _problem(c):
    """The framework's description of a single domain."""
    nd = 3 if c["nz"] > 1 else (2 if c["ny"] > 1 else 1)
    per = c["bc"] == "periodic"
    b = (BC.get(c["bc"], capi.BC_NATURAL), 0.0, (0.0, 0.0, 0.0), 0.0)
    g = None if c["gravity"] == 0.0 else tuple(c["gravity"] if a == nd - 1 else 0.0 for a in range(3))
    return capi.make_case(ndims=nd, nx=c["nx"], ny=c["ny"], nz=c["nz"], periodic=tuple(int(per or a >= nd) for a in range(3)),
                          recon=RECON[c["recon"]], limiter=capi.LIM_VENKAT if c["recon"] == "vk" else capi.LIM_BJ,
                          solver=RIEMANN[c["riemann"]], eps=c["eps"], cfl=c["cfl"], bc=[b] * 6, uniform_acceleration=g,
                          max_iter=10 ** 7, max_time=c["t_end"] if c["t_end"] > 0 else 1e30)


def _conserved(rho, u, v, w, p, gamma=1.4, p_inf=0.0):
    e = (p + gamma * p_inf) / (gamma - 1.0)
    return torch.stack([rho, rho * u, rho * v, rho * w, e + 0.5 * rho * (u * u + v * v + w * w)], dim=-1)


def _state(c, seed, device):
    """Initial state (nz, ny, nx, 5) of a single domain."""
    g = torch.Generator(device=device).manual_seed(int(seed) * 7919 + 13)
    r = np.random.default_rng(int(seed) + 1)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    x, y, z = [(torch.arange(n, device=device, dtype=torch.float64) + 0.5) / n for n in (nx, ny, nz)]
    Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
    o = torch.zeros_like(X)
    if c["scen"] == "tube":
        left = X < 0.5 + 0.05 * r.uniform(-1, 1)
        rl, ul, pl = 1.0 + 0.1 * r.uniform(-1, 1), 0.1 * r.uniform(-1, 1), 1.0 + 0.1 * r.uniform(-1, 1)
        rho = torch.where(left, rl, 0.125)
        return _conserved(rho, torch.where(left, ul, 0.0), o, o, torch.where(left, pl, 0.1))
    if c["scen"] == "shear":
        mid = (Y - 0.5).abs() < 0.25
        noise = 0.01 * (2.0 * torch.rand(X.shape, generator=g, device=device, dtype=torch.float64) - 1.0)
        return _conserved(torch.where(mid, 2.0, 1.0).double(), torch.where(mid, 0.5, -0.5).double(), noise, o, o + 2.5)
    if c["scen"] == "quadrants":
        q = [(r.uniform(0.3, 2.0), r.uniform(-0.6, 0.6), r.uniform(-0.6, 0.6), r.uniform(0.3, 2.0)) for _ in range(4)]
        f = [torch.where(Y > 0.5, torch.where(X > 0.5, q[0][k], q[1][k]), torch.where(X > 0.5, q[3][k], q[2][k])).double()
             for k in range(4)]
        return _conserved(f[0], f[1], f[2], o, f[3])
    cx, cy, cz = [0.5 + 0.02 * r.uniform(-1, 1) for _ in range(3)]
    hot = (X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2 < 0.01
    noise = 0.01 * (2.0 * torch.rand(X.shape, generator=g, device=device, dtype=torch.float64) - 1.0)
    return _conserved(1.0 + noise, o, o, o, torch.where(hot, c["p_in"], 0.1).double())


def _tubes(c, seed):
    """[(problem, initial state)] of a batch: sizes log-uniform, half ideal and half stiffened gas, two reconstructions."""
    r, sizes = np.random.default_rng(int(seed) * 31 + 5), np.random.default_rng(c["count"])
    out = []
    for k in range(c["count"]):
        n = int(round(math.exp(sizes.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        rho, p = np.exp(r.uniform(math.log(0.2), math.log(5.0), 2)), np.exp(r.uniform(math.log(0.2), math.log(5.0), 2))
        u = r.uniform(-0.5, 0.5, 2)
        stiff = k % 2 == 1
        gamma, p_inf = (4.4, 6.0) if stiff else (1.4, 0.0)
        prob = capi.make_case(ndims=1, nx=n, periodic=(0, 1, 1), gamma=gamma, eos=capi.EOS_STIFFENED if stiff else capi.EOS_IDEAL,
                              p_inf=p_inf, recon=capi.RECON_LINEAR2_LIM if (k // 2) % 2 else capi.RECON_PWC, solver=capi.RS_ROE,
                              cfl=0.5, max_time=1e30, max_iter=c["steps"], bc=[(capi.BC_NATURAL, 0.0, (0.0, 0.0, 0.0), 0.0)] * 6)
        left = torch.from_numpy((np.arange(n) + 0.5) / n < 0.5)
        f = [torch.where(left, float(a[0]), float(a[1])).double() for a in (rho, u, p)]
        o = torch.zeros(n, dtype=torch.float64)
        out.append((prob, _conserved(f[0], f[1], o, o, f[2], gamma, p_inf).reshape(1, 1, n, 5).numpy()))
    return out


def _requests(c, seed):
    """[(case, seed)] of a burst of square 2D Riemann problems, sides and solvers drawn at random."""
    r, kinds = np.random.default_rng(int(seed) * 17 + 3), np.random.default_rng(c["count"])
    sides = [s for s in (64, 128, 256, 512) if c["lo"] <= s <= c["hi"]]
    out = []
    for k in range(c["count"]):
        s = int(sides[kinds.integers(len(sides))]) if k else sides[-1]
        out.append((_one("", "mixed", "quadrants", s, s, riemann=["roe", "hllc"][kinds.integers(2)], steps=c["steps"]),
                    int(r.integers(1 << 30))))
    return out


# ---------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "solver":
        p = _problem(case)
        s = capi.Solver(p, capi.PRECISION_MIXED if case["prec"] == "mixed" else capi.PRECISION_FP64)
        ic = _state(case, seed, "cuda")
        if case["host"]:
            ic = np.ascontiguousarray(ic.cpu().numpy())
            out = np.empty_like(ic)
        else:
            ic = ic.contiguous()
            out = torch.empty_like(ic)
            torch.cuda.synchronize()
        return dict(case=case, solver=s, ic=ic, out=out)
    if case["kind"] == "batch":
        probs = _tubes(case, seed)
        need = sum(capi.batch_problem_bytes(p) for p, _ in probs)
        return dict(case=case, batch=capi.Batch(need + (16 << 20)), probs=probs)
    reqs = []
    for c, sd in _requests(case, seed):
        reqs.append((dict(_problem(c), max_iter=c["steps"]), np.ascontiguousarray(_state(c, sd, "cpu").numpy())))
    srv = capi.Server(memory_budget=4 << 30, order=capi.SERVE_SHORTEST_FIRST, max_cells=16 << 20)
    return dict(case=case, server=srv, reqs=reqs)


def _info(i):
    return {k: i[k] for k in ("iteration", "health", "time", "dt")}


def run(state):
    case = state["case"]
    if case["kind"] == "solver":
        s, ic, out = state["solver"], state["ic"], state["out"]
        if case["host"]:
            s.set_state(ic)
        else:
            s.set_state_device(ic.data_ptr())
        s.set_info(iteration=0, time=0.0)
        info = s.run() if case["t_end"] > 0 else s.step(case["steps"])
        if case["host"]:
            s.get_state(out=out)
        else:
            s.get_state_device(out.data_ptr())
        return dict(state=out, residual=np.array(info["residual"]), **_info(info))
    if case["kind"] == "batch":
        b = state["batch"]
        ids = [b.add(p, ic) for p, ic in state["probs"]]
        b.run()
        got = [b.get(i) for i in ids]
        for i in ids:
            b.remove(i)
    else:
        srv = state["server"]
        ids = [srv.submit(p, ic) for p, ic in state["reqs"]]
        got = [srv.wait(i)[:2] for i in ids]
    infos = [_info(i) for _, i in got]
    return dict(state=np.concatenate([u.reshape(-1) for u, _ in got]),
                iteration=np.array([i["iteration"] for i in infos]), health=np.array([i["health"] for i in infos]),
                time=np.array([i["time"] for i in infos]), dt=np.array([i["dt"] for i in infos]))


# ---------------------------------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------------------------------
def _flops(recon, riemann, nd):
    """Arithmetic of one cell for one step: its faces, its slopes and its update."""
    face = 190 if riemann == "roe" else 130
    slope = {"pwc": 0, "eno2": 5 * 6, "bj": 5 * 9, "vk": 5 * 30}[recon]
    return nd * (face + slope + 20) + 25


def _cell_steps(nx, ny, nz, steps):
    return float(nx) * ny * nz * steps


def work(case):
    """In and out once a pass; a state larger than the chip's caches crosses memory once each way every step."""
    if case["kind"] == "solver":
        cells = float(case["nx"]) * case["ny"] * case["nz"]
        nd = 3 if case["nz"] > 1 else (2 if case["ny"] > 1 else 1)
        steps = case["steps"]
        if case["t_end"] > 0:  # about 2.2 the fastest wave of the tube
            steps = int(case["t_end"] * 2.2 * case["nx"] / case["cfl"])
        trips = steps if cells * 40 > 129e6 else 1
        return {"bytes": 80.0 * cells * trips, "flops": cells * steps * _flops(case["recon"], case["riemann"], nd)}
    if case["kind"] == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])  # of the log-uniform sizes
        cells = case["count"] * mean
        return {"bytes": 80.0 * cells, "flops": cells * case["steps"] * _flops("bj", "roe", 1)}
    sides = [s for s in (64, 128, 256, 512) if case["lo"] <= s <= case["hi"]]
    cells = case["count"] * sum(s * s for s in sides) / len(sides)
    return {"bytes": 80.0 * cells, "flops": cells * case["steps"] * _flops("bj", "roe", 2)}


# ---------------------------------------------------------------------------------------------------
# the scheme in 64 bits
# ---------------------------------------------------------------------------------------------------
def _image(U, kind, a):
    """The state beyond a boundary face on axis a (component dimension last)."""
    V = U.clone()
    if kind == "symmetry":
        V[..., 1 + a] = -V[..., 1 + a]
    elif kind == "wall":
        V[..., 1:4] = -V[..., 1:4]
    return V


def _prim(U, g, pinf):
    r = U[..., 0]
    v = U[..., 1:4] / r[..., None]
    p = (g - 1.0) * (U[..., 4] - 0.5 * r * (v * v).sum(-1)) - g * pinf
    return r, v, p


def _normal_flux(U, v, p, a):
    F = U * v[..., a:a + 1]
    F[..., 1 + a] += p
    F[..., 4] += p * v[..., a]
    return F


def _face(UL, UR, a, riemann, g, pinf, eps):
    rl, vl, pl = _prim(UL, g, pinf)
    rr, vr, pr = _prim(UR, g, pinf)
    FL, FR = _normal_flux(UL, vl, pl, a), _normal_flux(UR, vr, pr, a)
    sl, sr = rl.sqrt(), rr.sqrt()
    ql, qr = sl / (sl + sr), sr / (sl + sr)
    v = ql[..., None] * vl + qr[..., None] * vr
    h = ql * (UL[..., 4] + pl) / rl + qr * (UR[..., 4] + pr) / rr
    q2 = (v * v).sum(-1)
    c = ((g - 1.0) * (h - 0.5 * q2)).sqrt()
    un = v[..., a]
    if riemann == "roe":
        lam = un.abs() + c

        def fix(z):
            z = z.abs()
            if not eps:
                return z
            e = eps * lam
            return torch.where(z < e, (z * z / e + e) * 0.5, z)
        l1, l3, l4 = fix(un), fix(un + c), fix(un - c)
        d = UR - UL
        dp, du, dr = pr - pl, vr[..., a] - vl[..., a], rr - rl
        rho = sl * sr
        a3, a4 = 0.5 * (dp + rho * c * du) / c ** 2, 0.5 * (dp - rho * c * du) / c ** 2
        one = torch.ones_like(h)
        r3 = torch.stack([one, v[..., 0], v[..., 1], v[..., 2], h], -1)
        e = torch.zeros_like(r3)
        e[..., 1 + a] = c
        e[..., 4] = c * un
        D = l1[..., None] * (d - a3[..., None] * (r3 + e) - a4[..., None] * (r3 - e))
        D = D + (l3 * a3)[..., None] * (r3 + e) + (l4 * a4)[..., None] * (r3 - e)
        return 0.5 * (FL + FR - D), lam
    cl, cr = (g * (pl + pinf) / rl).sqrt(), (g * (pr + pinf) / rr).sqrt()
    ul, ur = vl[..., a], vr[..., a]
    SL, SR = torch.minimum(ul - cl, un - c), torch.maximum(ur + cr, un + c)
    ml, mr = rl * (SL - ul), rr * (SR - ur)
    ss = (pr - pl + ul * ml - ur * mr) / (ml - mr)

    def star(U, F, v, p, m, S, u):
        k = m / (S - ss)
        W = k[..., None] * torch.cat([torch.ones_like(k)[..., None], v, torch.zeros_like(k)[..., None]], -1)
        W[..., 1 + a] = k * ss
        W[..., 4] = k * (U[..., 4] / U[..., 0] + (ss - u) * (ss + p / m))
        return F + S[..., None] * (W - U)
    F = torch.where((ss >= 0)[..., None], star(UL, FL, vl, pl, ml, SL, ul), star(UR, FR, vr, pr, mr, SR, ur))
    F = torch.where((SR <= 0)[..., None], FR, F)
    F = torch.where((SL >= 0)[..., None], FL, F)
    return F, torch.maximum(SL.abs(), SR.abs())


def _venkat(um, ui, d2, un, eps2):
    dm, q = (um - ui) / un, d2 / un
    return (dm * dm + eps2 + 2 * q * dm) / (dm * dm + 2 * q * q + dm * q + eps2)


def _evolve(U, h, bc, recon, riemann, g, pinf, cfl, eps, gravity, steps, t_end):
    """U (nz, ny, nx, 5) after `steps` steps (or to t_end), its time, iteration, last dt and residual norms."""
    nd = len(h)
    dim = [2, 1, 0]
    V = math.prod(h)
    t, it, dt = 0.0, 0, 0.0
    norms = torch.zeros(5, dtype=torch.float64, device=U.device)
    while it < steps and (t_end <= 0 or t < t_end):
        lo, hi = [], []
        for a in range(nd):
            n = U.shape[dim[a]]
            first, last = U.narrow(dim[a], 0, 1), U.narrow(dim[a], n - 1, 1)
            lo_g, hi_g = (last, first) if bc == "periodic" else (_image(first, bc, a), _image(last, bc, a))
            P = torch.cat([lo_g, U, hi_g], dim[a])
            lo.append(P.narrow(dim[a], 0, n))
            hi.append(P.narrow(dim[a], 2, n))
        D = []
        for a in range(nd):
            if recon == "pwc":
                D.append(torch.zeros_like(U))
            elif recon == "eno2":
                l, r = (U - lo[a]) / h[a], (hi[a] - U) / h[a]
                D.append(torch.where(l.abs() < r.abs(), l, r) * (0.5 * h[a]))
            else:
                D.append((hi[a] - lo[a]) / (2 * h[a]) * (0.5 * h[a]))
        if recon in ("bj", "vk"):
            umax, umin = U, U
            for w in lo + hi:
                umax, umin = torch.maximum(umax, w), torch.minimum(umin, w)
            lim = torch.ones_like(U)
            eps2 = (5.0 * V ** (1.0 / nd)) ** 3
            for d in D:
                for s in (d, -d):
                    if recon == "bj":
                        k = torch.where(s > 0, (umax - U) / s, torch.where(s < 0, (umin - U) / s, 1.0))
                        lim = torch.minimum(lim, k.clamp(max=1.0))
                    else:
                        un = 0.5 * (umax - umin)
                        k = torch.where(s > 0, _venkat(umax, U, s, un, eps2), _venkat(umin, U, s, un, eps2))
                        lim = torch.where((s != 0) & (un > 0), torch.minimum(lim, k), lim)
            D = [lim * d for d in D]
        R = torch.zeros_like(U)
        SR = torch.zeros_like(U[..., 0])
        least = float("inf")
        for a in range(nd):
            n, area = U.shape[dim[a]], V / h[a]
            up, dn = U + D[a], U - D[a]  # at the high and the low face of a cell
            first, last = dn.narrow(dim[a], 0, 1), up.narrow(dim[a], n - 1, 1)
            before, after = (last, first) if bc == "periodic" else (_image(first, bc, a), _image(last, bc, a))
            F, lam = _face(torch.cat([before, up], dim[a]), torch.cat([dn, after], dim[a]), a, riemann, g, pinf, eps)
            R = R - (F.narrow(dim[a], 1, n) - F.narrow(dim[a], 0, n)) * area
            SR = SR + area * (lam.narrow(dim[a], 0, n) + lam.narrow(dim[a], 1, n))
            least = min(least, float((V / (area * lam.narrow(dim[a], n, 1))).min()))
        if gravity:
            R[..., nd] += U[..., 0] * V * gravity
            R[..., 4] += U[..., nd] * V * gravity
        dt = cfl * min(least, float((V / SR).min()))
        U = U + dt * R / V
        norms = (V * R.abs()).reshape(-1, 5).sum(0)
        t, it = t + dt, it + 1
    return U, t, it, dt, norms


def exact(case, seed):
    if case["kind"] == "solver":
        nd = 3 if case["nz"] > 1 else (2 if case["ny"] > 1 else 1)
        U = _state(case, seed, "cuda")
        h = [1.0 / n for n in (case["nx"], case["ny"], case["nz"])[:nd]]
        U, t, it, dt, norms = _evolve(U, h, case["bc"], case["recon"], case["riemann"], 1.4, 0.0, case["cfl"], case["eps"],
                                      case["gravity"], 10 ** 7 if case["t_end"] > 0 else case["steps"], case["t_end"])
        full = case["prec"] == "fp64"  # the mixed path forms no norms unless asked to
        return dict(state=U, residual=norms if full else None, iteration=None, health=None, time=t, dt=dt)
    if case["kind"] == "batch":
        if case["count"] * case["steps"] > 8000:  # a tube after the other: too long
            return None
        got = [_evolve(torch.from_numpy(ic).cuda(), [1.0 / p["nx"]], "natural", "pwc" if p["recon"] == capi.RECON_PWC else "bj",
                       "roe", p["gamma"], p["p_inf"], p["cfl"], 0.0, 0.0, case["steps"], 0.0) for p, ic in _tubes(case, seed)]
    else:
        got = []
        for c, sd in _requests(case, seed):
            n = c["nx"]
            got.append(_evolve(_state(c, sd, "cpu").cuda(), [1.0 / n, 1.0 / n], "natural", c["recon"], c["riemann"], 1.4, 0.0,
                               c["cfl"], 0.0, 0.0, c["steps"], 0.0))
    return dict(state=torch.cat([g[0].reshape(-1) for g in got]), iteration=None, health=None,
                time=torch.tensor([g[1] for g in got], dtype=torch.float64), dt=torch.tensor([g[3] for g in got], dtype=torch.float64))
