"""The forecasts whose speed is measured, through the framework's public entry points.

A pass is what a driver does between two history outputs: it advances the
state that lives on the GPU by some RK steps and reads the result back (cell
averages, or the point values), or, with `call` "drop_in", it hands a step its
state as host arrays and takes the new state back, as a driver does that only
replaced its time-step routine.  Host buffers are pinned, as such a driver's
would be.

The flows are the seeded balanced flows of the framework's own configurations
(a tilted zonal jet in balance, a height perturbation of spherical harmonics, a
mountain on the larger grids), at their step sizes.

Split precision carries FP32 tendencies on an FP64 state.  It is compared on
the cell averages of the height after a few steps: later its roundings, which
differ between any two forms of the step, have grown past a comparison.

`exact` is the scheme of the model (multi-moment reconstruction, Riemann fluxes,
cubed-sphere halo, Runge-Kutta) in 64-bit torch, from the formulas alone.
"""
import math

import numpy as np
import torch

from mcv_sw_b200 import api

GRAVITY = 9.80616
OMEGA = 7.292e-5
RADIUS = 6.371e6
MEAN_PHI = 2.94e4
STAGES = {"RK3_TVD": 3, "RK4": 4}


def listed():
    def case(name, order, nc, scheme, precision, members, steps, call, flow):
        return dict(name=name, order=order, nc=nc, scheme=scheme, precision=precision, members=members, steps=steps,
                    call=call, flow=flow)

    return [
        # the smallest call: one step of the reference-sized grid, its state handed over as host arrays
        case("drop_in_step", 3, 32, "RK4", "fp64", 1, 1, "drop_in", "smooth"),
        # an hour of the same grid, the state kept on the GPU
        case("small_hour", 3, 32, "RK4", "fp64", 1, 23, "state", "smooth"),
        # the commonest grid of a serving stream, alone on the GPU
        case("serve_48", 4, 48, "RK3_TVD", "mixed", 1, 6, "height", "smooth"),
        # a pool of forecasts on a middle-sized grid of that stream
        case("serve_pool_96", 3, 96, "RK3_TVD", "mixed", 4, 6, "height", "smooth"),
        # a pool of several grids that advance together in one launch
        dict(case("group_48_96", 3, 96, "RK3_TVD", "mixed", 1, 6, "group", "smooth"), others="48,48,96"),
        # one degree in full precision
        case("one_degree", 4, 90, "RK3_TVD", "fp64", 1, 20, "state", "mountain"),
        # an odd number of cells, which no tile divides
        case("odd_181", 3, 181, "RK3_TVD", "fp64", 1, 20, "state", "smooth"),
        # the single large forecast, in both arithmetics
        case("large_mixed", 4, 256, "RK3_TVD", "mixed", 1, 6, "height", "rough"),
        case("large_fp64", 4, 256, "RK3_TVD", "fp64", 1, 8, "cells", "rough"),
        # the ensemble: many states of one grid in every launch
        case("ensemble_64", 3, 128, "RK4", "mixed", 64, 4, "height", "ensemble"),
        # the largest grid, in both arithmetics
        case("finest_mixed", 4, 1024, "RK4", "mixed", 1, 4, "height", "smooth"),
        case("finest_fp64", 4, 1024, "RK4", "fp64", 1, 3, "cells", "smooth"),
    ]


def draw(rng):
    order = rng.choice((3, 4))
    precision = rng.choice(("fp64", "mixed"))
    scheme = rng.choice(("RK3_TVD", "RK4"))
    nc = int(round(math.exp(rng.uniform(math.log(24), math.log(640)))))
    points = 6 * (nc * (order - 1) + 1) ** 2
    most = min(64 if precision == "mixed" else 16, max(1, 8e6 // points))
    members = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    case = dict(order=order, nc=nc, scheme=scheme, precision=precision, members=members)
    if precision == "mixed":
        case.update(steps=rng.randint(2, 6 if scheme == "RK3_TVD" else 4), call="height")
        if nc <= 128 and rng.random() < 0.25:
            case.update(members=1, call="group", others=",".join(str(rng.randint(24, 128)) for _ in range(rng.randint(1, 3))))
    elif nc <= 64 and members == 1 and rng.random() < 0.3:
        case.update(steps=1, call="drop_in")
    else:
        case.update(steps=rng.randint(4, 24 if nc <= 192 else 8), call="state" if nc <= 192 else "cells")
    case["flow"] = rng.choice(("smooth", "mountain", "rough" if nc >= 128 else "smooth", "ensemble"))
    return case


# ---------------------------------------------------------------- the inputs, from the case and the seed
def _grids(case):
    return [case["nc"]] + [int(x) for x in case.get("others", "").split(",") if x]


def _specs(case, seed):
    """For each grid the seeded flows of its members."""
    rng = np.random.default_rng([seed, case["order"], case["nc"], case["members"]])
    out = []
    for _ in _grids(case):
        flows = []
        for _ in range(case["members"]):
            u0, alpha, lmax, rms = 38.6, 0.05, 8, 10.0
            if case["flow"] == "rough":
                lmax, rms = 32, 20.0
            if case["flow"] == "ensemble":
                u0, alpha, lmax, rms = rng.uniform(20.0, 40.0), rng.uniform(0.0, math.pi / 2), 16, rng.uniform(5.0, 30.0)
            coef = rng.standard_normal((lmax + 1) ** 2)
            coef[0] = 0.0
            spec = dict(gh0=MEAN_PHI + (RADIUS * OMEGA * u0 + 0.5 * u0 * u0) / 3.0, u0=u0, alpha=alpha, lmax=lmax,
                        rms=rms, coef=coef, mountain=None)
            if case["flow"] in ("rough", "mountain"):
                spec["mountain"] = dict(h0=2000.0, efold=1.0e6, lon=rng.uniform(0.0, 2 * math.pi),
                                        lat=math.asin(rng.uniform(-1.0, 1.0) * math.sin(math.radians(20.0))))
            flows.append(spec)
        out.append(flows)
    return out


def _dt(order, nc):
    """CFL 0.45 on the spacing of the points with the fastest signal of a 40 m/s jet anywhere on the
    panel (a corner: sqrt(G^ii) is 1/R at most, each direction's gravity wave and wind summed)."""
    speed = 2.0 * (math.sqrt(1.45 * MEAN_PHI) + 45.0) / RADIUS
    return round(0.45 * (math.pi / 2 / nc / (order - 1)) / speed, 3)


class _State:
    pass


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def prepare(case, seed):
    st = _State()
    st.case, st.steppers, st.group = case, [], None
    for nc, flows in zip(_grids(case), _specs(case, seed)):
        s = api.Stepper(case["order"], nc, _dt(case["order"], nc), case["scheme"], case["members"], case["precision"],
                        RADIUS)
        s.set_geometry_equiangular()
        for m, spec in enumerate(flows):
            s.set_member_balanced_flow(m, spec)
        st.steppers.append(s)
    if case["call"] == "group":
        # a group runs one persistent tile form: the first handle's own choice where it is one
        forms, chosen = st.steppers[0].tuning()
        if not forms[chosen][0][5]:
            chosen = max(k for k, (shape, _) in enumerate(forms) if shape[5])
        st.group = api.Group(st.steppers, chosen)
    names = {"drop_in": ("u", "v", "phi"), "state": ("u", "v", "phi"), "cells": ("uC", "vC", "phiC")}
    st.names = names.get(case["call"], ("phiC",))
    st.out = []
    for s in st.steppers:
        shape = (6, s.npx, s.npx) if st.names[0] == "u" else (6, s.nc + 2, s.nc + 2)
        st.out += [{k: _pinned(shape) for k in st.names} for _ in range(s.members)]
    if case["call"] == "drop_in":
        st.start = {k: _pinned(st.out[0][k].shape) for k in st.names}
        st.steppers[0].get_state(0, st.start)
    return st


def _history(s, m, out):
    """The cell averages asked for, into the caller's arrays."""
    names = ("u", "v", "phi", "zonal", "merid", "uC", "vC", "phiC")
    args = [api._dp(out[k]) if k in out else None for k in names]
    if api.lib().mcv_get_history(s.h, m, *args) != 0:
        raise RuntimeError(api.lib().mcv_last_error().decode())


def run(st):
    case = st.case
    if case["call"] == "drop_in":
        s = st.steppers[0]
        s.set_state(0, st.start["u"], st.start["v"], st.start["phi"])
        s.step(case["steps"])
        s.get_state(0, st.out[0])
    elif st.group is not None:
        st.group.step(case["steps"])
    else:
        st.steppers[0].step(case["steps"])
    if case["call"] != "drop_in":
        k = 0
        for s in st.steppers:
            for m in range(s.members):
                if case["call"] == "state":
                    s.get_state(m, st.out[k])
                else:
                    _history(s, m, st.out[k])
                k += 1
    if st.names[0] != "u":
        return st.out if len(st.out[0]) > 1 else [o["phiC"] for o in st.out]
    # the prognostic points: beyond them lie the halo and its corners, which hold a fill value of 1e16
    h = st.steppers[0].H
    return [{k: v[:, h:-h, h:-h] for k, v in o.items()} for o in st.out]


def work(case):
    """Per stage and point: the stage's input (3 fields), its base where it is another field, the six
    metric scalars in full precision, the new state, the RK4 sum; split precision holds increments and
    the surface height in 32 bits and forms the metric from tables.  The result is read once more."""
    rk3 = case["scheme"] == "RK3_TVD"
    if case["precision"] == "fp64":
        stage = 8 * sum((12, 15, 15) if rk3 else (15, 21, 21, 18))
    else:
        stage = sum((40, 52, 64) if rk3 else (52, 76, 76, 76))
    points = sum(6 * (nc * (case["order"] - 1) + 1) ** 2 for nc in _grids(case)) * case["members"]
    fields = 3 if case["call"] in ("drop_in", "state", "cells") else 1
    copies = 8 * (fields + (3 if case["call"] == "drop_in" else 0))
    per_stage = {3: 105, 4: 120}[case["order"]]  # the operator's additions and multiplications at a point
    n = STAGES[case["scheme"]]
    return {"bytes": points * (case["steps"] * stage + copies), "flops": points * case["steps"] * n * per_stage}


# ---------------------------------------------------------------- 64-bit model in plain torch
# (panel, edge) -> neighbour panel, its edge, reversed; edges W E S N
_LINKS = [[(3, 1, 0), (1, 0, 0), (5, 3, 0), (4, 2, 0)], [(0, 1, 0), (2, 0, 0), (5, 1, 1), (4, 1, 0)],
          [(1, 1, 0), (3, 0, 0), (5, 2, 1), (4, 3, 1)], [(2, 1, 0), (0, 0, 0), (5, 0, 0), (4, 0, 1)],
          [(3, 3, 1), (1, 3, 0), (0, 3, 0), (2, 3, 1)], [(3, 2, 0), (1, 2, 1), (2, 2, 1), (0, 2, 0)]]
# the (panel, corner) triples that meet at the eight vertices; corners SW SE NW NE
_VERTICES = [[(0, 2), (3, 3), (4, 0)], [(0, 3), (1, 2), (4, 1)], [(0, 0), (3, 1), (5, 2)], [(0, 1), (1, 0), (5, 3)],
             [(2, 2), (1, 3), (4, 3)], [(2, 3), (3, 2), (4, 2)], [(1, 1), (2, 0), (5, 1)], [(2, 1), (3, 0), (5, 0)]]


def _sphere(panel, x, y):
    """Longitude and latitude of panel coordinates (tensors of one shape; panel a tensor of 0..5)."""
    a, b = torch.tan(x), torch.tan(y)
    r = torch.sqrt(a * a + b * b)
    side = panel < 4
    top = panel == 4
    lon = torch.where(side, x + panel * (math.pi / 2), torch.atan2(a, torch.where(top, -b, b)))
    lat = torch.where(side, torch.atan(b * torch.cos(x)), torch.where(top, 1.0, -1.0) * torch.atan2(torch.ones_like(r), r))
    return lon, lat


def _metric(x, y):
    """sqrt(G), the inverse metric and the metric at panel coordinates."""
    tx, ty = torch.tan(x), torch.tan(y)
    cx2, cy2 = torch.cos(x) ** 2, torch.cos(y) ** 2
    rho2 = 1 + tx * tx + ty * ty
    sg = RADIUS ** 2 / (cx2 * cy2 * rho2 * torch.sqrt(rho2))
    k = rho2 * cx2 * cy2 / RADIUS ** 2
    inv = (k * (1 + ty * ty), k * tx * ty, k * (1 + tx * tx))
    g = RADIUS ** 2 / (rho2 * rho2 * cx2 * cy2)
    return sg, inv, (g * (1 + tx * tx), -g * tx * ty, g * (1 + ty * ty))


def _rotations(panel, x, y):
    """A IG (covariant to sphere winds) and G IA (back), row major, from the panel's tangent vectors:
    with e1, e2 their zonal and meridional parts, A = [e1 e2] takes contravariant to sphere winds."""
    lon, lat = _sphere(panel, x, y)
    # Cartesian position on the unit sphere and its derivatives along x and y
    tx, ty = torch.tan(x), torch.tan(y)
    sx, sy = 1 + tx * tx, 1 + ty * ty
    rho2 = 1 + tx * tx + ty * ty
    r1, r3 = 1 / torch.sqrt(rho2), 1 / (rho2 * torch.sqrt(rho2))
    one, zero = torch.ones_like(tx), torch.zeros_like(tx)
    p3 = (one, tx, ty)
    d1 = [r1 * v - r3 * tx * sx * q for v, q in zip((zero, sx, zero), p3)]
    d2 = [r1 * v - r3 * ty * sy * q for v, q in zip((zero, zero, sy), p3)]

    def turned(v):
        # panel 0 has the axes (1, tan x, tan y); the others are turned onto the cube
        a, b, c = v
        th = panel * (math.pi / 2)
        cs, sn = torch.cos(th), torch.sin(th)
        side = (a * cs - b * sn, a * sn + b * cs, c)
        top, bottom = (-c, b, a), (c, b, -a)
        return [torch.where(panel < 4, s, torch.where(panel == 4, t, w)) for s, t, w in zip(side, top, bottom)]

    east = (-torch.sin(lon), torch.cos(lon), zero)
    north = (-torch.sin(lat) * torch.cos(lon), -torch.sin(lat) * torch.sin(lon), torch.cos(lat))
    dot = lambda u, v: RADIUS * sum(p * q for p, q in zip(u, v))  # noqa: E731
    e1, e2 = turned(d1), turned(d2)
    a = (dot(e1, east), dot(e2, east), dot(e1, north), dot(e2, north))
    _, (i11, i12, i22), (g11, g12, g22) = _metric(x, y)
    det = a[0] * a[3] - a[1] * a[2]
    ia = (a[3] / det, -a[1] / det, -a[2] / det, a[0] / det)
    to = (a[0] * i11 + a[1] * i12, a[0] * i12 + a[1] * i22, a[2] * i11 + a[3] * i12, a[2] * i12 + a[3] * i22)
    back = (g11 * ia[0] + g12 * ia[2], g11 * ia[1] + g12 * ia[3], g12 * ia[0] + g22 * ia[2], g12 * ia[1] + g22 * ia[3])
    return to, back


class _Model:
    def __init__(self, order, nc, dev):
        D, H = order, order - 1
        self.D, self.H, self.nc, self.dev = D, H, nc, dev
        self.n, self.np_ = nc * H + 1, nc * H + 1 + 2 * H
        n, np_ = self.n, self.np_
        self.dx = math.pi / 2 / nc
        self.c = (torch.arange(np_, dtype=torch.float64, device=dev) - H) * (self.dx / H) - math.pi / 4
        x, y = self.c.view(1, 1, -1), self.c.view(1, -1, 1)
        self.panel = torch.arange(6, dtype=torch.float64, device=dev).view(6, 1, 1)
        sg, inv, _ = _metric(x, y)
        self.sg, (self.i11, self.i12, self.i22) = sg, inv
        self.f = torch.stack([2 * OMEGA * torch.sin(_sphere(self.panel[p], x[0], y[0])[1]) for p in range(6)])
        # strips: 24 edges, inside lines 0..H and outside lines 0..H, n positions
        k = torch.arange(n, device=dev)
        lines = torch.arange(H + 1, device=dev).view(-1, 1)

        def point(e, d):
            full = (H + 1, n)
            a, b = (k.view(1, -1).expand(full), d.expand(full))
            i, j = ((b, a), (n - 1 - b, a), (a, b), (a, n - 1 - b))[e]
            return i + H, j + H

        src, dst, own, to_src, to_own, back = [], [], [], [], [], []
        for p in range(6):
            for e in range(4):
                q, e2, rev = _LINKS[p][e]
                for panel, edge, d, turn, idx, rot in ((q, e2, lines, rev, src, to_src), (p, e, lines, 0, own, to_own),
                                                       (p, e, -lines, 0, dst, back)):
                    i, j = point(edge, d)
                    if turn:
                        i, j = i.flip(-1), j.flip(-1)
                    idx.append((panel * np_ + j) * np_ + i)
                    r = _rotations(torch.full_like(self.c[i], float(panel)), self.c[i], self.c[j])
                    rot.append(torch.stack(r[1] if rot is back else r[0]))
        self.src, self.dst, self.own = (torch.stack(v) for v in (src, dst, own))  # [24, H+1, n]
        self.to_src, self.to_own, self.back = (torch.stack(v, 1) for v in (to_src, to_own, back))  # [4, 24, H+1, n]
        corner = lambda c: (0 if c in (0, 2) else 1, 0 if c < 2 else n - 1)  # noqa: E731 (edge W or E, position)
        self.vert = torch.tensor([[(p * 4 + corner(c)[0], corner(c)[1]) for p, c in v] for v in _VERTICES], device=dev)
        # halo line h of a panel lies on the neighbour's line h, at other positions along it
        xs = self.c[H:H + n]
        start, frac = [], []
        for h in range(1, H + 1):
            lon, lat = _sphere(torch.zeros_like(xs), xs, torch.full_like(xs, math.pi / 4 + h * self.dx / H))
            X = torch.atan(torch.sin(lon) / torch.tan(lat))
            cell = torch.clamp(torch.floor((X + math.pi / 4) / self.dx), 0, nc - 1)
            start.append(cell.long() * H)
            frac.append(X - (-math.pi / 4 + cell * self.dx))
        self.start, self.frac = torch.stack(start), torch.stack(frac)  # [H, n]

    # ---- initial state on all padded points
    def flow(self, spec):
        lon, lat = (torch.stack(v) for v in zip(*[_sphere(self.panel[p], self.c.view(1, -1), self.c.view(-1, 1))
                                                  for p in range(6)]))
        u0, al = spec["u0"], spec["alpha"]
        zonal = u0 * (torch.cos(lat) * math.cos(al) + torch.cos(lon) * torch.sin(lat) * math.sin(al))
        merid = -u0 * torch.sin(lon) * math.sin(al)
        s = -torch.cos(lon) * torch.cos(lat) * math.sin(al) + torch.sin(lat) * math.cos(al)
        phi = spec["gh0"] - (RADIUS * OMEGA * u0 + u0 * u0 / 2) * s * s
        L, c = spec["lmax"], spec["coef"]
        height = torch.zeros_like(phi)
        x, cl = torch.sin(lat), torch.cos(lat)
        pmm = torch.full_like(x, math.sqrt(0.5))  # normalised Legendre functions, upwards in the degree
        for m in range(L + 1):
            if m:
                pmm = -math.sqrt((2 * m + 1) / (2 * m)) * cl * pmm
            cm, sm = torch.cos(m * lon), torch.sin(m * lon)
            p1, p0 = pmm, torch.zeros_like(pmm)
            for l in range(m, L + 1):
                if l > m:
                    a = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
                    b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4 * (l - 1.0) ** 2 - 1)) if l > m + 1 else 0.0
                    p1, p0 = a * (x * p1 - b * p0), p1
                if l and m:
                    height += p1 * (c[l * l + l + m] * cm + c[l * l + l - m] * sm) / math.sqrt(math.pi)
                elif l:
                    height += p1 * c[l * l + l] / math.sqrt(2 * math.pi)
        w1 = torch.tensor([1.0, 4.0, 1.0] if self.D == 3 else [1.0, 3.0, 3.0, 1.0], dtype=torch.float64, device=self.dev)
        line = torch.zeros_like(self.c)
        for cell in range(self.nc):
            line[self.H + cell * self.H:self.H + cell * self.H + self.D] += w1
        w = line.view(1, -1, 1) * line.view(1, 1, -1) * self.sg
        phi += GRAVITY * height * (spec["rms"] / torch.sqrt((w * height * height).sum() / (6 * w.sum())))
        phis = torch.zeros_like(phi)
        if spec["mountain"]:
            t = spec["mountain"]
            ang = math.sin(t["lat"]) * x + math.cos(t["lat"]) * cl * torch.cos(lon - t["lon"])
            d = RADIUS * torch.acos(torch.clamp(ang, -1.0, 1.0))
            phis = GRAVITY * t["h0"] * torch.exp(-(d / t["efold"]) ** 2)
            phi -= phis
        u, v = torch.empty_like(phi), torch.empty_like(phi)
        for p in range(6):
            x, y = self.c.view(1, -1).expand(self.np_, -1), self.c.view(-1, 1).expand(-1, self.np_)
            b = _rotations(torch.full_like(x, float(p)), x, y)[1]
            u[p] = b[0] * zonal[p] + b[1] * merid[p]
            v[p] = b[2] * zonal[p] + b[3] * merid[p]
        return u, v, phi, phis

    # ---- one-dimensional reconstruction along the last axis of rows with their halo
    def ends(self, f):
        p = f.unfold(-1, self.D, self.H).unbind(-1)  # cells -1..nc
        if self.D == 3:
            return p, (-3 * p[0] + 4 * p[1] - p[2]) / self.dx, (p[0] - 4 * p[1] + 3 * p[2]) / self.dx
        return (p, (-11 * p[0] + 18 * p[1] - 9 * p[2] + 2 * p[3]) / (2 * self.dx),
                (11 * p[3] - 18 * p[2] + 9 * p[1] - 2 * p[0]) / (2 * self.dx))

    def slope(self, f, q, lam):
        """d f / dx at the points of the panel, Riemann fluxes between the cells."""
        p, fl, fr = self.ends(f)
        _, ql, qr = self.ends(q)
        face = 0.5 * ((fr[..., :-1] + fl[..., 1:]) - lam * (ql[..., 1:] - qr[..., :-1]))
        a, b = face[..., :-1], face[..., 1:]
        p = [v[..., 1:-1] for v in p]
        via = (p[-1] - p[0]) / self.dx
        if self.D == 3:
            inner = [1.5 * via - 0.25 * (a + b)]
        else:
            k = 2 / 3 * (p[0] - p[1] - p[2] + p[3]) / self.dx
            inner = [4 / 3 * via - (4 * a + 5 * b) / 27 - k, 4 / 3 * via - (5 * a + 4 * b) / 27 + k]
        out = torch.stack([a] + inner, -1).flatten(-2)
        return torch.cat([out, face[..., -1:]], -1)

    def tendency(self, u, v, phi, phis):
        H, n = self.H, self.n
        inner = slice(H, H + n)
        cu, cv = self.i11 * u + self.i12 * v, self.i12 * u + self.i22 * v
        pg = phi * self.sg
        E = phi + phis + 0.5 * (cu * u + cv * v)

        def sweep(flip, c, g, wind, other):
            pick = (lambda a: a.transpose(-1, -2)) if flip else (lambda a: a)
            rows = lambda a: pick(a)[..., inner, :]  # noqa: E731
            face = lambda a: pick(a)[..., inner, inner][..., ::H]  # noqa: E731
            lam = face(c).abs() + torch.sqrt(face(g.expand_as(phi)) * face(phi))
            sign = torch.where(face(c) < 0, -1.0, 1.0)
            return [pick(self.slope(rows(a), rows(b), s)) for a, b, s in
                    ((E, wind, lam), (pg * c, pg, lam), (other, other, sign))]

        ex, dx, vx = sweep(False, cu, self.i11, u, v)
        ey, dy, uy = sweep(True, cv, self.i22, v, u)
        sg, f, cu, cv = (a[..., inner, inner] for a in (self.sg, self.f, cu, cv))
        vort = vx - uy + sg * f
        return -ex + vort * cv, -ey - vort * cu, -dx - dy

    def complete(self, u, v, phi):
        """Boundary lines averaged over the panels that share them, halo lines from the neighbours."""
        M, D = u.shape[0], self.D
        flat = [a.reshape(M, -1) for a in (u, v, phi)]

        def strip(idx, rot):
            a, b, h = (x[:, idx] for x in flat)
            return rot[0] * a + rot[1] * b, rot[2] * a + rot[3] * b, h

        there, here = strip(self.src, self.to_src), strip(self.own, self.to_own)
        new = []
        H, n = self.H, self.n
        for a, b in zip(there, here):
            edge = 0.5 * (b[:, :, :1] + a[:, :, :1])
            for t in self.vert:
                mean = sum(b[:, s, 0, k] for s, k in t) / 3
                for s, k in t:
                    edge[:, s, 0, k] = mean
            at = self.start.view(1, 1, H, n).expand(M, 24, H, n)
            q = [torch.gather(a[:, :, 1:], -1, at + m) for m in range(D)]
            s = self.frac / self.dx
            if D == 3:
                halo = q[0] + (-3 * q[0] + 4 * q[1] - q[2]) * s + 2 * (q[0] - 2 * q[1] + q[2]) * s * s
            else:
                halo = (q[0] + (-11 * q[0] + 18 * q[1] - 9 * q[2] + 2 * q[3]) * s / 2
                        + 4.5 * (2 * q[0] - 5 * q[1] + 4 * q[2] - q[3]) * s * s
                        + 4.5 * (-q[0] + 3 * q[1] - 3 * q[2] + q[3]) * s ** 3)
            new.append(torch.cat([edge, halo], 2))
        z, m, h = new
        # the ends of the north and south edges are the vertices, which the other two edges hold
        z, m = self.back[0] * z + self.back[1] * m, self.back[2] * z + self.back[3] * m
        keep = torch.ones(24, H + 1, n, dtype=torch.bool, device=self.dev)
        for e in range(24):
            if e % 4 > 1:
                keep[e, 0, 0] = keep[e, 0, -1] = False
        at = self.dst[keep]
        for x, val in zip(flat, (z, m, h)):
            x[:, at] = val[:, keep]
        return [x.reshape(u.shape) for x in flat]

    def step(self, y, phis, dt, scheme):
        inner = (Ellipsis, slice(self.H, self.H + self.n), slice(self.H, self.H + self.n))
        sg = self.sg.expand_as(y[0])[inner]

        def stage(parts, rates):
            """The sum of weighted states (u, v, phiG) and of weighted tendencies, completed."""
            out = []
            for k in range(3):
                w = sg if k == 2 else 1.0
                val = sum(c * s[k][inner] * w for c, s in parts) + sum(c * r[k] for c, r in rates)
                a = parts[-1][1][k].clone()
                a[inner] = val / w
                out.append(a)
            return self.complete(*out)

        L = lambda s: self.tendency(*s, phis)  # noqa: E731
        if scheme == "RK3_TVD":
            y1 = stage([(1.0, y)], [(dt, L(y))])
            y2 = stage([(0.75, y), (0.25, y1)], [(0.25 * dt, L(y1))])
            return stage([(1 / 3, y), (2 / 3, y2)], [(2 / 3 * dt, L(y2))])
        k1 = L(y)
        k2 = L(stage([(1.0, y)], [(dt / 2, k1)]))
        k3 = L(stage([(1.0, y)], [(dt / 2, k2)]))
        k4 = L(stage([(1.0, y)], [(dt, k3)]))
        return stage([(1.0, y)], [(dt / 6, k1), (dt / 3, k2), (dt / 3, k3), (dt / 6, k4)])

    def average(self, f):
        """Weighted sums over the points of each cell, the model's own weights, a ring of zeros around."""
        D, H, n = self.D, self.H, self.n
        w = torch.tensor([1.0, 4.0, 1.0] if D == 3 else [1.0, 3.0, 3.0, 1.0], dtype=torch.float64, device=self.dev)
        cells = f[..., H:H + n, H:H + n].unfold(-1, D, H).unfold(-3, D, H)
        s = (cells * (w.view(-1, 1) * w / (36.0 if D == 3 else 80.0))).sum((-1, -2))
        return torch.nn.functional.pad(s, (1, 1, 1, 1))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for nc, flows in zip(_grids(case), _specs(case, seed)):
        model = _Model(case["order"], nc, dev)
        # members together, as far as the memory of a card goes
        group = max(1, int(4e7) // (6 * model.np_ ** 2))
        for m in range(0, len(flows), group):
            u, v, phi, phis = (torch.stack(a) for a in zip(*[model.flow(s) for s in flows[m:m + group]]))
            y = [u, v, phi]
            for _ in range(case["steps"]):
                y = model.step(y, phis, _dt(case["order"], nc), case["scheme"])
            for one in range(u.shape[0]):
                if case["call"] in ("drop_in", "state"):
                    h = model.H
                    out.append({k: a[one, :, h:-h, h:-h].cpu() for k, a in zip(("u", "v", "phi"), y)})
                elif case["call"] == "cells":
                    out.append({k: model.average(a[one]).cpu() for k, a in zip(("uC", "vC", "phiC"), y)})
                else:
                    out.append(model.average(y[2][one]).cpu())
    return out
