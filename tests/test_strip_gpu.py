"""The stage kernel's strip form (the last candidate) and its small tiles at the
sizes where their cuts can go wrong, and state transfers on both sides of the
line between three staging fields and one.

FP64 against the CPU oracle: relative L2 <= 1e-12, the parity tests' bound.
Split precision against FP64: a stage rounds its tendencies to FP32 after
differencing in FP64, some sixteen roundings of 2^-24 of an increment that is
at most (1 + 2 Omega dt) of the field, in each of the 12 stages of 3 RK4 steps.
"""
import numpy as np
import pytest

from mcv_sw_b200 import api, cases
from tests.helpers import interior, oracle_for
from tests.test_parity_gpu import TOL, compare

pytestmark = pytest.mark.gpu

STEPS = 3
OMEGA = 7.292e-5


def problem(order, nc, scheme, seed=23):
    geom = api.Geometry(order, nc, cases.EARTH_RADIUS)
    st = cases.finish(geom, *cases.balanced_flow(geom, np.random.default_rng(seed), mountain=True)[:4], scheme,
                      nsteps=STEPS)
    return geom, st


def stepper(geom, st, members, precision):
    s = api.Stepper(st.order, st.nc, st.dt, st.scheme, members=members, precision=precision,
                    radius=cases.EARTH_RADIUS)
    s.set_geometry(geom)
    for m in range(members):
        s.set_member(m, st.phi_s, st.u, st.v, st.phi)
    return s


def check(geom, st, o, out, precision, what):
    if precision == "fp64":
        errs = compare(geom, o, out)
        assert max(errs.values()) <= TOL, (what, errs)
        return
    bound = 4 * STEPS * 16 * 2.0 ** -24 * (1 + 2 * OMEGA * st.dt)
    for k in ("u", "v", "phi"):
        a, b = interior(out[k], geom.H, geom.n), interior(o.state(k), geom.H, geom.n)
        d = np.abs(a - b).max() / np.abs(b).max()
        assert d <= bound, (what, k, d, bound)


# one cell column and none left over (29, 58), a column of one or two cells more
# (30, 59), runs that end inside a column (61, 91), strips shorter than a warp's
# start (2, 3)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order,nc,scheme", [(3, 2, "RK4"), (4, 2, "RK3_TVD"), (4, 3, "RK4"), (3, 29, "RK3_TVD"),
                                             (4, 29, "RK4"), (3, 30, "RK4"), (4, 30, "RK3_TVD"), (3, 58, "RK3_TVD"),
                                             (3, 59, "RK4"), (4, 61, "RK3_TVD"), (3, 91, "RK4"), (4, 91, "RK4")])
def test_strips_at_their_edges(order, nc, scheme, precision):
    geom, st = problem(order, nc, scheme)
    o = oracle_for(st)
    o.step(STEPS)
    with stepper(geom, st, 1, precision) as s:
        s.select_tile(len(s.tuning()[0]) - 1)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)
        s.step(STEPS)
        check(geom, st, o, s.get_state(0), precision, nc)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order,nc,members", [(3, 9, 310), (4, 5, 200), (3, 31, 40)])
def test_strips_of_many_members(order, nc, members, precision):
    """More strips than warps: segments of two lengths (Nc=9), several passes,
    and an active list that leaves members out and is not in order."""
    geom, st = problem(order, nc, "RK4")
    o = oracle_for(st)
    o.step(STEPS)
    with stepper(geom, st, members, precision) as s:
        s.select_tile(len(s.tuning()[0]) - 1)
        for active in ([*range(members)], [*range(members - 1, 0, -2)]):
            for m in range(members):
                s.set_member(m, st.phi_s, st.u, st.v, st.phi)
            s.set_active(active)
            s.step(STEPS)
            outs = [s.get_state(m) for m in active]
            for m, out in zip(active, outs):
                for k in ("u", "v", "phi"):
                    assert np.array_equal(out[k], outs[0][k]), (m, k)
            check(geom, st, o, outs[0], precision, active[0])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("nc", [2, 3, 5, 9])
def test_every_form_on_tiny_grids(order, nc, precision):
    geom, st = problem(order, nc, "RK4")
    o = oracle_for(st)
    o.step(STEPS)
    with stepper(geom, st, 1, precision) as s:
        cands = s.tuning()[0]
        for i in range(len(cands)):
            s.select_tile(i)
            s.set_member(0, st.phi_s, st.u, st.v, st.phi)
            s.step(STEPS)
            check(geom, st, o, s.get_state(0), precision, cands[i][0])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc", [7, 137, 138])  # a field passes 8 MiB between 137 (418^2 points a panel with halo) and 138
def test_state_round_trip(nc, precision):
    rng = np.random.default_rng(nc)
    with api.Stepper(4, nc, 1.0, "RK4", precision=precision, radius=cases.EARTH_RADIUS) as s:
        s.set_geometry_equiangular()
        a = {k: rng.standard_normal((6, s.npx, s.npx)) for k in ("u", "v", "phi")}
        s.set_member(0, np.zeros_like(a["u"]), a["u"], a["v"], a["phi"])
        b = {k: rng.standard_normal((6, s.npx, s.npx)) for k in ("u", "v", "phi")}
        s.set_state(0, b["u"], b["v"], b["phi"])
        out = s.get_state(0)
        H = s.H
        n = s.npx - 2 * H
        for k in b:
            assert np.array_equal(interior(out[k], H, n), interior(b[k], H, n)), k
