"""The form of a group that names none.  The direct tiles that win on small grids
run one grid only: a split-precision group of such grids takes the fastest
persistent form of its first handle's record, bit for bit what the handles give
alone on it.  A direct tile that the caller has set, and a handle with no record,
are refused."""
import numpy as np
import pytest

from mcv_sw_b200 import api, cases

pytestmark = pytest.mark.gpu


def stepper(order, nc, scheme, seed, precision="mixed"):
    geom = api.Geometry(order, nc, cases.EARTH_RADIUS)
    st = cases.finish(geom, *cases.balanced_flow(geom, np.random.default_rng(seed))[:4], scheme, nsteps=1)
    s = api.Stepper(order, nc, st.dt, scheme, precision=precision, radius=cases.EARTH_RADIUS)
    s.set_geometry(geom)
    s.set_member(0, st.phi_s, st.u, st.v, st.phi)
    return s, st


def same(a, b):
    return all(np.array_equal(a[k], b[k]) for k in ("u", "v", "phi"))


@pytest.mark.parametrize("order,scheme", [(3, "RK4"), (4, "RK3_TVD")])
@pytest.mark.parametrize("sizes", [(4, 6), (32, 24), (48, 32), (96, 17)])
def test_group_of_small_grids(order, scheme, sizes):
    made = [stepper(order, nc, scheme, 3 + k) for k, nc in enumerate(sizes)]
    forms, chosen = made[0][0].tuning()
    timed = {i: ms for i, (shape, ms) in enumerate(forms) if shape[5] and ms >= 0}
    form = chosen if forms[chosen][0][5] else min(timed, key=timed.get)
    with api.Group([s for s, _ in made]) as g:
        g.step(3)
    for s, st in made:
        together = s.get_state(0)
        s.select_tile(form)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)
        s.step(3)
        assert same(together, s.get_state(0)), (s.nc, form)
        s.close()


def test_a_direct_tile_of_the_caller_is_refused():
    made = [stepper(4, nc, "RK4", nc)[0] for nc in (8, 12)]
    forms, _ = made[0].tuning()
    made[0].select_tile(min(i for i, (shape, _) in enumerate(forms) if not shape[5]))
    with pytest.raises(api.MCVError):
        api.Group(made)
    for s in made:
        s.close()


def test_a_handle_without_a_record_is_refused():
    made = [stepper(4, nc, "RK4", nc)[0] for nc in (8, 12)]
    with pytest.raises(api.MCVError):
        api.Group(made)
    for s in made:
        s.close()


def test_a_group_steps_handles_that_were_never_tuned():
    """Their own trials come with their own first step; a later group that names
    no form asks its first handle for them."""
    made = [stepper(4, nc, "RK4", nc) for nc in (48, 20)]
    forms = stepper(4, 48, "RK4", 48)[0].tuning()[0]
    form = min(i for i, (shape, _) in enumerate(forms) if shape[5])
    with api.Group([s for s, _ in made], form) as g:
        g.step(2)
    together = [s.get_state(0) for s, _ in made]
    with api.Group([s for s, _ in made]) as g:
        g.step(1)
    for (s, st), out in zip(made, together):
        s.select_tile(form)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)
        s.step(2)
        assert same(out, s.get_state(0)), s.nc
        s.close()


def test_a_group_of_handles_that_were_never_tuned_and_rest():
    """No member of the first handle is active, so it has nothing to time."""
    made = [stepper(4, nc, "RK4", nc) for nc in (48, 20)]
    tile = min(i for i, (shape, _) in enumerate(stepper(4, 48, "RK4", 48)[0].tuning()[0]) if shape[5])
    with api.Group([s for s, _ in made], tile) as g:
        g.step(1)
    made[0][0].set_active([])
    rests, steps = [s.get_state(0) for s, _ in made]
    with api.Group([s for s, _ in made]) as g:
        g.step(2)
    assert same(rests, made[0][0].get_state(0)) and not same(steps, made[1][0].get_state(0))
    for s, _ in made:
        s.close()
