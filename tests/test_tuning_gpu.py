"""What the autotuner tries: few forms on one grid, so that a new handle's first
step does not pay for those that cannot win there; the one it takes among them (or
the only one, untimed); in split precision a persistent form wherever a direct tile
is taken, which groups fall back on.  And the default choice against the oracle
(FP64, relative L2 <= 1e-12) on both sides of the lines between forms."""
import numpy as np
import pytest

from mcv_sw_b200 import api, cases
from tests.helpers import oracle_for
from tests.test_parity_gpu import TOL, compare

pytestmark = pytest.mark.gpu


def tuned(order, nc, members, precision):
    s = api.Stepper(order, nc, 10.0, "RK4", members, precision, cases.EARTH_RADIUS)
    s.set_geometry_equiangular()
    for m in range(members):
        s.set_member_balanced_flow(m, cases.balanced_flow_spec(s, np.random.default_rng(m)))
    forms, chosen = s.tuning()
    timed = [i for i, (_, ms) in enumerate(forms) if ms >= 0]
    return s, forms, chosen, timed


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [3, 4])
def test_few_forms_are_tried(order, precision):
    sizes = [(nc, 1) for nc in (2, 4, 9, 15, 16, 18, 19, 22, 23, 26, 27, 30, 31, 33, 34, 37, 38, 39, 41, 42, 44, 45, 46,
                                54, 55, 56, 60, 71, 77, 78, 86, 87, 92, 93, 95, 110, 118, 119, 124, 125, 174, 200, 213)]
    sizes += [(8, 8), (13, 16), (16, 16), (20, 12), (32, 8), (47, 2), (48, 4), (64, 8)]
    for nc, members in sizes:
        s, forms, chosen, timed = tuned(order, nc, members, precision)
        assert len(timed) <= 4 and len(timed) != 1, (nc, members, timed)
        assert not timed or min(timed, key=lambda i: forms[i][1]) == chosen, (nc, members)
        if precision == "mixed":
            assert forms[chosen][0][5] or any(forms[i][0][5] for i in timed), (nc, members)
        s.close()


@pytest.mark.parametrize("order", [3, 4])
def test_many_members_of_a_tiny_grid_try_all(order):
    s, forms, chosen, timed = tuned(order, 9, 40, "fp64")
    assert len(timed) == len(forms)
    s.close()


@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("nc", [15, 27, 38, 39, 55, 86, 95])
def test_the_default_choice(order, nc):
    geom = api.Geometry(order, nc, cases.EARTH_RADIUS)
    st = cases.finish(geom, *cases.balanced_flow(geom, np.random.default_rng(nc))[:4], "RK4", nsteps=2)
    o = oracle_for(st)
    o.step(2)
    with api.Stepper(order, nc, st.dt, "RK4", radius=cases.EARTH_RADIUS) as s:
        s.set_geometry(geom)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)
        s.step(2)
        errs = compare(geom, o, s.get_state(0))
        assert max(errs.values()) <= TOL, errs
