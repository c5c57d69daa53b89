"""Groups on every persistent form, and on strip cuts that a group of small grids
does not reach: each handle ends bit for bit where it ends alone on the same form.
And one handle whose strips are cut into runs that end inside a column, against
the CPU oracle (tests/test_strip_gpu.py's bounds).  Which cut a launch takes is
checked on the host (tests/test_cut.py), where these sizes come from."""
import numpy as np
import pytest

from mcv_sw_b200 import api, cases
from tests.helpers import oracle_for
from tests.test_strip_gpu import STEPS, check, problem, stepper

pytestmark = pytest.mark.gpu


def make(order, precision, scheme, grids, tile):
    out = []
    for k, (nc, members) in enumerate(grids):
        s = api.Stepper(order, nc, 0.2 * 2.0e4 / nc / (order - 1), scheme, members, precision, cases.EARTH_RADIUS)
        s.set_geometry_equiangular()
        for m in range(members):
            s.set_member_balanced_flow(m, cases.balanced_flow_spec(s, np.random.default_rng([k, m])))
        s.select_tile(tile)
        out.append(s)
    return out


def compare_group(order, precision, scheme, grids, tile):
    alone = make(order, precision, scheme, grids, tile)
    together = make(order, precision, scheme, grids, tile)
    for s in alone:
        s.step(3)
    with api.Group(together, tile) as g:
        g.step(3)
    for a, b in zip(alone, together):
        for m in range(a.members):
            x, y = a.get_state(m), b.get_state(m)
            for f in ("u", "v", "phi"):
                assert np.array_equal(x[f], y[f]), (tile, a.nc, m, f)
        a.close()
        b.close()


def persistent_forms(order, precision):
    (s,) = make(order, precision, "RK4", [(8, 1)], -1)
    forms = [i for i, (shape, _) in enumerate(s.tuning()[0]) if shape[5]]
    s.close()
    return forms


@pytest.mark.parametrize("scheme", ["RK3_TVD", "RK4"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [3, 4])
def test_every_persistent_form(order, precision, scheme):
    forms = persistent_forms(order, precision)
    assert len(forms) >= 2
    for tile in forms:
        compare_group(order, precision, scheme, [(10, 1), (17, 2), (24, 3), (33, 1)], tile)


# runs that go from one grid's columns into the next's; then segments, several to a warp
@pytest.mark.parametrize("order,precision,grids", [
    (3, "fp64", [(25, 12), (15, 29), (10, 29)]), (4, "fp64", [(10, 20), (17, 15), (24, 10)]),
    (3, "mixed", [(28, 3), (31, 12), (32, 8)]), (4, "mixed", [(10, 40), (17, 30), (24, 20)]),
    (4, "mixed", [(24, 16), (31, 10), (45, 6)]),
    (3, "fp64", [(9, 60), (16, 40), (25, 20)]), (4, "fp64", [(10, 40), (17, 30), (24, 20)])])
@pytest.mark.parametrize("scheme", ["RK3_TVD", "RK4"])
def test_strip_cuts_over_several_grids(order, precision, grids, scheme):
    compare_group(order, precision, scheme, grids, persistent_forms(order, precision)[-1])


@pytest.mark.parametrize("nc,precision", [(134, "fp64"), (162, "mixed"), (170, "mixed")])
@pytest.mark.parametrize("scheme", ["RK3_TVD", "RK4"])
def test_runs_that_end_inside_a_column(nc, precision, scheme):
    geom, st = problem(4, nc, scheme)
    o = oracle_for(st)
    o.step(STEPS)
    with stepper(geom, st, 1, precision) as s:
        s.select_tile(len(s.tuning()[0]) - 1)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)
        s.step(STEPS)
        check(geom, st, o, s.get_state(0), precision, nc)
