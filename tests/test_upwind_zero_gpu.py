"""The upwind side of dudy where the wind is zero: the reference replaces 0 by 1
before it takes c/|c| (src/spatial_operators_mod.F90:83-85), for a zero of either
sign.  Every FP64 form against the CPU oracle on a flow whose contravariant v is
-0.0 on the rows of points between cells, while u jumps between those rows and
the others, so that the two sides' derivatives differ at first order; relative
L2 <= 1e-12, the parity tests' bound."""
import numpy as np
import pytest

from mcv_sw_b200 import api, cases
from oracle.oracle import Oracle
from tests.test_parity_gpu import TOL, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,scheme", [(3, "RK4"), (4, "RK3_TVD")])
@pytest.mark.parametrize("nc", [6, 31])
def test_negative_zero_wind(order, nc, scheme):
    geom = api.Geometry(order, nc, cases.EARTH_RADIUS)
    rng = np.random.default_rng(5)
    st = cases.finish(geom, *cases.balanced_flow(geom, rng)[:4], scheme, nsteps=1)
    g12 = geom.matrixIG[..., 0, 1]
    u = cases.EARTH_RADIUS * rng.uniform(5.0, 15.0, geom.shape)
    rows = np.arange(geom.npx) % geom.H == 0  # padded rows of the points between cells
    u[:, rows, :] = np.copysign(0.0, -g12[:, rows, :])
    v = np.full(geom.shape, -0.0)
    o = Oracle(order, nc, st.dt, scheme, cases.EARTH_RADIUS)
    o.set_phi_s(st.phi_s)
    o.set_state_cov(u, v, st.phi)
    o.step(1)
    with api.Stepper(order, nc, st.dt, scheme, radius=cases.EARTH_RADIUS) as s:
        s.set_geometry(geom)
        s.set_member(0, st.phi_s, u, v, st.phi)
        cands = s.tuning()[0]
        for i, (shape, _) in enumerate(cands):
            s.select_tile(i)
            s.set_member(0, st.phi_s, u, v, st.phi)
            s.step(1)
            errs = compare(geom, o, s.get_state(0))
            assert max(errs.values()) <= TOL, (shape, errs)
