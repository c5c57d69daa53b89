"""The flag a stage kernel raises when its staged copies do not arrive, raised
here from the device by the library's own hook: a step and the autotuner's
trials report it, and setting the geometry again, either way, clears it."""
import ctypes

import numpy as np
import pytest

from mcv_sw_b200 import api, cases

pytestmark = pytest.mark.gpu


def raise_flag(s):
    f = api.lib().mcv_selftest_late
    f.argtypes, f.restype = [ctypes.c_void_p], ctypes.c_int
    assert f(s.h) == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("device", [False, True])
def test_late_copies_until_the_geometry_is_set_again(precision, device):
    geom = api.Geometry(3, 40, cases.EARTH_RADIUS)  # a grid on which several forms are timed
    st, _ = cases.small(seed=2, nc=40, geom=geom)

    def start(s):
        if device:
            s.set_geometry_equiangular()
        else:
            s.set_geometry(geom)
        s.set_member(0, st.phi_s, st.u, st.v, st.phi)

    with api.Stepper(3, 40, st.dt, "RK4", precision=precision, radius=cases.EARTH_RADIUS) as s:
        start(s)
        s.step(2)
        raise_flag(s)
        for _ in range(2):
            with pytest.raises(api.MCVError) as e:
                s.step(1)
            assert "did not arrive in time" in str(e.value)
        start(s)
        s.step(2)
        assert all(np.isfinite(x[:, geom.H:-geom.H, geom.H:-geom.H]).all() for x in s.get_state(0).values())
        # before the first step: the trials see it
        s.select_tile(-1)
        raise_flag(s)
        with pytest.raises(api.MCVError) as e:
            s.tuning()
        assert "did not arrive in time" in str(e.value)
        start(s)
        cands, chosen = s.tuning()
        assert 0 <= chosen < len(cands)
        s.step(1)
