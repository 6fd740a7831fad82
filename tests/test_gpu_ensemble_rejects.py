"""An upload that an ensemble refuses leaves the handle as it was."""
from __future__ import annotations

import numpy as np
import pytest

from nbody_b200 import Ensemble, scenarios
from nbody_b200 import _native as N
from nbody_b200.engine import NBodyError

pytestmark = pytest.mark.gpu
EPS = 1e-4


@pytest.mark.parametrize("field", ["px", "vx", "vz", "mass"])
@pytest.mark.parametrize("value", [np.nan, -np.inf])
def test_a_refused_upload_keeps_the_state(field, value):
    """Two handles with the same state, one of which is then given other
    bodies with one non-finite value: error status, and from there on the same
    bits as the handle that saw no such call."""
    sizes = [70, 300, 2100]
    systems = [scenarios.plummer(k, seed=k) for k in sizes]
    bad = [scenarios.plummer(k, seed=k + 1) for k in sizes]
    getattr(bad[1], field)[17] = value
    with Ensemble(sizes, ds_max_n=2048) as a, Ensemble(sizes, ds_max_n=2048) as b:
        for e in (a, b):
            e.set_state(systems)
            e.compute_forces(EPS)
        with pytest.raises(NBodyError) as err:
            a.set_state(bad)
        assert err.value.status == N.NB_ERR_NONFINITE
        for _ in range(2):
            got, want = a.get_state(), b.get_state()
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg=k)
            for e in (a, b):
                e.step(2, 1e-4, EPS)
        a.set_state(systems)
        np.testing.assert_array_equal(a.get_state()["vx"], np.concatenate([s.vx for s in systems]))


def test_a_refused_first_upload_leaves_no_state():
    systems = [scenarios.plummer(k, seed=k) for k in (64, 2100)]
    systems[0].vy[3] = np.nan
    with Ensemble([64, 2100], ds_max_n=2048) as e:
        with pytest.raises(NBodyError):
            e.set_state(systems)
        for call in (lambda: e.step(1, 1e-4, EPS), e.get_state, lambda: e.compute_forces(EPS)):
            with pytest.raises(NBodyError) as err:
                call()
            assert err.value.status == N.NB_ERR_STATE
