"""The single-domain FP32 step's own rounding over hundreds of steps with a
force along all axes, without and with faces: md5 of the populations after 34 (22
with a restored state) steps, the step the stop test ends on, md5 of u there."""
import hashlib

import numpy as np
import pytest

import lbm_b200 as L
from helpers import spheres

pytestmark = pytest.mark.gpu

PRESSURE = dict(sub_bc=0, in_bc=1, pressure=(1, 1, 0, 0, 0, 0), rho=(0.9995, 1.0005, 1, 1, 1, 1))
INLET = dict(sub_bc=1, in_bc=1, pressure=(0, 1, 0, 0, 0, 0), rho=(1, 1.0005, 1, 1, 1, 1), velocity=(1, 0, 0, 0, 0, 0),
             vel=(1e-4, 0, 0, 0, 0, 0))


def md5(a):
    return hashlib.md5(np.ascontiguousarray(a).tobytes()).hexdigest()[:10]


@pytest.mark.parametrize("bc,g,pops,steps,u", [
    (PRESSURE, (1e-6, 2e-7, 0.0), "b5c87d1c80", 534, "99754f9e39"),
    (INLET, (1e-6, 2e-7, 0.0), "c85fc75073", 454, "df4ba7438f"),
    (None, (1e-6, 2e-7, 3e-7), "68968bb283", 562, "33fdc35cc4")])
def test_flow_rounding(bc, g, pops, steps, u):
    mask = spheres((41, 37, 33), 0.6, 4.0, seed=7)
    with L.SinglePhase(mask, 0.1, g, precision="f32", bc=bc) as s:
        if bc is None:
            s.step(13)
            f, (rho, v) = s.populations(), s.fields()
            s.set_state(rho, v, f)
            s.step(9)
        else:
            for n in (1, 1, 2, 30):
                s.step(n)
        assert md5(s.populations()) == pops
        d = s.run_to_convergence(tol=1e-5, check_every=20, max_steps=1500)
        assert (d["step"], md5(s.fields()[1])) == (steps, u)
