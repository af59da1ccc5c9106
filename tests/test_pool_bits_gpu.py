"""The pool's own rounding, step for step: the stop test of a 16-bit solve is
decided by noise of the last bits, so the steps to convergence and the
permeabilities below are those of the pool's arithmetic and of no other."""
import numpy as np
import pytest

import lbm_b200 as L
from helpers import spheres

pytestmark = pytest.mark.gpu

# precision, tol, check_every -> steps of the six solves, first permeabilities, sum |u| of the first and the last
WANT = [
    ("f16", 1e-4, 50, [250, 300, 300, 400, 300, 250], ["0x1.32e1720000000p-2", "0x1.f309940000000p-3"],
     ["0x1.1f17151dbba6bp-4", "0x1.5aae67503d8dap-1"]),
    ("f16", 1e-5, 100, [600, 800, 400, 800, 500, 500], ["0x1.32e6560000000p-2", "0x1.f310ec0000000p-3"],
     ["0x1.1f1c4b5604da9p-4", "0x1.5aac06ff4ec0cp-1"]),
    ("f32", 1e-5, 50, [300, 350, 350, 450, 400, 300], ["0x1.32f08c0000000p-2", "0x1.f317280000000p-3"],
     ["0x1.1f26cbde133e3p-4", "0x1.5aac737cb715dp-1"]),
    ("f32", 1e-4, 50, [250, 300, 250, 400, 350, 250], ["0x1.32f08c0000000p-2", "0x1.f3171c0000000p-3"],
     ["0x1.1f26a1b70bfb6p-4", "0x1.5aaeb89b33654p-1"]),
]


@pytest.mark.parametrize("precision,tol,check,steps,perm,speed", WANT)
def test_pool_rounding(precision, tol, check, steps, perm, speed):
    masks = [spheres((e, e + 3, e - 2), 0.45, 4.0, seed=e) for e in (24, 29, 33, 38, 44, 51)]
    with L.Batch([(m, 0.1, (1e-6, 0.0, 0.0)) for m in masks], precision=precision) as b:
        r = b.run(tol=tol, check_every=check, max_steps=1500)
        assert [x["steps"] for x in r] == steps
        assert [float(np.float32(x["perm"][0])).hex() for x in r[:2]] == perm
        got = [float(np.abs(b.fields(i)[1]).sum()) for i in (0, 5)]
        assert np.allclose(got, [float.fromhex(s) for s in speed], rtol=1e-13, atol=0)  # the host's sum order
