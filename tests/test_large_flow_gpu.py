"""Single-phase steps at the sizes where their paths combine: two nodes per
thread beside the face kernel, and captured chains of dependent launches over
the row table with the L2 prefetch."""
import numpy as np
import pytest

import lbm_b200 as L
from helpers import spheres

pytestmark = pytest.mark.gpu

FACES = dict(sub_bc=0, in_bc=1, pressure=(1, 1, 0, 0, 0, 0), rho=(0.9995, 1.0005, 1, 1, 1, 1))


# The nodes between the x faces are the step kernel's; with an odd count the
# last pair of a step on the nodes' own slots has no second node: that slot is
# the face kernel's, which runs beside it.
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("precision,bar", [("f32", 1e-4), ("f16", 2e-2)])
def test_faces_with_two_nodes_per_thread(precision, bar, odd):
    mask = spheres((69, 64, 61), 0.68, 4.0, seed=12).copy()
    main = int((mask[:, :, 1:-1] == 0).sum())
    if main % 2 != odd:
        mask[tuple(np.argwhere(mask[:, :, 1:-1] == 0)[main // 2] + (0, 0, 1))] = 1
        main -= 1
    assert main % 2 == odd and main >= 148 * 1024

    def run(precision, compact):
        with L.SinglePhase(mask, 0.1, precision=precision, bc=FACES) as s:
            s.set_table_mode(compact)  # compact: one node per thread through the table
            for n in (1, 2, 18):
                s.step(n)
            return s.populations(), *s.fields()

    got = run(precision, 0)
    for a, b in zip(got, run(precision, 1)):
        assert np.array_equal(a, b)
    _, _, u64 = run("f64", 0)
    assert np.abs(got[2] - u64).max() <= bar * np.abs(u64).max()
