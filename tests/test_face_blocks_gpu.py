"""The face kernel at the node counts where its block size changes (32, 64 and
128 threads) and off their multiples, stepped from both phases: FP64 against
the CPU oracle byte for byte, the other storages against FP64."""
import numpy as np
import pytest

import lbm_b200 as L
from helpers import spheres

pytestmark = pytest.mark.gpu

# (shape, pores left in each x face): 2 x 12, 2 x 512, 2 x 513, 2 x 1500, 2 x 1501, 2 x 1700 face nodes
SIZES = [((9, 11, 10), 12), ((13, 31, 34), 512), ((13, 31, 34), 513), ((11, 47, 53), 1500), ((11, 47, 53), 1501),
         ((11, 47, 53), 1700)]
PRE, RHO = (1, 1, 0, 0, 0, 0), (0.9995, 1.0005, 1.0, 1.0, 1.0, 1.0)


def case(shape, pores):
    mask = spheres(shape, 0.8, 2.5, seed=4).copy()
    rng = np.random.default_rng(3)
    for face in (0, -1):
        plane = np.ones(mask[:, :, face].size, dtype=np.uint8)
        plane[rng.permutation(plane.size)[:pores]] = 0
        mask[:, :, face] = plane.reshape(mask[:, :, face].shape)
    return mask


def run(mask, precision, steps):
    with L.SinglePhase(mask, 0.1, (0.0, 0.0, 0.0), precision=precision,
                       bc=dict(sub_bc=0, in_bc=1, pressure=PRE, rho=RHO)) as s:
        for n in steps:
            s.step(n)
        return s.populations(), *s.fields()


@pytest.mark.parametrize("shape,pores", SIZES)
def test_faces_at_the_block_sizes(oracle_mod, shape, pores):
    mask = case(shape, pores)
    ref = oracle_mod.SinglePhaseRun(mask, 0.1, (0.0, 0.0, 0.0), bc=oracle_mod.Boundaries(in_bc=1, pre=PRE, p=RHO))
    ref.step(7)
    f_ref, u_ref, rho_ref = ref.fields()
    f, rho, u = run(mask, "f64", (1, 2, 4))
    assert np.array_equal(f[1:], f_ref[1:]) and np.array_equal(u[1:], u_ref[1:]) and np.array_equal(rho[1:], rho_ref[1:])
    for precision, bar in (("f64fast", 1e-10), ("f32", 1e-4), ("f16", 2e-2)):
        _, _, v = run(mask, precision, (1, 2, 4))
        assert np.abs(v - u).max() <= bar * np.abs(u).max()
