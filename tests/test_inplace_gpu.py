"""In-place streaming on the GPU: both phases of the population array, the
int32 and the row form of the pull table, one and two nodes per thread, at the
sizes where each begins, with odd node counts and periodic wraps."""
import numpy as np
import pytest

import lbm_b200 as L
from helpers import spheres

pytestmark = pytest.mark.gpu

G3 = (1e-5, 4e-6, -3e-6)


def exact_count_mask(shape, pores, seed):
    """A random mask with exactly `pores` pore cells."""
    nx, ny, nz = shape
    mask = np.ones(nx * ny * nz, dtype=np.uint8)
    mask[np.random.default_rng(seed).permutation(mask.size)[:pores]] = 0
    return mask.reshape(nz, ny, nx)


def solve(mask, precision, steps, **kw):
    with L.SinglePhase(mask, 0.1, G3, precision=precision, **kw) as s:
        for n in steps:
            s.step(n)
        return s.populations(), *s.fields()


@pytest.mark.parametrize("precision,bar", [("f64fast", 1e-10), ("f32", 1e-4), ("f16", 2e-2)])
@pytest.mark.parametrize("steps", [(1,), (2,), (3,), (2, 1, 18, 3)])
def test_every_phase_follows_the_bit_exact_kernel(precision, bar, steps):
    """The suite's bars of max |u| against the FP64 kernel, from states of
    both phases and calls that end in either."""
    mask = spheres((37, 29, 31), 0.5, 4.0, seed=5)
    _, _, u64 = solve(mask, "f64", steps)
    _, _, u = solve(mask, precision, steps)
    assert np.abs(u - u64).max() <= bar * np.abs(u64).max()


@pytest.mark.parametrize("first", [1, 2])
def test_state_set_in_either_phase_continues(first):
    mask = spheres((33, 21, 18), 0.55, 3.0, seed=9)
    with L.SinglePhase(mask, 0.1, G3, precision="f64") as a, L.SinglePhase(mask, 0.1, G3, precision="f64") as b:
        a.step(first)
        f, (rho, u) = a.populations(), a.fields()
        b.step(3)  # another phase and another state
        b.set_state(rho, u, f)
        a.step(5)
        b.step(5)
        assert np.array_equal(a.populations(), b.populations())


# the row form is built for solves above 90 MiB of populations and table
# (0.64 M nodes in FP32, 0.42 M in FP64); curve orders read the int32 table
@pytest.mark.parametrize("precision", ["f32", "f64", "f64fast", "f16"])
@pytest.mark.parametrize("shape,phi", [((113, 101, 119), 0.7), ((17, 223, 331), 0.8)])
def test_row_table_gives_the_int32_table_results(precision, shape, phi):
    mask = spheres(shape, phi, 4.5, seed=31)
    want = solve(mask, precision, (7,), ordering="morton")
    for block in (64, 256, 512):
        got = solve(mask, precision, (7,), block_size=block)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


# two nodes per thread from 148 * 1024 nodes on
@pytest.mark.parametrize("pores", [148 * 1024 - 1, 148 * 1024, 148 * 1024 + 1, 148 * 1024 + 33, 148 * 1024 + 255])
@pytest.mark.parametrize("precision", ["f32", "f16"])
def test_two_nodes_per_thread_at_its_first_sizes(pores, precision):
    mask = exact_count_mask((65, 61, 47), pores, seed=pores)
    runs = [solve(mask, precision, (4,), block_size=b) for b in (64, 256, 512)]
    compact = None
    with L.SinglePhase(mask, 0.1, G3, precision=precision) as s:
        s.set_table_mode(1)  # always one node per thread through the table
        s.step(4)
        compact = s.populations(), *s.fields()
    for r in runs:
        for a, b in zip(r, compact):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,bar", [("f32", 1e-4), ("f16", 2e-2)])
@pytest.mark.parametrize("check_every", [7, 8])
def test_pool_steps_in_place(precision, bar, check_every):
    """Chains of odd and even length (the pool's phase after them), tiles with
    odd remainders, against the bit-exact single-domain kernel."""
    masks = [spheres((e, e + 3, e - 2), 0.45, 3.5, seed=e) for e in (12, 23, 40)]
    steps = 3 * check_every
    with L.Batch([(m, 0.1, G3) for m in masks], precision=precision) as b:
        for _ in range(2):
            b.reset()
            res = b.run(tol=1e-30, check_every=check_every, max_steps=steps)
        for i, m in enumerate(masks):
            assert res[i]["steps"] == steps
            _, _, u64 = solve(m, "f64", (steps,))
            _, u = b.fields(i)
            assert np.abs(u - u64).max() <= bar * np.abs(u64).max()


@pytest.mark.parametrize("block", [128, 256, 512])
def test_large_pool_reads_the_row_table(block):
    masks = [spheres((e, e, e + 1), 0.6, 4.0, seed=e) for e in (71, 84)]  # 0.57 M nodes: 1024 tiles or more
    with L.Batch([(m, 0.1, G3) for m in masks] * 2, precision="f32", block=block) as b:
        b.run(tol=1e-30, check_every=5, max_steps=10)
        for i, m in enumerate(masks * 2):
            _, _, u64 = solve(m, "f64", (10,))
            _, u = b.fields(i)
            assert np.abs(u - u64).max() <= 1e-4 * np.abs(u64).max()


@pytest.mark.parametrize("lattice", [7, 19])
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape,phi", [((29, 23, 31), 0.5), ((121, 113, 101), 0.75)])
def test_solute_steps_in_place(lattice, precision, shape, phi):
    """States of both phases, calls of more and fewer steps than a captured
    chain, restored states; the large box reads the row table with 19
    directions.  One call of n steps equals n calls of one, bit for bit."""
    mask = spheres(shape, phi, 4.0, seed=77)
    n = int((mask == 0).sum())
    rng = np.random.default_rng(5)
    u = np.zeros((n + 1, 3))
    u[1:] = rng.uniform(-2e-3, 2e-3, (n, 3))
    c0 = rng.uniform(0.0, 1.0, mask.shape)
    kw = dict(u_nodes=u, precision=precision, lattice=lattice)
    with L.Solute(mask, c0, 0.01, **kw) as a, L.Solute(mask, c0, 0.01, **kw) as b:
        a.step(37)
        for _ in range(37):
            b.step(1)
        ga, ca = a.populations(), a.concentration()
        assert np.array_equal(ga, b.populations()) and np.array_equal(ca, b.concentration())
        assert abs(ca[1:].sum() - c0[mask == 0].sum()) <= 1e-5 * ca[1:].sum()
        b.step(2)
        b.set_state(ga, ca)
        a.step(18)
        b.step(18)
        ga, gb = a.populations(), b.populations()
        # the restored state takes C as given, the running one sums it again
        tol = 0.0 if precision == "f64" else 1e-6
        assert np.abs(ga - gb).max() <= tol
