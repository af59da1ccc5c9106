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


# Cubes in, below and above the sizes whose steps are not chained (19 K to 71 K
# nodes in FP64, 38 K to 152 K in FP32 and FP16), and boxes above 120 MiB of
# populations and table, where blocks prefetch (1.1 M nodes in FP16, 0.85 M in
# FP32, 0.56 M in FP64).
@pytest.mark.parametrize("shape,phi", [((17, 16, 19), 0.8), ((33, 35, 39), 0.8), ((45, 47, 51), 0.9),
                                       ((128, 121, 119), 0.7)])
@pytest.mark.parametrize("precision", ["f32", "f16", "f64", "f64fast"])
def test_a_call_equals_its_steps_one_by_one(precision, shape, phi):
    """Captured chains, single steps that follow one another and lone steps
    give the same bits."""
    mask = spheres(shape, phi, 4.5, seed=8)
    kw = dict(g=(1e-5, 4e-6, -3e-6), precision=precision)
    with L.SinglePhase(mask, 0.1, **kw) as a, L.SinglePhase(mask, 0.1, **kw) as b:
        for n in (37, 15, 33):
            a.step(n)
        for _ in range(85):
            b.step(1)
        assert np.array_equal(a.populations(), b.populations())
        for x, y in zip(a.fields(), b.fields()):
            assert np.array_equal(x, y)
        assert a.reduce() == b.reduce()


# FP32 reads the row form above 90 MiB (0.64 M nodes) where rows of cells are
# 100 cells or longer; other storages and curve orders read the int32 table.
@pytest.mark.parametrize("precision,ordering,shape,rows", [
    ("f32", "reference", (128, 101, 97), True), ("f32", "reference", (90, 128, 109), False),
    ("f32", "hilbert", (128, 101, 97), False), ("f32", "reference", (101, 80, 80), False),
    ("f16", "reference", (128, 121, 119), False), ("f64", "reference", (128, 101, 97), False),
    ("f64fast", "reference", (128, 101, 97), False)])
def test_where_the_row_form_is_read(precision, ordering, shape, rows):
    mask = spheres(shape, 0.8, 4.5, seed=2)
    with L.SinglePhase(mask, 0.1, (1e-6, 0.0, 0.0), precision=precision, ordering=ordering) as s:
        per_step = s.memory()["bytes_per_lu"] - 38 * {"f16": 2, "f32": 4}.get(precision, 8)
        assert per_step == 36 if not rows else 18 <= per_step < 19


def test_memory_counts_what_a_field_read_keeps():
    mask = spheres((33, 21, 18), 0.55, 3.0, seed=9)
    with L.SinglePhase(mask, 0.1, (1e-6, 0.0, 0.0)) as s:
        before = s.memory()["device_bytes"]
        s.fields()
        npad, rows = -(-s.count // 256) * 256, s.count + 1
        assert s.memory()["device_bytes"] - before == 8 * 4 * (npad + rows)
