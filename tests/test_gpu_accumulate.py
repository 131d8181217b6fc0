"""a += integral (the gather added to the values it finds): scalar forms, elasticity and batches, matrices whose slices
fit the device at once and larger ones. binary32: one rounded addition per entry, bit for bit. FP64: d2df (2^-48),
the sloppy double-float sum (2^-47 of both) and the plain assembly's own rounding: within 2^-45 (|old| + |added|)."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _forms(V, vector):
    u, v = V.element(), V.element()
    if vector:
        return [fpp.integrate(fpp.elements(V.mesh), fpp.inner(fpp.stress(u, lam, mu), fpp.grad(v))) for lam, mu in ((1.3, 0.6), (0.4, -0.9))]
    return [fpp.integrate(fpp.elements(V.mesh), k * fpp.inner(fpp.gradt(u), fpp.grad(v)) + m * (fpp.idt(u) * fpp.id(v)))
            for k, m in ((1.5, 0.7), (-0.8, 2.0))]


def _check(old, added, got, precision):
    if precision == "f32":
        assert np.array_equal(got.astype(np.float32), old.astype(np.float32) + added.astype(np.float32))
    else:
        assert np.all(np.abs(got - (old + added)) <= 2.0 ** -45 * (np.abs(old) + np.abs(added)))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("order,box,vector", [
    (1, (3, 2, 3), False), (1, (30, 29, 31), False), (2, (5, 4, 6), False), (2, (26, 25, 27), False), (3, (4, 5, 3), False),
    (3, (18, 17, 19), False), (1, (4, 3, 5), True), (1, (29, 28, 30), True), (2, (3, 4, 3), True), (2, (17, 16, 18), True),
])
def test_added_to_the_values(env, order, box, vector, precision):
    xyz, tets = meshgen.kuhn_box(*box, perturb=0.15, seed=31)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, order) if vector else fpp.Pch(M, order)
    a = fpp.form2(test=V, precision=precision)
    one, two = _forms(V, vector)
    a.assign(two)
    added = a.values()
    a.assign(one)
    old = a.values()
    a += two
    _check(old, added, a.values(), precision)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("size", [4, 14])
def test_batches(env, size, precision):
    forms, ones, twos = [], [], []
    for k in range(4):
        xyz, tets = meshgen.kuhn_box(size + k, perturb=0.15, seed=32 + k)
        V = fpp.Pch(fpp.Mesh(xyz, tets, env=env), 1 + k % 3)
        forms.append(fpp.form2(test=V, precision=precision))
        one, two = _forms(V, False)
        ones.append(one)
        twos.append(two)
    first, second = fpp.Batch(forms, ones), fpp.Batch(forms, twos)
    second.assemble()
    added = [f.values() for f in forms]
    first.assemble()
    old = [f.values() for f in forms]
    second.assemble(accumulate=True)
    for f, o, x in zip(forms, old, added):
        _check(o, x, f.values(), precision)
