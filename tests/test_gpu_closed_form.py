"""The closed-form P1/P2 element matrices (run on a GB300): element counts around a warp's 32 (full pieces by
bulk copy, the partial one by plain stores), mass or stiffness alone and far apart in size, a scaled mesh, a
device coefficient, and rules that do not integrate the products exactly (they keep the seven-term sums).

Tolerances: FP64 as in helpers; binary32 (c + 16) 2^-24 of the largest entry as in the gather tests."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from tests.helpers import assert_values_close, oracle_system

pytestmark = pytest.mark.gpu


def _mesh(count, scale=1.0):
    xyz, tets = meshgen.kuhn_box(3, 3, 4, perturb=0.15, seed=51)
    tets = tets[:count]
    used, new = np.unique(tets, return_inverse=True)
    return scale * xyz[used], np.ascontiguousarray(new.reshape(tets.shape).astype(np.int32))


def _values(env, xyz, tets, order, kappa, mass, precision="f64", quad=0):
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V, precision=precision)
    a.assign(fpp.integrate(fpp.elements(M), kappa * fpp.inner(fpp.gradt(u), fpp.grad(v)) + mass * (fpp.idt(u) * fpp.id(v)), quad=quad))
    return a.values()


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("count,scale,factor,mass", [(1, 1.0, 1.0, 1.0), (31, 1.0, 1.0, 0.0), (32, 1.0, 0.0, 1.0),
                                                      (33, 1e-3, 1.0, 1.0), (64, 40.0, 1e-6, 1.0), (95, 1.0, 1.0, 1e-5),
                                                      (216, 1.0, 1.0, 0.7)])
def test_element_counts(env, oracle, order, count, scale, factor, mass, precision):
    xyz, tets = _mesh(count, scale)
    kappa = factor * meshgen.lognormal_kappa(count, seed=52)
    ref = oracle_system(oracle, xyz, tets, order, kappa=kappa, mass=mass)[4]
    tol = dict(rtol=0.0, atol=(np.bincount(tets.reshape(-1)).max() + 16) * 2.0 ** -24) if precision == "f32" else {}
    assert_values_close(_values(env, xyz, tets, order, kappa, mass, precision), ref, what="%d elements" % count, **tol)


@pytest.mark.parametrize("order,quad", [(1, 1), (1, 2), (1, 5), (2, 1), (2, 2), (2, 3), (2, 4), (2, 8)])
def test_every_rule(env, oracle, order, quad):
    xyz, tets = _mesh(70)
    kappa = meshgen.lognormal_kappa(len(tets), seed=53)
    ref = oracle_system(oracle, xyz, tets, order, kappa=kappa, mass=0.7, qdeg=quad)[4]
    assert_values_close(_values(env, xyz, tets, order, kappa, 0.7, quad=quad), ref, what="degree %d" % quad)


def test_device_coefficient(env, oracle):
    xyz, tets = _mesh(70)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, 2)
    u, v = V.element(), V.element()
    kt = fpp.DeviceScalar(env, 1.375)
    a = fpp.form2(test=V)
    a.assign(fpp.integrate(fpp.elements(M), fpp.idt(u) * fpp.id(v) + 0.01 * kt * fpp.inner(fpp.gradt(u), fpp.grad(v))))
    ref = oracle_system(oracle, xyz, tets, 2, kappa=np.full(len(tets), 0.01 * 1.375), mass=1.0)[4]
    assert_values_close(a.values(), ref, what="kappa(t)")
