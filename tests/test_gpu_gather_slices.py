"""The sliced gather of the two-phase assembly at the edges of its plan (run on a GB300): fewer sums than a
slice, one element, elements and vertices in random order (bins whose elements share nothing), a vertex of
about 500 elements (more contributions than the plan's largest count class), '+=' onto other values.

Tolerances: FP64 as in helpers (1e-12 relative + 1e-14 of the largest entry); binary32 (c + 16) 2^-24 of the
largest entry, c the largest number of contributions of an entry (one rounding per addition, at most 16 in
an element entry)."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from tests.helpers import assert_values_close, oracle_system

pytestmark = pytest.mark.gpu


def _box(nx, ny, nz, shuffle):
    xyz, tets = meshgen.kuhn_box(nx, ny, nz, perturb=0.15, seed=31)
    if not shuffle:
        return xyz, tets
    rng = np.random.default_rng(32)
    new = rng.permutation(len(xyz))
    out = np.empty_like(xyz)
    out[new] = xyz
    return out, np.ascontiguousarray(new[tets][rng.permutation(len(tets))].astype(np.int32))


def _cone(m):
    """Tetrahedra from the centre of a sphere to a triangulation of m points on it."""
    from scipy.spatial import ConvexHull
    k = np.arange(m) + 0.5
    t, z = np.pi * (1 + 5 ** 0.5) * k, 1 - 2 * k / m
    r = np.sqrt(1 - z * z)
    pts = np.stack([r * np.cos(t), r * np.sin(t), z], 1)
    tri = ConvexHull(pts).simplices
    xyz = np.concatenate([[[0.01, -0.02, 0.015]], pts])
    return xyz, np.concatenate([np.zeros((len(tri), 1), np.int32), tri + 1], 1).astype(np.int32)


MESHES = {
    "one": lambda: (np.array([[0.0, 0, 0], [1, 0.1, 0], [0.2, 0.9, 0], [0.1, 0.2, 1.1]]), np.array([[0, 1, 2, 3]], np.int32)),
    "cube": lambda: _box(1, 1, 1, False),
    "bar": lambda: _box(17, 1, 2, False),
    "shuffled": lambda: _box(7, 5, 6, True),
    "cone": lambda: _cone(250),
}


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("name,order", [("one", 1), ("one", 3), ("cube", 2), ("bar", 1), ("bar", 3), ("shuffled", 1),
                                        ("shuffled", 2), ("shuffled", 3), ("cone", 1)])
def test_scalar_forms(env, oracle, name, order, precision):
    xyz, tets = MESHES[name]()
    kappa = meshgen.lognormal_kappa(len(tets), seed=33)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V, precision=precision)
    form = fpp.integrate(fpp.elements(M), kappa * fpp.inner(fpp.gradt(u), fpp.grad(v)) + fpp.idt(u) * fpp.id(v))
    a.assign(form)
    _, l2g, ia, ja, val = oracle_system(oracle, xyz, tets, order, kappa=kappa, mass=1.0)
    got = a.values()
    scale, count = np.abs(val).max(), np.bincount(tets.reshape(-1)).max()
    tol = dict(rtol=0.0, atol=(count + 16) * 2.0 ** -24) if precision == "f32" else {}
    assert_values_close(got, val, what=name, **tol)
    # an entry and its transpose are one sum
    row = np.repeat(np.arange(len(ia) - 1), np.diff(ia))
    assert np.array_equal(got, got[np.lexsort((row, ja))])
    a += form
    np.testing.assert_allclose(a.values(), 2 * got, rtol=1e-6 if precision == "f32" else 1e-13, atol=1e-30 * scale)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("name,order", [("one", 1), ("cube", 2), ("shuffled", 1), ("shuffled", 2)])
def test_elasticity(env, oracle, name, order, precision):
    xyz, tets = MESHES[name]()
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V, precision=precision)
    form = fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, 1.0, 0.5), fpp.grad(v)))
    a.assign(form)
    _, _, _, _, val = oracle_system(oracle, xyz, tets, order, ncomp=3, kind=1, lam=1.0, mu=0.5)
    got = a.values()
    count = np.bincount(tets.reshape(-1)).max()
    # binary32: a block entry is at most 9 products of 9 terms
    assert_values_close(got, val, what=name, **(dict(rtol=0.0, atol=(count + 96) * 2.0 ** -24) if precision == "f32" else {}))
    a += form
    scale = np.abs(val).max()
    np.testing.assert_allclose(a.values(), 2 * got, rtol=1e-6 if precision == "f32" else 1e-13, atol=1e-30 * scale)
