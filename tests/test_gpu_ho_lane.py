"""The lane-per-element kernel of curved P1/P2 tetrahedra (run on a GB300) at the edges of its blocks of 32
elements and four points: element counts around 32, every quadrature degree (1 to 31 points), mass and
stiffness alone, a scaled mesh, and a degenerate element in the last partial block.

Tolerance: 1e-12 relative + 1e-13 of the largest entry, the parity bound of the curved forms with room for the
cancelling entries of low-degree rules (a rule's weights may be negative)."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from tests.helpers import assert_values_close

pytestmark = pytest.mark.gpu


def _mesh(count, scale=1.0):
    """The first `count` tetrahedra of a curved box (vertices renumbered)."""
    xyz, tets, ho = meshgen.curved_box(3, amp=0.1, perturb=0.1, seed=41)
    tets, ho = tets[:count], ho[:count]
    used, new = np.unique(tets, return_inverse=True)
    return scale * xyz[used], np.ascontiguousarray(new.reshape(tets.shape).astype(np.int32)), scale * ho


def _values(env, xyz, tets, ho, order, kappa, mass, quad):
    M = fpp.Mesh(xyz, tets, env=env, ho=ho)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V)
    a.assign(fpp.integrate(fpp.elements(M), kappa * fpp.inner(fpp.gradt(u), fpp.grad(v)) + mass * (fpp.idt(u) * fpp.id(v)), quad=quad))
    return a.values()


@pytest.mark.parametrize("order,quad", [(1, q) for q in range(1, 6)] + [(2, q) for q in range(1, 8)])
def test_every_rule(env, oracle, order, quad):
    xyz, tets, ho = _mesh(33)
    kappa = meshgen.lognormal_kappa(len(tets), seed=42)
    N, l2g = oracle.dof_table(tets, order)
    ia, ja = oracle.pattern(N, l2g)
    ref = oracle.assemble_ho(order, xyz, tets, ho, l2g, ia, ja, kappa=kappa, mass=0.7, qdeg=quad)
    assert_values_close(_values(env, xyz, tets, ho, order, kappa, 0.7, quad), ref, atol=1e-13, what="degree %d" % quad)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("count,scale,mass", [(1, 1.0, 1.0), (31, 1.0, 0.0), (32, 1e-3, 1.0), (65, 50.0, 0.3)])
def test_element_counts(env, oracle, order, count, scale, mass):
    xyz, tets, ho = _mesh(count, scale)
    kappa = meshgen.lognormal_kappa(count, seed=43)
    N, l2g = oracle.dof_table(tets, order)
    ia, ja = oracle.pattern(N, l2g)
    ref = oracle.assemble_ho(order, xyz, tets, ho, l2g, ia, ja, kappa=kappa, mass=mass)
    assert_values_close(_values(env, xyz, tets, ho, order, kappa, mass, 0), ref, atol=1e-13, what="%d elements" % count)


def test_degenerate_element_is_reported(env):
    xyz, tets, ho = _mesh(34)
    ho = ho.copy()
    bad = xyz[tets[33]]
    flat = np.repeat(bad[:1], 4, axis=0)            # all nodes of the last element in one point
    xyz2 = np.concatenate([xyz, flat])
    tets2 = tets.copy()
    tets2[33] = len(xyz) + np.arange(4)
    ho[33] = flat[0]
    with pytest.raises(fpp.FgpuError) as e:
        _values(env, xyz2, tets2, ho, 2, 1.0, 1.0, 0)
    assert e.value.code == 3
    # the context stays usable
    assert np.isfinite(_values(env, xyz, tets, _mesh(34)[2], 2, 1.0, 1.0, 0)).all()
