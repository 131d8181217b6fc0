"""Curved P1/P2 tetrahedra at the element counts where the lane-per-element kernel changes from eight warps a block to
four (more blocks of 32 elements than a GB300's 152 SMs), for rules with fewer points than warps and for many.

Tolerance: 1e-12 relative + 1e-13 of the largest entry, the parity bound of the curved forms."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from tests.helpers import assert_values_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,quad", [(1, 1), (1, 5), (2, 1), (2, 2), (2, 6)])
@pytest.mark.parametrize("count", [152 * 32, 152 * 32 + 1, 5900])
def test_blocks_around_the_sms(env, oracle, order, quad, count):
    xyz, tets, ho = meshgen.curved_box(10, amp=0.1, perturb=0.1, seed=41)
    used, new = np.unique(tets[:count], return_inverse=True)
    xyz, tets, ho = xyz[used], np.ascontiguousarray(new.reshape(count, 4).astype(np.int32)), ho[:count]
    kappa = meshgen.lognormal_kappa(count, seed=42)
    M = fpp.Mesh(xyz, tets, env=env, ho=ho)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V)
    a.assign(fpp.integrate(fpp.elements(M), kappa * fpp.inner(fpp.gradt(u), fpp.grad(v)) + 0.7 * (fpp.idt(u) * fpp.id(v)), quad=quad))
    N, l2g = oracle.dof_table(tets, order)
    ia, ja = oracle.pattern(N, l2g)
    ref = oracle.assemble_ho(order, xyz, tets, ho, l2g, ia, ja, kappa=kappa, mass=0.7, qdeg=quad)
    assert_values_close(a.values(), ref, atol=1e-13, what="%d elements" % count)
