"""Elasticity summed from the elements' barycentric gradients: every quadrature degree that the entry point takes
(exact ones form the blocks inside the gather, the others store element blocks), each modulus alone, mirrored
elements, accumulation and a captured reassembly; against the binary64 row gather."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import _ffi, meshgen
from tests.helpers import assert_values_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,qdeg,lam,mu,flip", [(1, 0, 1.3, 0.4, True), (1, 1, 0.0, 0.7, False), (1, 2, 1.0, 0.0, False),
                                                    (2, 0, 1.3, 0.4, True), (2, 1, 1.0, 0.5, False), (2, 2, 0.0, 0.7, False),
                                                    (2, 3, 1.0, 0.0, False), (2, 4, 1e6, 1e-3, False)])
def test_matches_row_gather(env, order, qdeg, lam, mu, flip):
    xyz, tets = meshgen.kuhn_box(5, 3, 4, lengths=(1.0, 0.1, 3.0), perturb=0.2, seed=11)
    if flip:
        tets[::2] = tets[::2][:, [1, 0, 2, 3]]
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, order)
    u, v = V.element(), V.element()
    form = fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, lam, mu), fpp.grad(v)), quad=qdeg)
    ref = fpp.form2(test=V)
    ref.algo = _ffi.ALGO_GATHER
    ref.assign(form)
    a = fpp.form2(test=V)
    a.assign(form)
    want, got = ref.values(), a.values()
    assert_values_close(got, want, what="fused elasticity")
    f = fpp.form2(test=V, precision="f32")
    f.assign(form)
    # at most 24 elements, 4 products of two rounded vectors each, then two products and a sum
    assert np.abs(f.values() - want).max() <= (24 * 4 + 16) * 2.0 ** -24 * np.abs(want).max()
    with fpp.capture(env) as g:
        a.assign(form)
    a.zero()
    g.launch()
    assert np.array_equal(a.values(), got)
    a += form
    np.testing.assert_allclose(a.values(), 2 * got, rtol=1e-13, atol=1e-30 * np.abs(want).max())


def test_first_assembly_is_not_captured(env):
    xyz, tets = meshgen.kuhn_box(2)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, 2)
    u, v = V.element(), V.element()
    form = fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, 1.0, 0.5), fpp.grad(v)))
    fpp.form2(test=V).assign(form)                  # the space's plan is there, a second matrix has assembled nothing
    b = fpp.form2(test=V)
    with pytest.raises(Exception):
        with fpp.capture(env):
            b.assign(form)
