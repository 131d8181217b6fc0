"""A captured elasticity reassembly after an assembly of the same matrix by another quadrature rule: exact (formed in
the gather) after inexact (through the element buffer) and the other way round; replays give the bits of the plain
assembly. Without an earlier assembly of the matrix the capture is refused."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from tests.helpers import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("first,second", [(1, 0), (0, 1)])
def test_capture_after_another_rule(env, first, second, precision):
    xyz, tets = mesh(5, perturb=0.2, lengths=(4.0, 1.0, 1.0))
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, 2)
    u, v = V.element(), V.element()
    form = lambda quad: fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, 1.3, 0.6), fpp.grad(v)), quad=quad)  # noqa: E731
    a, b, c = (fpp.form2(test=V, precision=precision) for _ in range(3))
    b.assign(form(second))
    want = b.values()
    a.assign(form(first))
    assert not np.array_equal(a.values(), want)
    with fpp.capture(env) as g:
        a.assign(form(second))
    for _ in range(2):
        a.zero()
        g.launch()
        env.sync()
        assert np.array_equal(a.values(), want)
    with pytest.raises(fpp.FgpuError):
        with fpp.capture(env):
            c.assign(form(second))
    c.assign(form(second))
    assert np.array_equal(c.values(), want)
