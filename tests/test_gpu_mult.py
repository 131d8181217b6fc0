"""y = A x at the edges of its blocks of 128 rows and over rows of very different lengths, short (two lanes per row,
rows by length) and long ones (P3: the general kernel), against the matrix on the host."""
import numpy as np
import pytest
import scipy.sparse as sp

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,box", [(1, (1, 1, 1)), (1, (31, 1, 1)), (1, (42, 2, 0)), (1, (7, 3, 3)), (2, (7, 3, 3)), (2, (9, 8, 7)),
                                       (3, (4, 3, 5))])
def test_mult_matches_host(env, order, box):
    box = tuple(max(n, 1) for n in box)
    xyz, tets = meshgen.kuhn_box(*box, perturb=0.2, seed=4)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V)
    a.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v)) + fpp.idt(u) * fpp.id(v)))
    ia, ja, val = a.csr()
    A = sp.csr_matrix((val, ja, ia), shape=(V.ndof, V.ndof))
    x = np.random.default_rng(order).standard_normal(V.ndof)
    u.upload(x)
    y = fpp.DeviceVector(env, V.ndof)
    a.mult(u, y)
    # a row sum of at most 256 products, summed in any order
    bound = (256 + 2) * 2.0 ** -53 * (abs(A) @ np.abs(x))
    assert np.all(np.abs(y.to_numpy() - A @ x) <= 2 * bound)
