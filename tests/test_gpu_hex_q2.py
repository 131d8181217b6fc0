"""Q2 hexahedra by sum factorisation (seven elements per block): fewer elements than a block, a full block, one
more, several blocks with a remainder; both rules (8 and 27 points), stiffness or mass alone, a constant and an
elementwise coefficient, negatively oriented elements; FP64 values against the oracle."""
import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from oracle import hexoracle as ho
from tests.helpers import assert_values_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box,qdeg,k,mass,flip", [
    ((1, 1, 1), 4, 1.0, 0.7, False),
    ((3, 2, 1), 4, None, 0.7, False),
    ((7, 1, 1), 3, None, 0.0, False),
    ((2, 2, 2), 4, 0.0, 1.0, False),
    ((2, 2, 2), 2, None, 0.7, True),
    ((5, 3, 3), 1, 1.5, 0.7, False),
    ((5, 3, 3), 4, None, 0.7, True),
])
def test_hex_q2_matches_oracle(env, oracle, box, qdeg, k, mass, flip):
    xyz, hexes = meshgen.hex_box(*box, perturb=0.2)
    if flip:                                        # mirrored elements: det K < 0
        hexes = np.ascontiguousarray(hexes[:, [1, 0, 3, 2, 5, 4, 7, 6]])
    kappa = meshgen.lognormal_kappa(len(hexes)) if k is None else np.full(len(hexes), k)
    M = fpp.Mesh(xyz, hexes, env=env)
    V = fpp.Pch(M, 2)
    N, l2g = ho.dof_table(hexes, 2)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V, trial=V)
    a.assign(fpp.integrate(fpp.elements(M), (kappa if k is None else k) * fpp.inner(fpp.gradt(u), fpp.grad(v))
                           + mass * fpp.idt(u) * fpp.id(v), quad=qdeg))
    ia, ja = oracle.pattern(N, l2g)
    val = ho.assemble(2, xyz, hexes, l2g, ia, ja, kappa=kappa, mass=mass, qdeg=qdeg)
    assert_values_close(a.values(), val, what="Q2 hexahedra")
