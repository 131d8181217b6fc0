"""Sparse products of the device AMG set-up, at the sizes and shapes where their path changes: the
device-built hierarchy equals the host set-up's bit for bit (every operator, prolongator, aggregate map and
lambda_max), so each output entry is the same sum in the same order on every path."""
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen
from tests.test_gpu_amg_device import _assert_same, _host_and_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,box,cfg", [
    (1, (220, 1, 1), {}),                       # 884 rows: the smallest levels set up on the device
    (1, (700, 1, 1), {}),                       # 2804 rows: whole warps from the start
    (1, (3000, 1, 1), {}),                      # ten entries a row: counted first, then filled
    (2, (15, 13, 14), {}),                      # padded rows, eight lanes, odd sizes
    (3, (9, 8, 10), {}),                        # rows of 200 entries: 256 slots at once
    (2, (13, 12, 11), dict(threshold=0.2)),     # small aggregates: rows beyond the first tables
    (3, (8, 7, 9), dict(threshold=0.3)),        # the same, into the larger tables
])
def test_product_paths_equal_host(env, order, box, cfg):
    xyz, tets = meshgen.kuhn_box(*box, perturb=0.1, seed=9)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a = fpp.form2(test=V, trial=V)
    a.assign(fpp.integrate(fpp.elements(M), meshgen.lognormal_kappa(len(tets), seed=7) * fpp.inner(fpp.gradt(u), fpp.grad(v))
                           + fpp.idt(u) * fpp.id(v)))
    host, dev, ndev = _host_and_device(env, a, **cfg)
    assert ndev >= 1
    _assert_same(host, dev)
