"""Device AMG set-up with a near null space: products whose rows have more columns (129 to 192) than a group of
eight lanes can sort but fewer than its table has room for. The device-built hierarchy equals the host set-up's bit
for bit; that such rows exist is read off the host hierarchy (the prolongator has the pattern of A P0)."""
import ctypes as C

import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import _ffi, meshgen
from tests.test_gpu_amg_device import _assert_same, _levels, _p

pytestmark = pytest.mark.gpu


def _vectors(V, xyz, count):
    """the rigid body modes, and for eight vectors two products of their rotations' components"""
    B = [m.to_numpy() for m in V.rigid_body_modes()]
    if count == 8:
        x, y, z = B[3][1::3], -B[3][0::3], -B[4][1::3]
        o = np.zeros_like(x)
        B += [np.stack((x * y, o, o), 1).ravel(), np.stack((o, y * z, o), 1).ravel()]
    return B


@pytest.mark.parametrize("box,threshold,count,level", [
    ((9, 8, 8), 0.2, 6, 1),
    ((8, 7, 7), 0.1, 8, 0),
    ((16, 14, 14), 0.1, 6, 1),
    ((16, 14, 14), 0.0, 6, None),               # none that long
])
def test_rows_longer_than_a_group_sorts(env, box, threshold, count, level):
    xyz, tets = meshgen.kuhn_box(*box, lengths=(4.0, 1.0, 1.0), perturb=0.1, seed=3)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pchv(M, 2)
    u, v = V.element(), V.element()
    a, l = fpp.form2(test=V, trial=V), fpp.form1(test=V)
    a.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, 1.0, 0.5), fpp.grad(v))))
    l.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.cst_vec(0, 0, -1), fpp.id(v))))
    a += fpp.on(fpp.markedfaces(M, 0.0), rhs=l, element=u, expr=0.0, type="elimination_symmetric")
    B = np.ascontiguousarray(np.stack(_vectors(V, xyz, count)))
    vecs = [fpp.DeviceVector(env, V.ndof) for _ in range(count)]
    for d, b in zip(vecs, B):
        d.upload(np.ascontiguousarray(b))
    arr = (C.c_void_p * count)(*[d.h.value for d in vecs])
    c = _ffi.AmgCfg(threshold, 0, 0, 0, 0, 0)
    c.block_size, c.nns_count, c.nns, c.nns_host = 3, count, C.cast(arr, C.c_void_p), B.ctypes.data
    ia, ja, val = a.csr()
    ia, ja, val = np.ascontiguousarray(ia, np.int64), np.ascontiguousarray(ja, np.int32), np.ascontiguousarray(val)
    hh, hd = C.c_void_p(), C.c_void_p()
    assert env.lib.fgpu_amg_host_build(len(ia) - 1, _p(ia), _p(ja), _p(val), C.byref(c), 16, C.byref(hh)) == 0
    env.check(env.lib.fgpu_amg_device_build(env.h, a.h, C.byref(c), C.byref(hd)))
    try:
        host, dev, ndev = _levels(env.lib, hh), _levels(env.lib, hd), env.lib.fgpu_amg_host_device_levels(hd)
    finally:
        env.lib.fgpu_amg_host_destroy(hh)
        env.lib.fgpu_amg_host_destroy(hd)
    if level is not None:
        assert ndev > level
        A, P, _, _ = host[0][level]
        n, rows = len(A[0]) - 1, np.diff(P[0])
        assert n >= 4096 and len(A[1]) / n * count > 600      # eight lanes, 256 slots
        assert np.any((rows > 128) & (rows <= 192))
    _assert_same(host, dev)
