"""The host assembly in one, two, four and twelve transfers (by the number of values), elements in order and shuffled,
by the copy engine and by kernel stores: the bits of the device assembly, in repeated passes. Kernel stores are a
launch per transfer (one transfer up to 4 M values, where the copy engine's gather may be in two launches)."""
import ctypes as C

import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import _ffi, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,box,more,shuffle", [
    (1, (10, 9, 11), 1, False),
    (2, (13, 14, 12), 0, False),                # two gather launches and copies, one and one store kernel
    (2, (13, 14, 12), 0, True),
    (2, (27, 29, 30), 4, False),
    (2, (27, 29, 30), 1, True),                 # shuffled: no row is complete before the last part
    (3, (31, 30, 30), 12, False),
])
def test_transfers(env, order, box, more, shuffle):
    import torch
    xyz, tets = meshgen.kuhn_box(*box, perturb=0.1, seed=2)
    if shuffle:
        tets = np.ascontiguousarray(tets[np.random.default_rng(6).permutation(len(tets))])
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    a, b = fpp.form2(test=V), fpp.form2(test=V)
    d = _ffi.FormDesc()
    d.kind, d.kappa, d.mass, d.quad_degree, d.algo = _ffi.FORM_LAPLACE_MASS, 1.5, 0.7, 0, _ffi.ALGO_TWO_PHASE
    env.check(env.lib.fgpu_assemble_matrix_dev(env.h, a.h, C.byref(d), None, 0))
    want = a.values()
    out = torch.empty(a.nnz, dtype=torch.float64, pin_memory=True)
    launches = {}
    try:
        for mode in ("auto", "copy", "direct"):
            env.set_host_transfer(mode)
            for _ in range(3):
                out.zero_()
                b.zero()
                n0 = env.launches()
                env.check(env.lib.fgpu_assemble_matrix_host(env.h, b.h, C.byref(d), C.c_void_p(out.data_ptr())))
                launches[mode] = env.launches() - n0
                assert np.array_equal(out.numpy(), want)
                assert np.array_equal(b.values(), want)
    finally:
        env.set_host_transfer("auto")
    assert launches["auto"] == launches["copy"]
    assert launches["direct"] - launches["copy"] == more
