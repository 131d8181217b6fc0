"""The host assembly of matrices whose gather runs in quarters (more sums than fit the device at once): elements in
order (rows leave while later quarters run) and shuffled (no row is complete before the end), by kernel stores and by
the copy engine; the same bits as the device assembly, also in a second pass."""
import ctypes as C

import numpy as np
import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import _ffi, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
def test_host_values_in_quarters(env, shuffle, mode):
    import torch
    xyz, tets = meshgen.kuhn_box(25, 22, 24, perturb=0.1, seed=2)
    if shuffle:
        tets = np.ascontiguousarray(tets[np.random.default_rng(6).permutation(len(tets))])
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, 2)
    a, b = fpp.form2(test=V), fpp.form2(test=V)
    d = _ffi.FormDesc()
    d.kind, d.kappa, d.mass, d.quad_degree, d.algo = _ffi.FORM_LAPLACE_MASS, 1.5, 0.7, 0, _ffi.ALGO_TWO_PHASE
    env.check(env.lib.fgpu_assemble_matrix_dev(env.h, a.h, C.byref(d), None, 0))
    want = a.values()
    out = torch.empty(a.nnz, dtype=torch.float64, pin_memory=True)
    env.check(env.lib.fgpu_set_host_transfer(env.h, mode))
    try:
        for _ in range(2):
            out.zero_()
            env.check(env.lib.fgpu_assemble_matrix_host(env.h, b.h, C.byref(d), C.c_void_p(out.data_ptr())))
            assert np.array_equal(out.numpy(), want)
            assert np.array_equal(b.values(), want)
    finally:
        env.check(env.lib.fgpu_set_host_transfer(env.h, 0))
