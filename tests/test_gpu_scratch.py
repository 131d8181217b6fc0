"""What solves keep of their device scratch: it goes back on request and the next solve gives the same bits; a batch is
given its two-phase buffers when they fit into the free memory and what is kept together."""
import gc

import numpy as np
import pytest
import torch

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _system(env, n):
    xyz, tets = meshgen.kuhn_box(n, perturb=0.15, seed=61)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, 2)
    u, v = V.element(), V.element()
    a, l = fpp.form2(test=V), fpp.form1(test=V)
    a.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v)) + fpp.idt(u) * fpp.id(v)))
    l.assign(fpp.integrate(fpp.elements(M), fpp.cst(1.0) * fpp.id(v)))
    return a, l, u


def _solve(system):
    a, l, u = system
    a._amg = None
    u.zero()
    a.solve(l, u, rtol=1e-8, pc="gamg")
    out = u.to_numpy()
    a._amg = None
    gc.collect()
    return out


def _free():
    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_scratch_goes_back_on_request():
    env = fpp.Environment()
    system = _system(env, 24)
    want = _solve(system)
    before = _free()
    env.release_scratch()
    released = _free() - before
    total = torch.cuda.mem_get_info()[1]
    assert 0 < released <= total // 64 + (64 << 20)
    assert np.array_equal(_solve(system), want)


def test_batch_counts_what_is_kept():
    env = fpp.Environment()
    big = _system(env, 36)
    forms, integrals = [], []
    for k in range(4):
        xyz, tets = meshgen.kuhn_box(20, perturb=0.1, seed=k)
        V = fpp.Pch(fpp.Mesh(xyz, tets, env=env), 2)
        u, v = V.element(), V.element()
        forms.append(fpp.form2(test=V))
        integrals.append(fpp.integrate(fpp.elements(V.mesh), fpp.inner(fpp.gradt(u), fpp.grad(v)) + fpp.idt(u) * fpp.id(v)))
    _solve(big)
    before = _free()
    env.release_scratch()
    kept = _free() - before
    need = 4 * 48000 * 55 * 8                       # the element buffers alone
    assert kept > 4 * need                          # (a tenth more and the gather maps are within this)
    _solve(big)                                     # kept again
    ballast = torch.empty(_free() - need // 2, dtype=torch.uint8, device="cuda")
    try:
        batch = fpp.Batch(forms, integrals)
        batch.set_algo("two_phase")                 # refused where the buffers were not allocated
        batch.assemble()
    finally:
        del ballast
        torch.cuda.empty_cache()
    ref = fpp.form2(test=forms[0].space)
    ref.assign(integrals[0])
    assert np.array_equal(forms[0].values(), ref.values())
