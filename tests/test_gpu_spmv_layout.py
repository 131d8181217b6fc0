"""The CG's product layout for matrices below 2^20 nonzeros: by rule unless a tuning file is named; then the candidates
are timed and the pick is recorded as a measurement."""
import os

import pytest

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _system(env, order, n):
    xyz, tets = meshgen.kuhn_box(n, n + 1, n - 1, perturb=0.15, seed=41)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a, l = fpp.form2(test=V), fpp.form1(test=V)
    a.assign(fpp.integrate(fpp.elements(M), 0.01 * fpp.inner(fpp.gradt(u), fpp.grad(v)) + fpp.idt(u) * fpp.id(v)))
    l.assign(fpp.integrate(fpp.elements(M), fpp.sine_source() * fpp.id(v)))
    return a, l, u


def test_a_tuning_file_holds_timed_picks(tmp_path):
    cache = os.path.join(str(tmp_path), "tune.txt")
    env = fpp.Environment(tune=True, tune_cache=cache)
    a, l, u = _system(env, 2, 9)
    count = []
    for _ in range(2):
        u.zero()
        n0 = env.launches()
        a.solve(l, u, rtol=1e-10, pc="jacobi")
        count.append(env.launches() - n0)
    picks = [ln.split() for ln in open(cache) if ln.startswith("spmv|")]
    assert len(picks) == 1
    assert count[0] - count[1] >= 24            # six launches of each of four or five candidates
