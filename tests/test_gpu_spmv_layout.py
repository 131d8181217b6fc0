"""The CG's product layout for matrices below 2^20 nonzeros: by rule (16, 8 or 4 lanes a row, or SELL) unless a tuning
file is named; then the candidates are timed and the pick is recorded as a measurement. Every layout gives the
oracle's solution of a well-conditioned system, and the same bits in another context."""
import os

import numpy as np
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


# rows and mean lengths of each class: 16 lanes, 8, 4, SELL (P1 40: also in binary32)
@pytest.mark.parametrize("order,n", [(2, 4), (3, 6), (2, 10), (1, 16), (2, 14), (1, 28), (1, 40)])
def test_layouts_solve(env, oracle, order, n):
    a, l, u = _system(env, order, n)
    assert a.nnz < 1 << 20
    ia, ja, val = a.csr()
    b = l.to_numpy()
    want, _ = oracle.pcg(ia, ja, val, b, rtol=1e-13)[:2]
    got = {}
    for key, kw in (("f64", {}), ("mixed", dict(mixed=True)), ("df64", dict(arith="df64"))):
        u.zero()
        st = a.solve(l, u, rtol=1e-11, pc="jacobi", **kw)
        assert st["rel_residual"] <= 1e-11
        got[key] = u.to_numpy()
        assert np.linalg.norm(got[key] - want) <= 1e-8 * np.linalg.norm(want)
    a2, l2, u2 = _system(fpp.Environment(), order, n)
    a2.solve(l2, u2, rtol=1e-11, pc="jacobi")
    assert np.array_equal(u2.to_numpy(), got["f64"])


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
