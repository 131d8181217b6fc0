"""Device scratch kept between calls (run on a GB300): contexts on their own streams and threads, each reusing
its freed blocks while the other's work is in flight, give the bits that one context gives alone; a context's
blocks go back to the driver when it is closed."""
import threading

import numpy as np
import pytest
import torch

import feelpp_gb300 as fpp
from feelpp_gb300 import meshgen

pytestmark = pytest.mark.gpu

SIZES = [(1, 9), (2, 7), (1, 14), (2, 5)]


def _solve(env, order, n, pc):
    xyz, tets = meshgen.kuhn_box(n, perturb=0.15, seed=61)
    M = fpp.Mesh(xyz, tets, env=env)
    V = fpp.Pch(M, order)
    u, v = V.element(), V.element()
    a, l = fpp.form2(test=V), fpp.form1(test=V)
    a.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v))))
    l.assign(fpp.integrate(fpp.elements(M), fpp.cst(1.0) * fpp.id(v)))
    a += fpp.on(fpp.boundaryfaces(M), rhs=l, element=u, expr=0.0, type="elimination_symmetric")
    a.solve(l, u, rtol=1e-10, pc=pc)
    return u.to_numpy()


def _work(out, key, env):
    try:
        out[key] = [_solve(env, order, n, pc) for _ in range(3) for order, n in SIZES for pc in ("jacobi", "gamg")]
    except Exception as e:  # noqa: BLE001 - reported by the main thread
        out[key] = e


def test_threads_and_streams_share_nothing(env):
    ref = [_solve(env, order, n, pc) for order, n in SIZES for pc in ("jacobi", "gamg")]
    out = {}
    envs = [fpp.Environment(tune=True) for _ in range(3)]
    threads = [threading.Thread(target=_work, args=(out, k, e)) for k, e in enumerate(envs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(3):
        assert not isinstance(out[k], Exception), out[k]
        for got, want in zip(out[k], ref * 3):
            assert np.array_equal(got, want)


def test_a_closed_context_keeps_nothing():
    def once():
        env = fpp.Environment(tune=True)
        _solve(env, 2, 12, "gamg")
        env.sync()
        import gc
        gc.collect()
        env.close()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    once()
    free = [once() for _ in range(4)]
    assert max(free) - min(free) <= 64 << 20      # no growth from context to context (driver granularity aside)
