"""The scratch pool's key: a kept block goes to later work of the same stream on the same device only. On the CPU
over a fake runtime (tests/cpp/pool_fake.cpp: two devices, cudaStreamLegacy and cudaStreamPerThread, the bound, an
allocation that fails); on a GB300, contexts on cudaStreamPerThread in three threads give the bits that one context
on its own stream gives."""
import os
import subprocess
import threading

import numpy as np
import pytest

from tests.conftest import ROOT


def test_blocks_by_device_and_stream(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "pool_fake")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(cuda, "include"), "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "feelpp_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", "pool_fake.cpp"),
                    os.path.join(ROOT, "feelpp_gb300", "csrc", "pool.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def _problems(env):
    import feelpp_gb300 as fpp
    from feelpp_gb300 import meshgen
    out = []
    for order, n in [(1, 9), (2, 7), (1, 14), (2, 5)]:
        xyz, tets = meshgen.kuhn_box(n, perturb=0.15, seed=61)
        M = fpp.Mesh(xyz, tets, env=env)
        V = fpp.Pch(M, order)
        u, v = V.element(), V.element()
        a, l = fpp.form2(test=V), fpp.form1(test=V)
        a.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v))))
        l.assign(fpp.integrate(fpp.elements(M), fpp.cst(1.0) * fpp.id(v)))
        a += fpp.on(fpp.boundaryfaces(M), rhs=l, element=u, expr=0.0, type="elimination_symmetric")
        out.append((a, l, u))
    env.sync()
    return out


def _solve(problems, out, key):
    try:
        got = []
        for a, l, u in problems * 3:
            for pc in ("jacobi", "gamg"):
                u.zero()
                a.solve(l, u, rtol=1e-10, pc=pc)
                got.append(u.to_numpy())
        out[key] = got
    except Exception as e:  # noqa: BLE001 - reported by the main thread
        out[key] = e


@pytest.mark.gpu
def test_per_thread_streams(env):
    """The problems are made one after another (their synchronous copies would break into another thread's graph
    capture on a stream that waits for the legacy one); the solves and AMG set-ups run at once."""
    import feelpp_gb300 as fpp
    per_thread = 2                                  # cudaStreamPerThread
    out = {}
    _solve(_problems(env), out, "ref")
    probs = [_problems(fpp.Environment(stream=per_thread, tune=True)) for _ in range(3)]
    threads = [threading.Thread(target=_solve, args=(p, out, k)) for k, p in enumerate(probs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in ("ref", 0, 1, 2):
        assert not isinstance(out[k], Exception), out[k]
        for got, want in zip(out[k], out["ref"]):
            assert np.array_equal(got, want)
