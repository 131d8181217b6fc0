"""Error of the P3 Laplace + mass matrix against Gauss quadrature in binary64 (perf/cases.py: exact). With the
records' determinant and metric as renormalised double-float sums it is 1.113e-14 of the matrix in the Frobenius norm
in this case, with compensated dot products 1.200e-14; the bound lies between, a hundredth above the first for the
order of the reference's own sums."""
import importlib.util
import os

import pytest
import torch

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


def test_p3_records_are_renormalised(env):
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    case = dict(kind="assemble", order=3, nx=17, ny=18, nz=16, dtype="f64")
    got = cases.run(cases.prepare(case, 3))
    want = cases.exact(case, 3)
    assert torch.linalg.norm(got - want.to(got.device)) <= 1.125e-14 * torch.linalg.norm(want)
