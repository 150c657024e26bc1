"""Iteration limits of real systems on the mixed path.  The resident kernel runs
CG for both methods, but a limit that was enough for the method asked for stays
enough: a CG request's bounds each inner solve between two FP64 residuals
(restarted refinement), a BiCGSTAB request's counts iterations of two products
each.  A limit below what the solve needs still ends it."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs, rel2
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


# both take 75 to 92 products to 12 digits
@pytest.mark.parametrize("method,maxit", [("CG", 30), ("BICGSTAB", 60)])
def test_limit_is_enough(method, maxit, oracle_mod):
    P = workloads.disc(32, 3, 0.0, 8)
    om = oracle_mod.Mesh(P.coords, P.elems)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    val = om.assemble(cm, ck, ca, 0.0, False)
    X = oracle_mod.solve_direct(om.rowptr, om.colidx, val, qvec, "nd", om.coords)
    s = capi.FwdSolver(gm, method, 1e-12, "ICH", False, maxit=maxit, precision="mixed")
    s.reset(cm, ck, ca, 0.0)
    x, res = s.calc_fields(qvec)
    assert all(r[1] == 0 for r in res), res
    assert method == "CG" or max(r[0] for r in res) <= maxit
    assert all(rel2(x[c], X[c]) < 1e-10 for c in range(len(qvec)))


@pytest.mark.parametrize("method,most", [("CG", 12), ("BICGSTAB", 1)])
def test_small_limit_ends(method, most):
    P = workloads.disc(16, 3, 0.0, 8)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    s = capi.FwdSolver(gm, method, 1e-12, "ICH", False, maxit=1, precision="mixed")
    s.reset(cm, ck, ca, 0.0)
    _, res = s.calc_fields(qvec)
    assert all(r[1] == 1 and 0 < r[0] <= most for r in res), res
