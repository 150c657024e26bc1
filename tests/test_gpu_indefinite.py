"""Systems that are not positive definite (negative absorption coefficients,
which an unconstrained reconstruction step can reach): the mixed path solves
them with the batched BiCGSTAB and CG, as it does every block that the resident
CG cannot take.  The residuals are formed here in FP64 from the oracle's
matrix; the solve's bound is 1e-10 |b|, rounding adds about 1e-14 |A||x|."""
import numpy as np
import pytest
import scipy.sparse as sp

from tests.gpu_util import gpu_problem_inputs
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,scale", [("BICGSTAB", -0.2), ("CG", -0.2), ("CG", -0.5), ("CG", -1.0)])
def test_negative_absorption(method, scale, oracle_mod):
    P = workloads.disc(16, 3, 0.0, 8)
    om = oracle_mod.Mesh(P.coords, P.elems)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    val = om.assemble(cm * scale, ck, ca, 0.0, False)
    A = sp.csr_matrix((val, om.colidx, om.rowptr), shape=(P.n, P.n))
    assert sp.linalg.eigsh(A, 1, which="SA", return_eigenvectors=False)[0] < 0
    s = capi.FwdSolver(gm, method, 1e-10, "ICH", False, maxit=400, precision="mixed")
    s.reset(cm * scale, ck, ca, 0.0)
    x, res = s.calc_fields(qvec)
    assert all(r[1] == 0 for r in res), res
    for c in range(len(qvec)):
        r = np.linalg.norm(qvec[c] - A @ x[c])
        assert r <= 1e-10 * np.linalg.norm(qvec[c]) + 1e-14 * np.linalg.norm(abs(A) @ abs(x[c]))
