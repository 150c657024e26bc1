"""CG requests of the mixed path take their true residuals from FP64 products,
and the norm that they report from squares of more than FP32: |b - A x| / |b|
as reported against the same formed in extended precision from the returned
field.  Bound: a row's product of at most 12 terms and a difference in FP64,
13 2^-53 (|A||x| + |b|), and 2^-40 of the norm itself for its sum in pairs of
floats (about 2^-46 a term)."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rings", [16, 32, 48])
@pytest.mark.parametrize("tol", [1e-3, 1e-5, 1e-10])
def test_reported_residual(rings, tol):
    P = workloads.disc(rings, 3, 0.0, 8)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    s = capi.FwdSolver(gm, "CG", tol, "ICH", False, precision="mixed")
    s.set_backward_error(0.0)
    s.reset(cm, ck, ca, 0.0)
    rp, ci = gm.csr()
    assert np.max(np.diff(rp)) <= 12
    row = np.repeat(np.arange(P.n), np.diff(rp))
    val = s.system_matrix().astype(np.longdouble)
    x, res = s.calc_fields(qvec)
    for c in range(len(qvec)):
        b, y = qvec[c].astype(np.longdouble), x[c].astype(np.longdouble)
        ax, mag = np.zeros((2, P.n), np.longdouble)
        np.add.at(ax, row, val * y[ci])
        np.add.at(mag, row, abs(val * y[ci]))
        norm = lambda v: float(np.sqrt((v * v).sum()))
        nr, nb = norm(b - ax), norm(b)
        assert abs(res[c][2] * nb - nr) <= 13 * 2.0 ** -53 * norm(mag + abs(b)) + 2.0 ** -40 * nr
