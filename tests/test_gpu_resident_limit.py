"""The iteration limit of the resident solve: columns of one cluster wait for
each other's corrections, so at the limit some have made fewer iterations than
it.  They report status 1, and nothing solves them again: a cut-off solve takes
the launches of a whole one (the kernel and its preparation), wherever the
limit falls."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("freq,k", [(0.0, 700), (100.0, 400)])
def test_limit_is_no_failure(freq, k):
    P = workloads.disc(16, 3, freq, 8)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    rng = np.random.default_rng(5)
    # point sources and smooth right-hand sides: they reach their triggers at different iterations
    B = np.concatenate([qvec, mvec, rng.random((k - len(qvec) - len(mvec), P.n)) ** rng.uniform(0, 40, (k - len(qvec) - len(mvec), 1))])
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", P.complex, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(freq))
    s.calc_fields(B)

    def run(maxit):
        s.set_tol(1e-12, maxit)
        c0 = capi.launch_count()
        _, res = s.calc_fields(B)
        return capi.launch_count() - c0, res

    whole, res = run(0)
    assert all(r[1] == 0 for r in res)
    waited = 0
    for maxit in range(3, 1 + max(r[0] for r in res)):
        n, res = run(maxit)
        assert n == whole, (maxit, n, whole)
        assert all(r[1] in (0, 1) and r[0] <= maxit for r in res)
        waited += sum(r[1] == 1 and r[0] < maxit for r in res)
    assert waited > 0  # the case is there
