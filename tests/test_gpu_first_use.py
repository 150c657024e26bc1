"""Data that a mesh builds at its first use (the partitions of the cluster
kernels): solvers of two threads that meet on a new mesh get the fields that
one solver alone gets, to the last bit."""
import threading

import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_two_threads_on_a_new_mesh(freq, precision, monkeypatch):
    monkeypatch.setenv("TOASTGPU_IC_PERSISTENT", "1")
    P = workloads.disc(20, 3, freq, 8)

    def solve(gm, inputs, out, i):
        cm, ck, ca, qvec, _ = inputs
        s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", P.complex, precision=precision)
        s.reset(cm, ck, ca, capi.omega_of(freq))
        out[i] = s.calc_fields(qvec)[0]

    ref = [None]
    gm = capi.Mesh(P.coords, P.elems)
    solve(gm, gpu_problem_inputs(P, gm), ref, 0)
    for _ in range(3):
        gm = capi.Mesh(P.coords, P.elems)
        inputs = gpu_problem_inputs(P, gm)
        out = [None, None]
        threads = [threading.Thread(target=solve, args=(gm, inputs, out, i)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(o is not None and np.array_equal(o, ref[0]) for o in out)
