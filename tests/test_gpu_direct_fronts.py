"""The direct solver's dense fronts at their edges, against the oracle's direct
solve: a mesh of a single leaf block, one split, fronts of many panels (3D),
right-hand sides that do not fill a CTA's group of 8, and a resolve after a
new reset.  Two exact FP64 solves in different orderings: round-off apart
(1e-13 in L2, as the other direct tests hold it)."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs, rel2
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

MESHES = [("leaf", lambda f: workloads.disc(2, 3, f, 4)), ("split", lambda f: workloads.disc(4, 3, f, 4)),
          ("disc721", lambda f: workloads.disc(15, 3, f, 6)), ("cyl1016", lambda f: workloads.cylinder(6, 8, 3, f))]


@pytest.mark.parametrize("freq", [0.0, 100.0])
@pytest.mark.parametrize("name,factory", MESHES, ids=[m[0] for m in MESHES])
def test_fronts_match_oracle(oracle_mod, name, factory, freq):
    P = factory(freq)
    om = oracle_mod.Mesh(P.coords, P.elems)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    omega = capi.omega_of(freq)
    s = capi.FwdSolver(gm, "DIRECT", 1e-10, "NONE", P.complex)
    for scale in (1.0, 1.3):
        s.reset(cm * scale, ck, ca, omega)
        val = om.assemble(cm * scale, ck, ca, omega, P.complex)
        for k in (1, 7, 8, 17):
            B = np.concatenate([qvec, mvec])[np.arange(k) % (len(qvec) + len(mvec))]
            phi, res = s.calc_fields(B)
            X = oracle_mod.solve_direct(om.rowptr, om.colidx, val, B.astype(phi.dtype), "nd", om.coords)
            assert rel2(phi, X) < 1e-13
            assert all(r[0] == 0 and r[1] == 0 and r[2] < 1e-13 for r in res), res
