"""Counts past one grid dimension's 65535 blocks on the smallest mesh: detectors
of the element Jacobian (tiles of 64) and right-hand sides of the direct solver
(groups of 8)."""
import numpy as np
import pytest

from tests.gpu_util import rel2
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def test_element_detectors(oracle_mod):
    P = workloads.disc(1, 3, 0.0, 4)
    gm = capi.Mesh(P.coords, P.elems)
    nm = 64 * 65535 + 70
    rng = np.random.default_rng(4)
    F, A = rng.uniform(0.5, 1.5, (1, P.n)), rng.uniform(0.5, 1.5, (nm, P.n))
    lm = np.array([0, 64 * 65535 - 1, 64 * 65535, nm - 1], np.int32)
    ofs, y = np.array([0, len(lm)], np.int32), rng.uniform(0.5, 1.5, len(lm))
    s = capi.FwdSolver(gm, "CG", 1e-12, "NONE", False)
    J = s.jacobian_el(F, A, y, capi.Links(ofs, lm))
    ref = oracle_mod.jacobian_el(oracle_mod.Mesh(P.coords, P.elems), F, A[lm], y, ofs, np.arange(len(lm), dtype=np.int32))
    assert rel2(J, ref) < 1e-13  # a sum of 9 products an entry, a few roundings each


def test_direct_right_hand_sides(oracle_mod):
    P = workloads.disc(1, 3, 0.0, 4)
    gm = capi.Mesh(P.coords, P.elems)
    om = oracle_mod.Mesh(P.coords, P.elems)
    cm, ck, ca = capi.optical_coefficients(P.mua, P.mus, P.nref)
    B = np.random.default_rng(5).uniform(0.5, 1.5, (8 * 65535 + 5, P.n))
    s = capi.FwdSolver(gm, "DIRECT", 1e-10, "NONE", False)
    s.reset(cm, ck, ca, 0.0)
    x, res = s.calc_fields(B)
    A = np.zeros((P.n, P.n))
    A[np.repeat(np.arange(P.n), np.diff(om.rowptr)), om.colidx] = om.assemble(cm, ck, ca, 0.0, False)
    assert rel2(x, np.linalg.solve(A, B.T).T) < 1e-13  # two FP64 solves of 7 unknowns
    assert all(r[1] == 0 for r in (res[0], res[-1]))
