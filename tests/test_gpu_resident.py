"""The mixed path's resident solve (one kernel on thread-block clusters, CG with
a factorised sparse approximate inverse) against the oracle's exact FP64 solve,
at the sizes where its splits change: fewer nodes than a slice of 32 rows, one
CTA and clusters of 2 to 16, odd column counts, columns in a partly filled
cluster, real and complex systems, a nonzero guess, and a zero right-hand side.

Bound: the solve stops at a componentwise backward error of 1e-10, which for
these systems leaves the fields within 1e-10 in L2 (the bound that the other
mixed-path tests use)."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs, rel2, small_cyl
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def disc(rings, freq):
    return workloads.disc(rings, 3, freq, 8)


CASES = [("disc19", lambda f: disc(2, f)), ("disc217", lambda f: disc(8, f)), ("disc331", lambda f: disc(10, f)),
         ("disc1261", lambda f: disc(20, f)), ("disc3169", lambda f: disc(32, f)), ("cyl", lambda f: small_cyl(f)),
         ("cyl4634", lambda f: workloads.cylinder(10, 14, 1, f))]


@pytest.fixture(scope="module", params=CASES, ids=[c[0] for c in CASES])
def mesh(request, oracle_mod):
    P = {f: request.param[1](f) for f in (0.0, 100.0)}
    return P, oracle_mod.Mesh(P[0.0].coords, P[0.0].elems), capi.Mesh(P[0.0].coords, P[0.0].elems)


@pytest.mark.parametrize("freq", [0.0, 100.0])
@pytest.mark.parametrize("k", [1, 3, 16])
def test_fields_match_exact(mesh, oracle_mod, freq, k):
    P, om, gm = mesh[0][freq], mesh[1], mesh[2]
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    omega = capi.omega_of(freq)
    B = np.concatenate([qvec, mvec])[np.arange(k) % (len(qvec) + len(mvec))]
    if k > 1:
        B = B.copy()
        B[1] = 0.0
    val = om.assemble(cm, ck, ca, omega, P.complex)
    X = oracle_mod.solve_direct(om.rowptr, om.colidx, val, B.astype(complex if P.complex else float), "nd", om.coords)
    for method in ("BICGSTAB",) if P.complex else ("BICGSTAB", "CG"):
        s = capi.FwdSolver(gm, method, 1e-12, "ICH", P.complex, precision="mixed")
        s.reset(cm, ck, ca, omega)
        c0 = capi.launch_count()
        phi, res = s.calc_fields(B)
        assert capi.launch_count() - c0 < 40  # one kernel and its preparation, no launch per iteration
        assert all(r[1] == 0 for r in res), res
        assert all(rel2(phi[c], X[c]) < 1e-10 for c in range(k) if np.any(B[c]))
        assert k == 1 or not np.any(phi[1])
        # from a nonzero guess, and from the solution itself
        phi2, res2 = s.calc_fields(B, phi0=0.5 * X + 1e-3 * np.abs(X).max())
        assert all(r[1] == 0 for r in res2), res2
        assert all(rel2(phi2[c], X[c]) < 1e-10 for c in range(k) if np.any(B[c]))


@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_large_blocks_take_the_batched_kernels(oracle_mod, freq):
    """More columns than the on-chip solve takes: the batched kernels, same fields."""
    P = disc(24, freq)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    B = np.concatenate([qvec, mvec])
    k = len(B)
    big = np.tile(B, ((3000 if P.complex else 6000) // k, 1))
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", P.complex, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(freq))
    a, _ = s.calc_fields(B)
    b, res = s.calc_fields(big)
    assert all(r[1] == 0 for r in res)
    assert rel2(b[:k], a) < 1e-10 and rel2(b[-k:], a) < 1e-10


def test_iteration_limit(oracle_mod):
    """A solve cut off by its iteration limit reports it and keeps its count."""
    P = disc(16, 100.0)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", True, maxit=5, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(100.0))
    _, res = s.calc_fields(qvec)
    assert all(r[1] == 1 and 0 < r[0] <= 5 for r in res), res
