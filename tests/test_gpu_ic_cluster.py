"""The IC(0) apply of the batched methods on thread-block clusters against the
launch-per-level kernels: both add the same products in the same order, so the
iterations and the fields are the same to the last bit.  Sizes: one CTA to a
whole cluster, levels of a few rows, column counts that leave a cluster's last
group partly filled."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs, small_cyl
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

CASES = [("disc19", lambda f: workloads.disc(2, 3, f, 8)), ("disc217", lambda f: workloads.disc(8, 3, f, 8)),
         ("disc1261", lambda f: workloads.disc(20, 3, f, 8)), ("cyl", lambda f: small_cyl(f)),
         ("cyl4634", lambda f: workloads.cylinder(10, 14, 1, f))]


@pytest.mark.parametrize("make", [c[1] for c in CASES], ids=[c[0] for c in CASES])
@pytest.mark.parametrize("freq,method,precision", [(100.0, "BICGSTAB", "fp64"), (100.0, "GMRES", "fp64"),
                                                   (0.0, "CG", "fp64"), (0.0, "BICGSTAB", "fp64"),
                                                   (100.0, "GMRES", "mixed")])
def test_cluster_sweep_is_bit_identical(make, freq, method, precision, monkeypatch):
    P = make(freq)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    src = np.concatenate([qvec, mvec])
    for k in (1, 3, 7, 33):
        B = src[np.arange(k) % len(src)] * (1.0 + 0.1 * np.arange(k))[:, None]
        out = []
        for mode in ("0", "1"):
            monkeypatch.setenv("TOASTGPU_IC_PERSISTENT", mode)
            s = capi.FwdSolver(gm, method, 1e-10, "ICH", P.complex, precision=precision)
            s.reset(cm, ck, ca, capi.omega_of(freq))
            out.append(s.calc_fields(B))
        assert [r[:2] for r in out[0][1]] == [r[:2] for r in out[1][1]]
        assert np.array_equal(out[0][0], out[1][0])
