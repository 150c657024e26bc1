"""How an IC(0) apply runs is a matter of sizes alone: the same solve takes the
same launches whatever was solved before it, and the first solve of a column
count takes no more than the next (nothing is timed)."""
import numpy as np
import pytest

from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_no_timed_choice(freq, monkeypatch):
    monkeypatch.delenv("TOASTGPU_IC_PERSISTENT", raising=False)
    P = workloads.disc(24, 3, freq, 8)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca = capi.optical_coefficients(P.mua, P.mus, P.nref)
    B = np.random.default_rng(2).random((200, P.n))

    def launches(k):
        s = capi.FwdSolver(gm, "BICGSTAB", 1e-10, "ICH", P.complex, maxit=3, precision="fp64")
        s.reset(cm, ck, ca, capi.omega_of(freq))
        c0 = capi.launch_count()
        s.calc_fields(B[:k])
        return capi.launch_count() - c0

    first = {k: launches(k) for k in (1, 40, 200)}
    assert first == {k: launches(k) for k in (200, 40, 1)}
    # on clusters: far fewer than a launch per level
    levels = []
    for mode in ("0", "1"):
        monkeypatch.setenv("TOASTGPU_IC_PERSISTENT", mode)
        levels.append(launches(40))
    assert first[40] == levels[1] < levels[0]
