"""The mixed path's batched kernels on meshes that the resident solve would
take (TOASTGPU_RESIDENT=0), and the resident solve at the ends of its range:
whole clusters of 16, tolerances that ask for FP64 residuals, and a mesh whose
rows its preconditioner does not hold."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs, rel2
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu

IC_CASES = [("cyl_fd", lambda: workloads.cylinder(rings=6, layers=8, seed=3)),   # 80 + 80 optodes: k = 160
            ("disc_cw", lambda: workloads.disc(24, 2, 0.0, 16))]                  # 16 + 16: k = 32


@pytest.mark.parametrize("factory", [c[1] for c in IC_CASES], ids=[c[0] for c in IC_CASES])
def test_ic_apply_variants_bit_identical(factory, monkeypatch):
    """A launch per level and one launch on clusters, in the batched processes."""
    monkeypatch.setenv("TOASTGPU_RESIDENT", "0")
    P = factory()
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    L = capi.Links(P.qm.link_ofs, P.qm.link_m)
    method = "BICGSTAB" if P.complex else "CG"
    outs, launches = [], []
    for v in ("0", "1"):
        monkeypatch.setenv("TOASTGPU_IC_PERSISTENT", v)
        s = capi.FwdSolver(gm, method, 1e-12, "ICH", P.complex, precision="mixed")
        c0 = capi.launch_count()
        outs.append(s.forward_path(cm, ck, ca, capi.omega_of(P.freq_mhz), qvec, mvec, L))
        launches.append(capi.launch_count() - c0)
    assert launches[0] > launches[1] > 100  # two ways, neither the resident kernel
    for key in ("dphi", "aphi", "proj", "J"):
        assert np.array_equal(np.asarray(outs[0][key]), np.asarray(outs[1][key])), key
    assert [r[:2] for r in outs[0]["results"]] == [r[:2] for r in outs[1]["results"]]


def exact(om, oracle_mod, P, cm, ck, ca, B):
    val = om.assemble(cm, ck, ca, capi.omega_of(P.freq_mhz), P.complex)
    return oracle_mod.solve_direct(om.rowptr, om.colidx, val, B.astype(complex if P.complex else float), "nd", om.coords)


@pytest.mark.parametrize("freq,method,mode", [(100.0, "BICGSTAB", 2), (100.0, "BICGSTAB", 1), (0.0, "BICGSTAB", 2),
                                              (0.0, "BICGSTAB", 0), (0.0, "CG", 2)])
@pytest.mark.parametrize("k", [3, 40])
def test_processes_match_exact(freq, method, mode, k, oracle_mod, monkeypatch):
    monkeypatch.setenv("TOASTGPU_RESIDENT", "0")
    P = workloads.disc(24, 3, freq, 20)
    om, gm = oracle_mod.Mesh(P.coords, P.elems), capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, mvec = gpu_problem_inputs(P, gm)
    B = np.concatenate([qvec, mvec])[:k]
    X = exact(om, oracle_mod, P, cm, ck, ca, B)
    s = capi.FwdSolver(gm, method, 1e-12, "ICH", P.complex, precision="mixed")
    s.set_reliable_updates(mode)
    s.reset(cm, ck, ca, capi.omega_of(freq))
    c0 = capi.launch_count()
    x, res = s.calc_fields(B)
    assert capi.launch_count() - c0 > 100
    assert all(r[1] == 0 for r in res), res
    # a componentwise backward error of 1e-10, as the resident solve's tests hold it
    assert all(rel2(x[c], X[c]) < 1e-10 for c in range(k))


@pytest.mark.parametrize("resident", ["0", "1"])
@pytest.mark.parametrize("freq,method", [(100.0, "BICGSTAB"), (0.0, "BICGSTAB"), (0.0, "CG")])
def test_tolerance_below_the_float_float_residual(freq, method, resident, oracle_mod, monkeypatch):
    monkeypatch.setenv("TOASTGPU_RESIDENT", resident)
    P = workloads.disc(12, 3, freq, 8)
    om, gm = oracle_mod.Mesh(P.coords, P.elems), capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    X = exact(om, oracle_mod, P, cm, ck, ca, qvec)
    s = capi.FwdSolver(gm, method, 5e-14, "ICH", P.complex, precision="mixed")
    s.set_backward_error(5e-14)
    s.reset(cm, ck, ca, capi.omega_of(freq))
    x, res = s.calc_fields(qvec)
    assert all(r[1] == 0 and r[2] <= 5e-14 for r in res), res
    # 2000 times finer than the bound that leaves the fields within 1e-10
    assert all(rel2(x[c], X[c]) < 1e-12 for c in range(len(qvec)))


@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_whole_clusters_of_16(freq, oracle_mod):
    P = workloads.cylinder(12, 16, 1, freq)  # 7504 nodes: two rounds of rows for 8 CTAs, one for 16
    om, gm = oracle_mod.Mesh(P.coords, P.elems), capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", P.complex, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(freq))
    log0 = capi.tuner_log()
    x, res = s.calc_fields(qvec[:2])
    assert "k=2: resident solve" in capi.tuner_log()[len(log0):] and "16 CTAs" in capi.tuner_log()[len(log0):]
    X = exact(om, oracle_mod, P, cm, ck, ca, qvec[:2])
    assert all(r[1] == 0 for r in res) and all(rel2(x[c], X[c]) < 1e-10 for c in range(2))


@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_hub_with_many_neighbours(freq, oracle_mod):
    """A wheel of 120 spokes: the hub has more neighbours before it in the layout
    than a row of the approximate inverse holds, so the batched kernels run."""
    m = 120
    a = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(a), np.sin(a)], 1)
    coords = np.concatenate([[[0.0, 0.0]], 4 * ring, 8 * ring])
    i, j = 1 + np.arange(m), 1 + (np.arange(m) + 1) % m
    elems = np.concatenate([np.stack([0 * i, i, j], 1), np.stack([i, i + m, j], 1),
                            np.stack([j, i + m, j + m], 1)]).astype(np.int32)
    n = len(coords)
    om, gm = oracle_mod.Mesh(coords, elems), capi.Mesh(coords, elems)
    cm, ck, ca = capi.optical_coefficients(np.full(n, 0.02), np.full(n, 1.0), np.full(n, 1.4))
    B = np.random.default_rng(3).random((5, n))
    val = om.assemble(cm, ck, ca, capi.omega_of(freq), freq > 0)
    X = oracle_mod.solve_direct(om.rowptr, om.colidx, val, B.astype(complex if freq else float), "nd", om.coords)
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-12, "ICH", freq > 0, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(freq))
    c0 = capi.launch_count()
    x, res = s.calc_fields(B)
    assert capi.launch_count() - c0 > 40
    assert all(r[1] == 0 for r in res) and all(rel2(x[c], X[c]) < 1e-10 for c in range(5))


@pytest.mark.parametrize("freq,mb", [(0.0, 20), (100.0, 14)])
def test_block_size_rule(freq, mb):
    """Past the rule's line (20 MB of vector; 14 for complex values on a 3D mesh
    of more than 18000 nodes) the batched kernels run, up to it the resident one."""
    P = workloads.box(27, 27, 25, seed=1, nq=64, freq_mhz=freq)
    assert P.n > 18000
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    s = capi.FwdSolver(gm, "BICGSTAB", 1e-10, "ICH", P.complex, maxit=2, precision="mixed")
    s.reset(cm, ck, ca, capi.omega_of(freq))
    line = (mb << 20) // (P.n * (8 if P.complex else 4))
    for k, resident in ((line, True), (line + 1, False)):
        c0 = capi.launch_count()
        s.calc_fields(qvec[np.arange(k) % len(qvec)])
        assert (capi.launch_count() - c0 < 20) == resident, (k, capi.launch_count() - c0)
