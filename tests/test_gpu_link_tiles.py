"""The link tiles of the grid and element Jacobian kernels: source groups of 8
and 4 with remainders, detector chunks of 4 to 64, links missing at random,
against the oracle.  An entry is a sum of at most 16 products of a few roundings
each: 1e-13 (FP64) is 1000 of them, 2e-6 (FP32) is 32 of 2^-24."""
import numpy as np
import pytest

from tests.golden_util import load
from tests.gpu_util import rel2
from toastpp_gb300 import capi

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1.0), (5, 3, 1.0), (8, 5, 0.6), (9, 17, 1.0), (16, 63, 0.5), (7, 64, 1.0), (17, 65, 0.7), (2, 130, 0.05)]


def fields(name, nq, nm, share):
    g = load(name)
    rng = np.random.default_rng(1000 * nq + nm)
    n = len(g["coords"])
    cplx = np.iscomplexobj(g["proj"])

    def draw(*shape):
        x = rng.uniform(0.5, 1.5, shape)
        return x * np.exp(1j * rng.uniform(-0.5, 0.5, shape)) if cplx else x
    pick = rng.random((nq, nm)) < share
    ofs = np.concatenate([[0], np.cumsum(pick.sum(1))]).astype(np.int32)
    lm = np.nonzero(pick)[1].astype(np.int32)
    return g, draw(nq, n), draw(nm, n), draw(max(1, len(lm)))[:len(lm)], ofs, lm


def compare(J, J32, ref):
    assert J.shape == ref.shape
    assert rel2(J, ref) < 1e-13
    assert rel2(J32.astype(np.float64), ref) < 2e-6


@pytest.mark.parametrize("nq,nm,share", SIZES)
@pytest.mark.parametrize("name", ["disc_cw_el", "disc_fd_el", "cyl_cw_el", "cyl_fd_el"])
def test_element_links_against_oracle(name, nq, nm, share, oracle_mod):
    g, F, A, proj, ofs, lm = fields(name, nq, nm, share)
    if len(lm) == 0:
        pytest.skip("no link drawn")
    gm = capi.Mesh(g["coords"], g["elems"])
    s = capi.FwdSolver(gm, g["solver"], 1e-12, g["precon"], np.iscomplexobj(F))
    L = capi.Links(ofs, lm)
    ref = oracle_mod.jacobian_el(oracle_mod.Mesh(g["coords"], g["elems"]), F, A, proj, ofs, lm)
    compare(s.jacobian_el(F, A, proj, L), s.jacobian_el(F, A, proj, L, fp32=True), ref)


@pytest.mark.parametrize("nq,nm,share", SIZES)
@pytest.mark.parametrize("name", ["disc_cw_grid", "disc_fd_grid", "cyl_cw_grid", "cyl_fd_grid"])
def test_grid_links_against_oracle(name, nq, nm, share, oracle_mod):
    g, F, A, proj, ofs, lm = fields(name, nq, nm, share)
    if len(lm) == 0:
        pytest.skip("no link drawn")
    gm = capi.Mesh(g["coords"], g["elems"])
    s = capi.FwdSolver(gm, g["solver"], 1e-12, g["precon"], np.iscomplexobj(F))
    r, L = capi.Raster(gm, g["bdim"]), capi.Links(ofs, lm)
    ref = oracle_mod.jacobian_grid(oracle_mod.Mesh(g["coords"], g["elems"]), g["bdim"], F, A, proj, ofs, lm)
    compare(s.jacobian_grid(r, F, A, proj, L), s.jacobian_grid(r, F, A, proj, L, fp32=True), ref)
