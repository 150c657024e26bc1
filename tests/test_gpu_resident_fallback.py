"""Columns that the resident solve cannot finish (here: more residual
replacements than max_outer = 1 allows) go to the batched kernels in a block of
their own; the columns that met their bounds keep their fields and counts."""
import numpy as np
import pytest

from tests.gpu_util import gpu_problem_inputs
from toastpp_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def setup(freq):
    P = workloads.disc(16, 3, freq, 8)
    gm = capi.Mesh(P.coords, P.elems)
    cm, ck, ca, qvec, _ = gpu_problem_inputs(P, gm)
    # point sources take more than 4 replacements of 1e-3, smooth right-hand sides do not
    hard, easy = qvec[:4], np.ones((4, P.n)) + 0.1 * np.arange(4)[:, None]

    def solver(max_outer):
        s = capi.FwdSolver(gm, "BICGSTAB", 1e-8, "ICH", P.complex, precision="mixed")
        s.set_refinement(1e-3, max_outer)
        s.set_backward_error(1e-8)
        s.reset(cm, ck, ca, capi.omega_of(freq))
        return s
    return solver, hard, easy, (cm, ck, ca, capi.omega_of(freq))


@pytest.mark.parametrize("guess", [0.0, 1e-3])
@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_only_failed_columns_are_solved_again(freq, guess):
    solver, hard, easy, _ = setup(freq)
    B = np.empty((8, hard.shape[1]))
    B[0::2], B[1::2] = hard, easy
    whole, res = solver(12).calc_fields(B, phi0=np.full(B.shape, guess))
    assert all(r[1] == 0 for r in res)
    s = solver(1)
    c0 = capi.launch_count()
    part, res1 = s.calc_fields(B, phi0=np.full(B.shape, guess))
    assert capi.launch_count() - c0 > 100          # the batched kernels ran
    assert [r[:2] for r in res1[1::2]] == [r[:2] for r in res[1::2]]
    assert np.array_equal(part[1::2], whole[1::2])
    # the others: what the batched kernels give from the same start, alone
    alone, resa = solver(1).calc_fields(hard, phi0=np.full(hard.shape, guess))
    assert [r[:2] for r in res1[0::2]] == [r[:2] for r in resa]
    assert np.array_equal(part[0::2], alone)


@pytest.mark.parametrize("freq", [0.0, 100.0])
def test_whole_request(freq):
    """The same through the path that starts from zero without reading a guess."""
    solver, hard, easy, args = setup(freq)
    L = capi.Links.all_to_all(len(hard), len(easy))
    a = solver(1).forward_path(*args, hard, easy, L)
    b = solver(1).calc_fields(np.concatenate([hard, easy]))
    assert [r[:2] for r in a["results"]] == [r[:2] for r in b[1]]
    assert np.array_equal(np.concatenate([a["dphi"], a["aphi"]]), b[0])
