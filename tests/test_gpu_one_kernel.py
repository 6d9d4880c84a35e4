"""Which problems iterate in one kernel, by the launches of a solve: the
separate kernels of a group of 16 iterations are five an iteration and one
for p and x, the one kernel's group two; in FP64 four an iteration and one a
launch of 64."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import _lib, assembly, survey
from test_gpu_survey_kernels import SMALL, _ragged

pytestmark = pytest.mark.gpu


def _survey_launches(torch, cells, S):
    """(kernel launches, groups of 16 iterations) of a solve with variant 35"""
    m, nus, b = _ragged(torch, cells, S, 1)
    A = assembly.Assembly(m)
    sv = survey.Survey(A, nus)
    sv.set_spmv_variant(35)
    n0 = _lib.kernel_launches()
    code, st = sv.solve(b, torch.zeros_like(b), eps=1e-5, maxiter=1000, verify=False)
    n = _lib.kernel_launches() - n0
    assert code == 0
    sv.close()
    A.close()
    return n, -(-max(st["iterations"]) // 16)


def _fp64_launches(torch, cells):
    m, nus, b = _ragged(torch, cells, 1, 1)
    A = assembly.Assembly(m)
    cx = A.cocr(nus[0])
    n0 = _lib.kernel_launches()
    code, st = cx.solve(b[0], torch.zeros_like(b[0]), eps=1e-5, maxiter=1000)
    n = _lib.kernel_launches() - n0
    assert code == 0
    cx.close()
    A.close()
    return n, st.iterations


@pytest.mark.parametrize("cells,S", SMALL + [((14, 14, 14), 9)])
def test_survey(gpu, cells, S):
    n, groups = _survey_launches(gpu, cells, S)
    # beyond 218,880 rows x systems, and with more than 8 lanes, the separate kernels
    if (cells, S) in (SMALL[-1], ((14, 14, 14), 9)):
        assert n >= 81 * groups
    else:
        assert n <= 2 * groups + 16


@pytest.mark.parametrize("cells", [(2, 2, 2), (14, 13, 12), (33, 31, 32), (41, 42, 40), (42, 42, 43)])
def test_fp64(gpu, cells):
    n, its = _fp64_launches(gpu, cells)
    if cells == (42, 42, 43):
        assert n >= 4 * its
    else:
        assert n <= -(-its // 64) + 16


def test_separate_kernels_on_request(gpu, monkeypatch):
    """For programs that run many small solves from several threads."""
    monkeypatch.setenv("MTGPU_ONE_KERNEL", "0")
    n, groups = _survey_launches(gpu, (17, 16, 15), 5)
    assert n >= 81 * groups
    n, its = _fp64_launches(gpu, (14, 13, 12))
    assert n >= 4 * its
