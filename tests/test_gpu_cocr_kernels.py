"""The FP64 solver's one-kernel iterations where their sizes turn: one block,
1, 2 and 3 rows a thread, the separate kernels beyond (218,880 rows), and
launches of any number of iterations."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import assembly, survey
from test_gpu_survey_kernels import _ragged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(2, 2, 2), (4, 9, 3), (24, 24, 25), (33, 31, 32), (41, 42, 40),
                                   (42, 42, 43)])
def test_fp64_iterations(gpu, cells):
    """The solution reaches the true residual, which another kernel evaluates;
    the count is the double-float solver's within 3 (the bound the survey's
    tests hold the two to); and neither depends on how many iterations a
    launch runs, to the last bit."""
    torch = gpu
    m, nus, b = _ragged(torch, cells, 1, sum(cells))
    A = assembly.Assembly(m)
    cx = A.cocr(nus[0])
    runs = []
    for ipl in (0, 1, 7):
        x = torch.zeros_like(b[0])
        code, st = cx.solve(b[0], x, eps=1e-8, maxiter=4000, iterations_per_launch=ipl)
        assert code == 0
        runs.append((st.iterations, st.residual_rel, st.true_residual_rel, x))
    for r in runs[1:]:
        assert r[:3] == runs[0][:3] and torch.equal(r[3], runs[0][3])
    x = torch.zeros_like(b[0])
    code, st = cx.solve(b[0], x, eps=1e-8, maxiter=4000, stop_on_true_residual=True)
    y = torch.empty_like(x)
    cx.spmv(x, y)
    assert code == 0 and float((b[0] - y).norm() / b[0].norm()) < 1.0001e-8
    sv = survey.Survey(A, nus)
    _, s32 = sv.solve(b, torch.zeros_like(b), eps=1e-8, maxiter=4000, verify=False)
    assert abs(s32["iterations"][0] - runs[0][0]) <= 3
    # out of iterations: the state after exactly maxiter of them
    code, st = cx.solve(b[0], torch.zeros_like(b[0]), eps=1e-30, maxiter=3)
    assert code == -3 and st.iterations == 4
    sv.close()
    cx.close()
    A.close()
