"""The FP64 solver where it runs out of something: iterations, when it stops
on the true residual."""
import pytest

from mtcalc_with_dfp_cocr_gb300 import assembly
from test_gpu_survey_kernels import _ragged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,eps", [((4, 9, 3), 1e-3), ((14, 13, 12), 1e-4), ((24, 24, 25), 1e-6),
                                       ((33, 31, 32), 1e-8), ((42, 42, 43), 1e-6)])
def test_true_residual_with_few_iterations(gpu, cells, eps):
    """The smoothed residual passes eps a few iterations before the true one
    on these systems.  With maxiter from just before the first stop to beyond
    the second, and any launch length, the call either reaches the true
    residual within maxiter or says that it ran out."""
    torch = gpu
    m, nus, b = _ragged(torch, cells, 1, sum(cells))
    A = assembly.Assembly(m)
    cx = A.cocr(nus[0])

    def solve(maxiter, true, ipl):
        x = torch.zeros_like(b[0])
        code, st = cx.solve(b[0], x, eps=eps, maxiter=maxiter, stop_on_true_residual=true,
                            iterations_per_launch=ipl)
        return code, st.iterations, st.true_residual_rel, x

    first, last = solve(4000, False, 1), solve(4000, True, 1)
    assert first[0] == last[0] == 0 and first[1] < last[1] and last[2] < eps <= first[2]
    for maxiter in sorted({first[1] - 1, first[1], last[1] - 1, last[1], last[1] + 5, 200}):
        for ipl in (0, 1, 16, 64):
            code, it, res, x = solve(maxiter, True, ipl)
            if maxiter >= last[1]:
                assert (code, it, res) == (0, last[1], last[2]) and torch.equal(x, last[3])
            else:
                assert code == -3 and it == maxiter + 1 and res >= eps
    cx.close()
    A.close()
