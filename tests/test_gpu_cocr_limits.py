"""The FP64 solver where it runs out of something: iterations, when it stops
on the true residual; range, where the squares of its sums pass FP64's."""
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


@pytest.mark.parametrize("cells", [(14, 13, 12), (33, 31, 32), (42, 42, 43)])
@pytest.mark.parametrize("e", [-60, 300, 450])
def test_right_hand_sides_of_any_size(gpu, cells, e):
    """Every operation scales exactly with the right-hand side: b 2^e gives x
    2^e, also where (a, w) and (z, s) are beyond 1e154 and their squares
    beyond FP64's range.  Small ones end in the reference's breakdown test,
    (a, w) < 1e-40, whose bound does not scale."""
    torch = gpu
    m, nus, b = _ragged(torch, cells, 1, 2)
    A = assembly.Assembly(m)
    cx = A.cocr(nus[0])
    out = []
    for scale in (1.0, 2.0 ** e):
        x = torch.zeros_like(b[0])
        code, st = cx.solve(b[0] * scale, x, eps=1e-5, maxiter=2000)
        out.append((code, st.iterations, st.residual_rel, x / scale))
    assert out[0][0] == 0
    if e < 0:
        assert out[1][0] == -2
    else:
        assert out[0][:3] == out[1][:3] and torch.equal(out[0][3], out[1][3])
    cx.close()
    A.close()
