"""Memory of surveys of several batches."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import survey
from test_gpu_survey_kernels import _problem

pytestmark = pytest.mark.gpu


def test_batches_that_fit_without_groups(gpu):
    """Four batches of 32 systems in the memory that they take with the s
    vectors of one iteration each: the first ones leave the last ones theirs,
    and the counts and residuals are those of a survey with room."""
    torch = gpu
    S = 128
    nus, alfas = list(np.repeat(np.logspace(-1, 1, S // 2), 2)), [1, 0] * (S // 2)
    w, A, b = _problem(torch, "c1", nus, alfas)
    x = torch.zeros_like(b)
    survey.Survey(A, nus[:32]).close()      # what a first survey loads stays loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    vec = 16 * 32 * w.mesh.nb
    free = torch.cuda.mem_get_info()[0]
    sv = survey.Survey(A, nus)
    used = free - torch.cuda.mem_get_info()[0]
    assert sv.batches == 4 and used > 4 * 17 * vec      # groups of 16
    ref = sv.solve(b, x, verify=False)
    sv.close()
    short = used - 4 * 15 * vec + (100 << 20)
    filler = torch.empty(torch.cuda.mem_get_info()[0] - short, dtype=torch.uint8, device="cuda")
    sv = survey.Survey(A, nus)
    x.zero_()
    got = sv.solve(b, x, verify=False)
    sv.close()
    del filler
    torch.cuda.empty_cache()
    assert got[0] == ref[0] == 0
    assert got[1]["iterations"] == ref[1]["iterations"]
    assert got[1]["residual_rel"] == ref[1]["residual_rel"]
    assert max(got[1]["true_residual_rel"]) < 1e-7
    A.close()
