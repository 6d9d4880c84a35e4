"""Which form of the iteration a survey gets, whatever was created before it
on the same assembly."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import _lib, survey
from test_gpu_survey_kernels import _problem

pytestmark = pytest.mark.gpu


def _run(torch, A, nus, b):
    """variant, kernel launches, iterations and solution of a survey"""
    sv = survey.Survey(A, nus)
    x = torch.zeros_like(b)
    n0 = _lib.kernel_launches()
    code, st = sv.solve(b, x, verify=False)
    n = _lib.kernel_launches() - n0
    assert code == 0
    out = sv.tuning()[0], n, st["iterations"], x
    sv.close()
    return out


def test_one_system_after_a_survey_of_33(gpu):
    """The 33rd system is a batch of one that runs beside another, so without
    the one-kernel iteration, and its form is chosen by timing.  A single
    small system created afterwards still iterates in one kernel, as it does
    on a fresh assembly."""
    torch = gpu
    nus, alfas = list(np.logspace(-1, 1, 33)), [k % 2 for k in range(33)]
    _, A, b = _problem(torch, "c1", nus, alfas)
    alone = _run(torch, A, nus[:1], b[:1])
    assert alone[0] == 35 and alone[1] < alone[2][0]       # fewer launches than iterations
    many = survey.Survey(A, nus)
    assert many.batches == 2
    many.close()
    again = _run(torch, A, nus[:1], b[:1])
    assert again[:3] == alone[:3] and torch.equal(again[3], alone[3])
    A.close()
