"""The one-kernel iterations when a wait of their grid barrier runs out: the
solve fails whatever block it was and at whatever barrier, and the next solve
on the same object is right."""
import pytest

from mtcalc_with_dfp_cocr_gb300 import _lib, assembly, survey
from test_gpu_survey_kernels import _ragged

pytestmark = pytest.mark.gpu

POLLS = [1, 2, 4, 8, 16, 32, 64, 128, 256, 512, 1024]


def _failures(torch, monkeypatch, solve, bounds=POLLS):
    """solve() -> its outputs.  With the waits bounded to a few polls a solve
    either raises or gives what it gives otherwise."""
    ref = solve()
    failed = []
    for polls in bounds:
        monkeypatch.setenv("MTGPU_BARRIER_POLLS", str(polls))
        try:
            out = solve()
        except _lib.MtgpuError as e:
            assert "grid barrier" in str(e) and str(_lib.MTGPU_ERR_TIMEOUT) in str(e)
            failed.append(polls)
        else:
            assert out[0] == ref[0] and torch.equal(out[1], ref[1]), polls
        monkeypatch.delenv("MTGPU_BARRIER_POLLS")
        if failed and failed[-1] == polls:
            out = solve()
            assert out[0] == ref[0] and torch.equal(out[1], ref[1]), polls
    return failed


@pytest.mark.parametrize("cells,S", [((24, 24, 25), 2), ((31, 27, 22), 1), ((14, 13, 12), 8)])
def test_survey_wait_runs_out(gpu, monkeypatch, cells, S):
    torch = gpu
    m, nus, b = _ragged(torch, cells, S, 3)
    A = assembly.Assembly(m)
    sv = survey.Survey(A, nus)
    sv.set_spmv_variant(35)

    def solve():
        x = torch.zeros_like(b)
        code, st = sv.solve(b, x, eps=1e-6, maxiter=2000, verify=False)
        assert code == 0
        return (st["iterations"], st["residual_rel"]), x

    # (the first wait, to its bound of two seconds)
    assert _failures(torch, monkeypatch, solve, [1, 1]) == [1, 1]
    sv.close()
    A.close()


@pytest.mark.parametrize("cells", [(14, 13, 12), (24, 24, 25)])
def test_fp64_wait_runs_out(gpu, monkeypatch, cells):
    torch = gpu
    m, nus, b = _ragged(torch, cells, 1, 3)
    A = assembly.Assembly(m)
    cx = A.cocr(nus[0])

    def solve():
        x = torch.zeros_like(b[0])
        code, st = cx.solve(b[0], x, eps=1e-6, maxiter=2000)
        assert code == 0
        return (st.iterations, st.residual_rel), x

    # one poll is over before the other blocks have arrived
    assert 1 in _failures(torch, monkeypatch, solve)
    cx.close()
    A.close()
