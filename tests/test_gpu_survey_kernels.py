"""The survey solver's kernels where their sizes and ranges turn: the
matrix-free products on meshes of a few cells, odd extents and chunk
remainders; grid sums near FP32's largest values; groups of fewer than 16
iterations where memory is short."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import _lib, assembly, normal1d, survey, workloads
from mtcalc_with_dfp_cocr_gb300.mesh import Layer, layered_model
from test_matfree_formula import assembled

pytestmark = pytest.mark.gpu


def _lines(rng, n, lo):
    return lo + np.concatenate([[0.0], np.cumsum(rng.uniform(40.0, 160.0, n))])


@pytest.mark.parametrize("cells,S", [
    ((2, 2, 2), 1), ((2, 2, 2), 32), ((2, 3, 17), 2), ((17, 2, 5), 3), ((16, 16, 4), 1),
    ((5, 33, 3), 8), ((13, 7, 18), 16), ((3, 17, 16), 32), ((33, 3, 2), 5)])
def test_matrix_free_products_on_ragged_meshes(gpu, cells, S):
    """Variants 32, 33 and 35 against the assembled matrix, row by row.  A
    row is at most 33 products of 48-bit factors and as many sums, each
    within 2^-47 of the sum of the terms' magnitudes: 64 2^-47 (|A| |x|)."""
    torch = gpu
    rng = np.random.default_rng(sum(cells) + S)
    x, y = _lines(rng, cells[0], -300.0), _lines(rng, cells[1], -500.0)
    z = _lines(rng, cells[2], 0.0)
    z -= z[max(1, cells[2] - 1)]
    m = layered_model(x, y, z, [Layer(0.0, 0.01)],
                      cell_sigma=10.0 ** rng.uniform(-3, 0, int(np.prod(cells))))
    nus = list(10.0 ** rng.uniform(-2, 2, S))
    A = assembly.Assembly(m)
    sv = survey.Survey(A, nus)
    v = rng.standard_normal((S, m.nb)) + 1j * rng.standard_normal((S, m.nb))
    xd = torch.from_numpy(v.view(np.float64)).cuda()
    yd = torch.empty_like(xd)
    mats = [assembled(m, 2.0 * np.pi * nu)[0] for nu in nus]
    for variant in (32, 33, 35):
        if variant == 33 and S == 1:
            continue
        sv.set_spmv_variant(variant)
        sv.spmv(xd, yd)
        got = yd.cpu().numpy().view(np.complex128)
        for k in range(S):
            bound = 64 * 2.0 ** -47 * (abs(mats[k]) @ abs(v[k]))
            assert np.all(np.abs(got[k] - mats[k] @ v[k]) <= bound), (variant, k)
    sv.close()
    A.close()


def _problem(torch, name, nus, alfas):
    w = workloads.make(name)
    tops, sig = [l.top for l in w.mesh.layers], [l.sigma for l in w.mesh.layers]
    tabs = [normal1d.solve_1d(nu, tops, sig) for nu in nus]
    A = assembly.Assembly(w.mesh)
    b = torch.empty(len(nus), 2 * w.mesh.nb, dtype=torch.float64, device="cuda")
    A.rhs(nus, alfas, tabs[0][0], np.stack([t[1] for t in tabs]), np.stack([t[2] for t in tabs]), b)
    return w, A, b


@pytest.mark.parametrize("S", [1, 2, 4, 9])
def test_sums_near_fp32_range(gpu, S):
    """Right-hand sides times a power of two: every operation of the solver
    scales exactly, so the solutions do too, also where the squares of the
    residual pass 2^100 and the sums over threads are carried scaled down."""
    torch = gpu
    nus, alfas = list(np.logspace(-1, 1, S)), [k % 2 for k in range(S)]
    _, A, b = _problem(torch, "small", nus, alfas)
    b *= 2.0 ** (20 - np.floor(np.log2(b.abs().max().item())))
    sv = survey.Survey(A, nus)
    out = []
    for e in (0, 36):
        x = torch.zeros_like(b)
        code, st = sv.solve(b * 2.0 ** e, x, verify=False)
        assert code == 0
        out.append((x, st["iterations"]))
    assert (b * 2.0 ** 36).square().max().item() > 2.0 ** 100
    assert out[0][1] == out[1][1]
    assert torch.equal(out[0][0] * 2.0 ** 36, out[1][0])
    sv.close()
    A.close()


def test_shorter_groups_where_memory_is_short(gpu):
    """With little free memory the solver keeps the s vectors of fewer
    iterations and applies p and x more often: more launches, and the same
    iteration, which reads neither, so its counts and residuals are the same
    to the last bit; x reaches the true residual."""
    torch = gpu
    nus, alfas = list(np.repeat(np.logspace(-1, 1, 16), 2)), [1, 0] * 16
    _, A, b = _problem(torch, "c1", nus, alfas)
    res = []
    for short in (False, True):
        filler = None
        torch.cuda.empty_cache()
        if short:
            filler = torch.empty(torch.cuda.mem_get_info()[0] - (1400 << 20), dtype=torch.uint8,
                                 device="cuda")
        sv = survey.Survey(A, nus)
        sv.set_spmv_variant(32)
        n0 = _lib.kernel_launches()
        code, st = sv.solve(b, torch.zeros_like(b), verify=False)
        assert code == 0
        res.append((st["iterations"], st["residual_rel"], _lib.kernel_launches() - n0))
        code, st = sv.solve(b, torch.zeros_like(b), verify=True)
        assert code == 0 and max(st["true_residual_rel"]) < 1e-8
        sv.close()
        del filler
    assert res[0][:2] == res[1][:2]
    assert res[1][2] > res[0][2]
    A.close()
    torch.cuda.empty_cache()


# cells and systems with 1, 2 and 3 rows x systems a thread in the one-kernel
# iteration, single blocks, and one beyond its range (218,880 rows x systems)
SMALL = [((2, 2, 2), 1), ((3, 2, 5), 8), ((4, 9, 3), 3), ((17, 16, 15), 5), ((31, 27, 22), 1),
         ((24, 24, 25), 2), ((33, 31, 32), 2), ((33, 34, 32), 2)]


def _ragged(torch, cells, S, seed):
    rng = np.random.default_rng(seed)
    x, y = _lines(rng, cells[0], -300.0), _lines(rng, cells[1], -500.0)
    z = _lines(rng, cells[2], 0.0)
    z -= z[max(1, cells[2] - 1)]
    m = layered_model(x, y, z, [Layer(0.0, 0.01)],
                      cell_sigma=10.0 ** rng.uniform(-3, 0, int(np.prod(cells))))
    nus = list(10.0 ** rng.uniform(0, 2, S))
    b = torch.from_numpy(rng.standard_normal((S, 2 * m.nb))).cuda()
    return m, nus, b


@pytest.mark.parametrize("cells,S", SMALL)
def test_iterations_in_one_kernel(gpu, cells, S):
    """Variant 35 of a small problem runs its iterations in one kernel.  After
    5 iterations the residuals are those of variant 32's separate kernels: a
    wrong or missing term shows at 1e-3; rounding (2^-46 an operation) stays
    below 1e-7 unless the sums cancel by 2^20, and below 5 x 64 2^-46 of |b|
    where nothing but rounding is left of the residual.  Solved to 1e-6 the
    counts are variant 32's within the 3 that rounding moves them elsewhere, and
    a second solve is the same to the last bit."""
    torch = gpu
    m, nus, b = _ragged(torch, cells, S, 7 * S + sum(cells))
    A = assembly.Assembly(m)
    sv = survey.Survey(A, nus)
    res, its = {}, {}
    for v in (32, 35):
        sv.set_spmv_variant(v)
        _, st = sv.solve(b, torch.zeros_like(b), eps=1e-13, maxiter=5, verify=False)
        res[v] = np.array(st["residual_rel"])
        _, st = sv.solve(b, torch.zeros_like(b), eps=1e-6, maxiter=2000, verify=False)
        its[v] = np.array(st["iterations"])
    assert np.all(np.abs(res[35] - res[32]) <= 1e-7 * res[32] + 320 * 2.0 ** -46)
    runs = []
    for _ in range(2):
        x = torch.zeros_like(b)
        code, st = sv.solve(b, x, eps=1e-6, maxiter=2000, verify=False)
        assert code == 0 and np.all(np.abs(np.array(st["iterations"]) - its[32]) <= 3)
        runs.append((st["iterations"], st["residual_rel"], x))
    assert runs[0][:2] == runs[1][:2] and torch.equal(runs[0][2], runs[1][2])
    sv.close()
    A.close()


def test_one_kernel_iterations_from_two_threads(gpu):
    """Two surveys solved at the same time from two threads on their own
    streams: each launch of the one-kernel iteration needs the whole chip, and
    both end with what they give alone."""
    import threading
    torch = gpu
    probs = []
    for cells, S in (((24, 24, 25), 2), ((31, 27, 22), 1)):
        m, nus, b = _ragged(torch, cells, S, 5)
        A = assembly.Assembly(m)
        sv = survey.Survey(A, nus)
        sv.set_spmv_variant(35)
        x = torch.zeros_like(b)
        _, st = sv.solve(b, x, eps=1e-6, maxiter=2000, verify=False)
        probs.append((A, sv, b, x, st["iterations"]))
    ok = [0, 0]

    def work(i):
        A, sv, b, ref, its = probs[i]
        for _ in range(4):
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            code, st = sv.solve(b, x, eps=1e-6, maxiter=2000, verify=False)
            ok[i] += code == 0 and st["iterations"] == its and bool(torch.equal(x, ref))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert ok == [4, 4]
    for A, sv, *_ in probs:
        sv.close()
        A.close()


@pytest.mark.parametrize("unit,S,e", [(1e4, 2, 57), (1e4, 4, 57), (1e6, 2, 54), (1e6, 4, 54)])
@pytest.mark.parametrize("form", ["32", "34", "fused preconditioner"])
def test_block_sums_beyond_fp32_range(gpu, monkeypatch, form, unit, S, e):
    """The forms that add a block's threads in FP64 pass the sum on in FP32
    numbers: at these sizes (length unit, right-hand side 2^e) it is beyond
    2^128 while each thread's is not, and the solutions still scale exactly."""
    torch = gpu
    rng = np.random.default_rng(5)
    cells = (20, 19, 24)
    x, y = unit * _lines(rng, cells[0], -300.0), unit * _lines(rng, cells[1], -500.0)
    z = _lines(rng, cells[2], 0.0)
    z = unit * (z - z[cells[2] - 1])
    m = layered_model(x, y, z, [Layer(0.0, 0.01 / unit ** 2)],
                      cell_sigma=10.0 ** rng.uniform(-3, 0, int(np.prod(cells))) / unit ** 2)
    nus = list(10.0 ** rng.uniform(0, 2, S))
    b = torch.from_numpy(rng.standard_normal((S, 2 * m.nb))).cuda()
    monkeypatch.setenv("MTGPU_PREC_TILE", "1" if form == "fused preconditioner" else "0")
    A = assembly.Assembly(m)
    sv = survey.Survey(A, nus)
    sv.set_spmv_variant(34 if form == "34" else 32)
    assert sv.preconditioner()[0] == (form == "fused preconditioner")
    out = []
    for scale in (1.0, 2.0 ** e):
        u = torch.zeros_like(b)
        code, st = sv.solve(b * scale, u, eps=1e-4, maxiter=300, verify=False)
        assert code == 0 and st["fp64_iterations"] == [0] * S
        out.append((st["iterations"], u / scale))
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1])
    sv.close()
    A.close()
