"""The smoothing projection's two column groupings: few systems are solved two
columns a block, many four a block with a partial last group."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from mtcalc_with_dfp_cocr_gb300 import assembly, normal1d, receivers, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [71, 128])
def test_many_systems_equal_each_alone(gpu, S):
    """Both solve to a residual of 1e-14 with a condition number below 30; E
    and H are held to the bounds that the comparisons with the oracle use."""
    torch = gpu
    m = workloads.make("c1").mesh
    rec = np.load(os.path.join(GOLDEN, "smoothing.npz"))["rec_c1"]
    A = assembly.Assembly(m)
    R = receivers.Receivers(A, rec, output="smooth")
    rng = np.random.default_rng(S)
    z, us, uc = normal1d.solve_1d(1.0, [l.top for l in m.layers], [l.sigma for l in m.layers])
    x = torch.from_numpy(rng.standard_normal((S, 2 * m.nb))).cuda()
    alfas = [k % 2 for k in range(S)]
    E, H, _ = R.fields(x, [1.0] * S, alfas, z, np.stack([us] * S), np.stack([uc] * S))
    for k in (0, 3, S // 2, S - 1):
        e, h, _ = R.fields(x[k:k + 1].contiguous(), [1.0], alfas[k:k + 1], z, us[None], uc[None])
        assert float((E[k] - e[0]).abs().max() / e.abs().max()) < 1e-11
        assert float((H[k] - h[0]).abs().max() / h.abs().max()) < 1e-10
    A.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e200])
def test_values_without_a_projection(gpu, value):
    """An edge value that is not finite, or whose squares are not, leaves its
    system's fields without a value instead of the background's, and the
    other systems' as they are, within the bounds above (the columns of a block
    end their inner iterations together)."""
    torch = gpu
    m = workloads.make("c1").mesh
    rec = np.load(os.path.join(GOLDEN, "smoothing.npz"))["rec_c1"]
    A = assembly.Assembly(m)
    R = receivers.Receivers(A, rec, output="smooth")
    z, us, uc = normal1d.solve_1d(1.0, [l.top for l in m.layers], [l.sigma for l in m.layers])
    x = torch.from_numpy(np.random.default_rng(1).standard_normal((3, 2 * m.nb))).cuda()
    ref = R.fields(x, [1.0] * 3, [1, 0, 1], z, np.stack([us] * 3), np.stack([uc] * 3))
    x[1, ::2] = value          # the real parts
    got = R.fields(x, [1.0] * 3, [1, 0, 1], z, np.stack([us] * 3), np.stack([uc] * 3))
    for g, r, tol in zip(got[:2], ref[:2], (1e-11, 1e-10)):
        for k in (0, 2):
            assert float((g[k] - r[k]).abs().max() / r[k].abs().max()) < tol
        if tol == 1e-11 or not np.isfinite(value):       # (the curl of equal values is 0)
            assert bool(torch.isnan(g[1].real).all() | torch.isnan(g[1].imag).all())
    A.close()
