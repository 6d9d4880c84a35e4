"""The smoothing projection on a large station layout: subdomains of 43,200
and 21,600 nodes, more than a block's shared memory holds of a direction, by
clusters of 8, 4 and 2 blocks and by single ones.  Those subdomains are boxes
of a tensor mesh, where the mass matrix is a product of three tridiagonal
ones: the oracle's projection is then three small solves instead of a sparse
factorisation."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import assembly, normal1d, receivers, workloads
from oracle import pyoracle as O
from oracle import smoothing

TWO_PI = 2.0 * 3.1415926535897932384626433832795


def _mass1d(x):
    h = np.diff(x)
    m = np.zeros((len(x), len(x)))
    for i, v in enumerate(h):
        m[i:i + 2, i:i + 2] += v * np.array([[2.0, 1.0], [1.0, 2.0]]) / 6.0
    return m


def box_project(m, cells, nodes, values):
    """smoothing.project where the subdomain is a box."""
    xyz = m.xyz()[nodes]
    X, Y, Z = (np.unique(xyz[:, d]) for d in range(3))
    n = (len(Z), len(Y), len(X))
    assert len(nodes) == np.prod(n) and len(cells) == np.prod(np.array(n) - 1)
    assert np.array_equal(xyz[:, 0].reshape(n), np.broadcast_to(X, n))
    h = [np.diff(v) for v in (Z, Y, X)]
    vol = h[0][:, None, None] * h[1][None, :, None] * h[2][None, None, :]
    f = (vol[..., None] / 8.0) * values.reshape(tuple(np.array(n) - 1) + (-1,))
    rhs = np.zeros(n + (values.shape[1],), values.dtype)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                rhs[dz:n[0] - 1 + dz, dy:n[1] - 1 + dy, dx:n[2] - 1 + dx] += f
    for axis, v in enumerate((Z, Y, X)):
        t = np.moveaxis(rhs, axis, 0)
        t = np.linalg.solve(_mass1d(v), t.reshape(len(v), -1)).reshape(t.shape)
        rhs = np.moveaxis(t, 0, axis)
    return rhs.reshape(len(nodes), -1)


def test_box_projection_is_the_oracles():
    m = workloads.make("c1").mesh
    rec = workloads.make("c1").receivers
    cells, nodes = smoothing.subdomain(m, smoothing.locate(m, rec, False), -1)
    v = np.random.default_rng(0).standard_normal((len(cells), 2)) + 1j
    a, b = box_project(m, cells, nodes, v), smoothing.project(m, cells, nodes, v)
    assert np.abs(a - b).max() / np.abs(b).max() < 1e-12


@pytest.fixture(scope="module")
def case():
    """The survey configuration's layout, one random solution and its smoothed A, curl A."""
    w = workloads.make("c3")
    v = np.random.default_rng(3).standard_normal(2 * w.mesh.nb)
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(smoothing, "project", box_project)
        return w, v, smoothing.smoothed_fields(w.mesh, w.receivers, v)


@pytest.mark.gpu
@pytest.mark.parametrize("S", [1, 3, 7, 16])
def test_large_layout(gpu, case, S):
    """The solution as the first and the last of S systems, other ones between."""
    torch = gpu
    w, v, (a, c) = case
    m, rec = w.mesh, w.receivers
    A = assembly.Assembly(m)
    R = receivers.Receivers(A, rec, output="smooth")
    assert R.smoothing_info()["nodes"] == [43200, 21600]
    x = np.random.default_rng(S).standard_normal((S, 2 * m.nb))
    x[0] = x[S - 1] = v
    z, us, uc = normal1d.solve_1d(1.0, [l.top for l in m.layers], [l.sigma for l in m.layers])
    alfas = [k % 2 for k in range(S)]
    E, H, _ = R.fields(torch.from_numpy(x).cuda(), [1.0] * S, alfas, z, np.stack([us] * S), np.stack([uc] * S))
    for k in {0, S - 1}:
        e, h, _ = O.receiver_fields(a, c, TWO_PI, *O.normal_field(rec, z, us, uc, alfas[k], TWO_PI))
        # the bounds of the comparisons on smaller subdomains
        assert np.abs(E[k].cpu().numpy() - e).max() / np.abs(e).max() < 1e-11
        assert np.abs(H[k].cpu().numpy() - h).max() / np.abs(h).max() < 1e-10
    R.close()
    A.close()
