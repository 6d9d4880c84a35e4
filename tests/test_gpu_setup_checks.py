"""What the set-up's comparisons of two forms of an operator let through."""
import numpy as np
import pytest

from mtcalc_with_dfp_cocr_gb300 import assembly, normal1d, solver, workloads
from mtcalc_with_dfp_cocr_gb300.slae_io import mesh_to_solve_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["diagonal", "off-diagonal"])
def test_a_nan_in_the_matrix_is_not_overlooked(gpu, entry):
    """The matrix-free operator is made from the mesh: it may stand for a
    SLAE only where the two products agree, and a NaN agrees with nothing."""
    w = workloads.make("small")
    m = w.mesh
    z, us, uc = normal1d.solve_1d(1.0, [l.top for l in m.layers], [l.sigma for l in m.layers])
    A = assembly.Assembly(m)
    s = A.block2x2(1.0, 1, z, us, uc, eps=1e-8)
    mesh = mesh_to_solve_mesh(m)
    code, x, st = solver.pcocr_2x2_folded(s, mesh, double_float=True)
    assert code == 0 and st.spmv_variant >= 32 and 0.0 <= st.matfree_check < 1e-9
    (s.di if entry == "diagonal" else s.gg)[-1 if entry == "diagonal" else len(s.gg) // 2] = np.nan
    code, x, st = solver.pcocr_2x2_folded(s, mesh, maxiter=4, double_float=True)
    assert st.spmv_variant < 32 and not st.matfree_check < 1e-9
    assert code != 0
    A.close()
