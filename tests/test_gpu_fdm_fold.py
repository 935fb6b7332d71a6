"""The FP64 dense inverse on folded directions: every combination of ends that
folds or does not, even and odd unknown counts, a single unknown, parts that
end on, before and after a tile edge, against the tensor-product operator
assembled from the mesh's GLL tables.

Tolerance: A x - r within 1e-11 of (|A| |x| + |r|) row by row, the bound the
suite holds the dense inverse to (about 20 times the rounding of four products
of a few hundred terms each with eigenvectors accurate to the last bits).
"""
import numpy as np
import pytest

from test_gpu_apply_tiles import system

pytestmark = pytest.mark.gpu

P, CH, BOX = (True, True), (True, False), (False, False)
N4, TB, ALL = (False,) * 4, (True, True, False, False), (True,) * 4

CASES = [
    (1, 1, 2, BOX, ALL),                            # one unknown
    (1, 3, 3, BOX, (True, False, True, False)),     # neither direction folds
    (3, 5, 2, P, N4), (5, 3, 3, P, N4),             # odd periodic counts
    (3, 4, 8, CH, TB), (9, 7, 5, CH, N4),
    (11, 6, 6, BOX, ALL), (7, 8, 4, BOX, N4),
    (6, 7, 7, BOX, (True, True, False, True)),      # x ends differ, y folds
    (13, 9, 5, BOX, (False, True, True, True)),     # y ends differ, x folds
    (17, 12, 6, P, N4), (43, 29, 3, BOX, ALL),      # several tiles
    (33, 50, 8, CH, TB), (150, 101, 6, BOX, ALL),   # 64 x 64 tiles
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_inverse(segpu, case):
    import torch
    nx, ny, N, per, walls = CASES[case]
    keep, ls, apply, n = system(segpu, nx, ny, N, per, walls)
    r = np.random.default_rng(case).standard_normal(n)
    rd = torch.tensor(r, device="cuda")
    x = torch.full((n + 2,), 7.0, device="cuda", dtype=torch.float64)
    x[1:-1] = float("nan")  # every entry is written
    ls.fdm_apply(rd.data_ptr(), x.data_ptr() + 8)
    torch.cuda.synchronize()
    got = x.cpu().numpy()
    assert got[0] == 7.0 and got[-1] == 7.0
    got = got[1:-1]
    assert (np.abs(apply(got) - r) <= 1e-11 * (apply(got, True) + np.abs(r))).all()
    # the same bits again
    y = torch.zeros(n, device="cuda", dtype=torch.float64)
    ls.fdm_apply(rd.data_ptr(), y.data_ptr())
    assert np.array_equal(y.cpu().numpy(), got)


@pytest.mark.parametrize("nx,ny,N,per,walls", [(12, 9, 6, CH, TB), (7, 9, 5, P, N4),
                                               (20, 11, 7, BOX, ALL)])
def test_smooth_solve_takes_one_step(segpu, nx, ny, N, per, walls):
    """The low modes carried apart: a smooth right-hand side meets rtol 1e-10
    in one refinement step."""
    m = segpu.Mesh("m", [nx, ny], "legendre", N, [0.0, 0.0], [1.0, 1.0], list(per))
    b = segpu.BCs(*walls, m)
    u, f = segpu.Field("u", m, 1, b), segpu.Field("f", m, 1, b)
    X = m.verts
    f.vals = np.cos(2 * np.pi * X[:, 0]) * np.sin(2 * np.pi * X[:, 1]) + 0.5
    ls = segpu.HelmholtzEqn(u, f, -1.0, -1.0, 1.0, 0,
                            segpu.solver_opts(rtol=1e-10, mode=segpu.MODE_EXACT,
                                              method=segpu.METHOD_FDM))
    st = ls.Solve()
    assert st["reason"] == 2 and st["its"] == 1, st
