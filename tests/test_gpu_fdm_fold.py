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


# where the inverse folds (from 4,096 unknowns where both directions do, from
# 32,768 where one does, and with any direction of more than 256), the sizes
# on either side, and where it does not: odd and even rows
ROUTES = [
    (17, 15, 4, P, N4), (17, 16, 4, P, N4),               # 4,080 and 4,352 unknowns
    (13, 23, 5, P, N4), (11, 13, 6, BOX, ALL), (16, 11, 6, BOX, N4), (13, 10, 7, CH, TB),
    (51, 1, 5, BOX, ALL), (1, 52, 5, BOX, ALL), (2, 52, 5, CH, N4),  # 254 and 259 long
    (30, 29, 6, BOX, (True, True, False, True)), (30, 37, 6, BOX, (True, True, False, True)),
    (31, 36, 6, BOX, (False, True, True, True)), (37, 37, 5, BOX, (False, True, True, True)),
    (9, 11, 5, BOX, (True, False, True, False)), (10, 11, 4, BOX, (True, False, False, True)),
    (52, 3, 5, BOX, (False, True, True, False)), (101, 99, 7, BOX, (True, False, True, False)),
]


@pytest.mark.parametrize("case", range(len(ROUTES)))
@pytest.mark.parametrize("offset", [0, 1])
def test_routes(segpu, case, offset):
    """Input on and off a 16-byte boundary, output beside guards."""
    import torch
    nx, ny, N, per, walls = ROUTES[case]
    keep, ls, apply, n = system(segpu, nx, ny, N, per, walls)
    r = np.random.default_rng(case + 50).standard_normal(n)
    rd = torch.zeros(n + 1, device="cuda", dtype=torch.float64)
    rd[offset:n + offset] = torch.tensor(r)
    x = torch.full((n + 2,), float("nan"), device="cuda", dtype=torch.float64)
    x[0] = x[-1] = 7.0
    torch.cuda.synchronize()
    ls.fdm_apply(rd.data_ptr() + 8 * offset, x.data_ptr() + 8)
    segpu.synchronize()
    got = x.cpu().numpy()
    assert got[0] == 7.0 and got[-1] == 7.0
    got = got[1:-1]
    assert (np.abs(apply(got) - r) <= 1e-11 * (apply(got, True) + np.abs(r))).all()


@pytest.mark.parametrize("nx,ny,N,per,walls", [(9, 11, 5, BOX, (True, False, True, False)),
                                               (7, 6, 4, BOX, ALL), (20, 17, 5, BOX, ALL)])
def test_zero_right_hand_side(segpu, nx, ny, N, per, walls):
    """A solve that is decided before its first step adds nothing, on either
    route, also after a solve that left other values in the work arrays."""
    m = segpu.Mesh("m", [nx, ny], "legendre", N, [0.0, 0.0], [1.0, 1.0], list(per))
    u, f = segpu.Field("u", m, 1, segpu.BCs(*walls, m)), segpu.Field("f", m, 1, None)
    ls = segpu.HelmholtzEqn(u, f, -1.0, -1.0, 1.0, 0,
                            segpu.solver_opts(rtol=1e-10, mode=segpu.MODE_EXACT,
                                              method=segpu.METHOD_FDM))
    f.vals = 1.0 + m.verts[:, 0]
    assert ls.Solve()["reason"] == 2 and np.abs(u.vals).max() > 0
    f.vals = 0.0
    st = ls.Solve()
    assert st["its"] == 0 and st["reason"] in (2, 3)
    bot, top, left, right = walls
    g = u.vals.reshape(ny * N + 1, nx * N + 1)
    assert not g[int(bot):ny * N + 1 - int(top), int(left):nx * N + 1 - int(right)].any()


def test_setup_memory(segpu):
    """A direction of n unknowns keeps its folded factors, about n^2 doubles,
    and no full matrix beside them."""
    import torch

    def solve(nx):
        m = segpu.Mesh("m", [nx, 2], "legendre", 6, [0.0, 0.0], [1.0, 1.0], [True, False])
        u, f = segpu.Field("u", m, 1, segpu.BCs(*TB, m)), segpu.Field("f", m, 1, None)
        f.vals = np.cos(2 * np.pi * m.verts[:, 0])
        ls = segpu.HelmholtzEqn(u, f, -1.0, -1.0, 1.0, 0,
                                segpu.solver_opts(rtol=1e-10, mode=segpu.MODE_EXACT,
                                                  method=segpu.METHOD_FDM))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        assert ls.Solve()["reason"] == 2
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0]

    solve(37)  # cuSOLVER's and the kernels' own memory
    n = 401 * 6
    assert solve(401) <= 8 * 1.5 * n * n + (8 << 20)


@pytest.mark.parametrize("nx,ny,N,per,walls", [(37, 20, 6, CH, TB), (9, 8, 5, BOX, ALL), (7, 9, 5, P, N4),
                                               (16, 8, 6, P, N4), (9, 11, 5, BOX, (True, False, True, False))])
@pytest.mark.parametrize("first", ["fp64", "mixed", "bf16"])
def test_precisions_in_any_order(segpu, nx, ny, N, per, walls, first):
    """The low precisions take the eigenvectors from the FP64 factors, whichever
    precision set a direction up (other element counts per `first`: fresh
    directions): solutions agree at rtol 1e-11 to 1e-9. (Square elements: BF16
    refinement does not contract at aspect ratio 4.)"""
    precs = {"fp64": segpu.PREC_FP64, "mixed": segpu.PREC_MIXED, "bf16": segpu.PREC_BF16}
    nx += {"fp64": 0, "mixed": 16, "bf16": 32}[first] * (1 if nx != 16 else 0)
    m = segpu.Mesh("m", [nx, ny], "legendre", N, [0.0, 0.0], [nx / ny, 1.0], list(per))
    u, f = segpu.Field("u", m, 1, segpu.BCs(*walls, m)), segpu.Field("f", m, 1, None)
    X = m.verts
    f.vals = np.cos(2 * np.pi * X[:, 0] * ny / nx) * np.sin(2 * np.pi * X[:, 1]) + 0.5
    ls = segpu.HelmholtzEqn(u, f, -1.0, -1.0, 1.0, 0)
    out = []
    for name in [first] + [k for k in precs if k != first] + ["fp64"]:
        u.vals = 0.0
        ls.set_opts(segpu.solver_opts(rtol=1e-11, mode=segpu.MODE_EXACT, method=segpu.METHOD_FDM,
                                      precision=precs[name], max_it=100))
        assert ls.Solve()["reason"] == 2, name
        out.append(u.vals)
    for v in out[:-1]:
        assert np.abs(v - out[-1]).max() <= 1e-9 * np.abs(out[-1]).max()
