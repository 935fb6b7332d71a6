"""The operator apply at the edges of its tiles, every order, against the
tensor-product operator assembled from the mesh's own GLL tables in FP64.

Meshes of one tile, one element more or less than whole tiles, several tiles
with interior ones, and sizes on both sides of every staging rule: rows of an
odd, even and multiple-of-four number of unknowns, first columns at every
offset from an 8-byte boundary, tiles that end the array, x off alignment.

Tolerances: the sums run over at most 4N + 8 products, so FP64 results are
within 64 rounding errors (64 * 2^-53, about 7e-15) of the row's sum of
magnitudes, FP32 arithmetic within 64 * 2^-24 (about 4e-6).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P, CH, BOX = (True, True), (True, False), (False, False)
WALLS = {P: (False,) * 4, CH: (True, True, False, False), BOX: (True,) * 4, "nat": (False,) * 4}


def dense_1d(ne, N, w, Kh, periodic, lo, hi):
    nv = ne * N + 1
    K, W = np.zeros((nv, nv)), np.zeros(nv)
    for e in range(ne):
        s = slice(e * N, e * N + N + 1)
        K[s, s] += Kh
        W[s] += w
    if periodic:
        K[0] += K[-1]
        K[:, 0] += K[:, -1]
        W[0] += W[-1]
    return K[lo:hi, lo:hi], W[lo:hi]


def system(S, nx, ny, N, per, walls):
    m = S.Mesh("m", [nx, ny], "legendre", N, [0.0, 0.0], [1.0, 0.7], list(per))
    b = S.BCs(*walls, m)
    u = S.Field("u", m, 1, b)
    ls = S.HelmholtzEqn(u, None, -3.0, -1.0, 0.5, 0, S.solver_opts(mode=S.MODE_EXACT))
    x, w, D = m.gll()
    Kh = D.T @ np.diag(w) @ D
    bot, top, left, right = walls
    X = (int(left), nx * N + (0 if per[0] or right else 1))
    Y = (int(bot), ny * N + (0 if per[1] or top else 1))
    Kx, Wx = dense_1d(nx, N, w, Kh, per[0], *X)
    Ky, Wy = dense_1d(ny, N, w, Kh, per[1], *Y)
    hx, hy = 1.0 / nx, 0.7 / ny
    al, bx, by = -3.0 * hx * hy / 4, -0.5 * hy / hx, -0.5 * hx / hy

    def apply(v, mag=False):
        f = np.abs if mag else (lambda z: z)
        v = f(v.reshape(len(Wy), len(Wx)))
        return (f(al) * Wy[:, None] * Wx * v + f(bx) * Wy[:, None] * (v @ f(Kx).T)
                + f(by) * Wx * (f(Ky) @ v)).ravel()

    return (m, b, u), ls, apply, len(Wx) * len(Wy)


def sizes(N):
    ex = 64 // N  # elements of a tile row; a tile has four element rows
    return [(2, 2), (ex, 4), (ex + 1, 5), (max(2, ex - 1), 3), (3 * ex, 12), (3 * ex + 2, 13)]


KINDS = [(P, WALLS[P]), (CH, WALLS[CH]), (BOX, WALLS[BOX]), (BOX, WALLS["nat"]),
         (BOX, (False, True, True, False))]


@pytest.mark.parametrize("N", range(2, 13))
@pytest.mark.parametrize("kind", range(len(KINDS)))
def test_fp64(segpu, N, kind):
    import torch
    for nx, ny in sizes(N):
        keep, ls, apply, n = system(segpu, nx, ny, N, *KINDS[kind])
        assert ls.vecSize == n
        x = np.random.default_rng(nx * 100 + ny).standard_normal(n)
        xd = torch.tensor(np.concatenate([[0.0], x]), device="cuda")
        y = torch.full((n + 2,), 7.0, device="cuda", dtype=torch.float64)
        ls.apply(xd.data_ptr() + 8, y.data_ptr() + 8)
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        assert got[0] == 7.0 and got[-1] == 7.0
        assert (np.abs(got[1:-1] - apply(x)) <= 64 * 2.0 ** -53 * apply(x, True)).all(), (nx, ny)


@pytest.mark.parametrize("N", range(2, 13))
@pytest.mark.parametrize("kind", range(len(KINDS)))
@pytest.mark.parametrize("half", [False, True])
def test_reduced_precision(segpu, N, kind, half):
    import torch
    dt = torch.float16 if half else torch.bfloat16
    for k, (nx, ny) in enumerate(sizes(N) + [(3 * (64 // N) + 1, 12), (3 * (64 // N) + 3, 12)]):
        keep, ls, apply, n = system(segpu, nx, ny, N, *KINDS[kind])
        x = torch.tensor(np.random.default_rng(nx * 100 + ny).standard_normal(n)).to(dt)
        off = k % 5  # 2-byte steps off alignment
        xd = torch.zeros(n + 8, device="cuda", dtype=dt)
        xd[off:off + n] = x.cuda()
        y = torch.full((n + 2,), 7.0, device="cuda", dtype=torch.float32)
        ls.apply_low(xd.data_ptr() + 2 * off, y.data_ptr() + 4,
                     segpu.PREC_FP16 if half else segpu.PREC_BF16)
        torch.cuda.synchronize()
        got = y.cpu().numpy().astype(np.float64)
        assert got[0] == 7.0 and got[-1] == 7.0
        xr = x.double().numpy()
        assert (np.abs(got[1:-1] - apply(xr)) <= 64 * 2.0 ** -24 * apply(xr, True)).all(), (nx, ny)


@pytest.mark.parametrize("N,ny", [(2, 262142), (3, 262145)])
def test_tallest_meshes(segpu, N, ny):
    """More rows of unknowns than a grid's y dimension of tiles covers (65535
    tiles of 4 N), FP64 and BF16, against the residual's kernel (r = 0 - A x,
    which steps over its tiles) at the tolerances above, row sums of
    magnitudes bounded by 4 times the largest element entries."""
    import torch
    m = segpu.Mesh("m", [1, ny], "legendre", N, [0.0, 0.0], [1.0, float(ny)], [False, False])
    u = segpu.Field("u", m, 1, segpu.BCs(False, False, False, False, m))
    ls = segpu.HelmholtzEqn(u, None, -3.0, -1.0, 0.5, 0, segpu.solver_opts(mode=segpu.MODE_EXACT))
    n = ls.vecSize
    xb = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(N)).bfloat16()
    x = xb.double()
    y, r, zero = (torch.zeros(n, device="cuda", dtype=torch.float64) for _ in range(3))
    yf = torch.full((n,), float("nan"), device="cuda")
    ls.residual(x.data_ptr(), zero.data_ptr(), r.data_ptr())
    y.fill_(float("nan"))
    torch.cuda.synchronize()
    ls.apply(x.data_ptr(), y.data_ptr())
    ls.apply_low(xb.data_ptr(), yf.data_ptr(), segpu.PREC_BF16)
    segpu.synchronize()
    gx, gw, D = m.gll()
    Kh = np.abs(D.T @ np.diag(gw) @ D)
    scale = float(x.abs().max()) * 4.0 * (3.0 * gw.max() ** 2 / 4 + Kh.sum(1).max() * gw.max())
    assert float((y + r).abs().max()) <= 64 * 2.0 ** -53 * scale
    assert float((yf.double() + r).abs().max()) <= 64 * 2.0 ** -24 * scale


# 16-bit tiles of orders 2 to 4 four times as high (from 1184 tiles on; wide
# meshes of order 2, others one tile wide), the last tile cut short, rows of a
# multiple of four unknowns and not; order 5 just as narrow on the plain tile
TALL = [(2, 33, 2370, P), (2, 100, 1187, P), (2, 101, 1186, "nat"), (2, 9, 4799, BOX),
        (3, 20, 4741, CH), (3, 1, 4745, BOX), (4, 15, 4747, BOX), (4, 16, 4739, P), (5, 7, 4741, CH)]


@pytest.mark.parametrize("case", range(len(TALL)))
def test_tall_tiles(segpu, case):
    """FP64 and 16-bit applies against the residual's kernel, as above."""
    import torch
    N, nx, ny, per = TALL[case]
    walls = WALLS[per]
    m = segpu.Mesh("m", [nx, ny], "legendre", N, [0.0, 0.0], [1.0, ny / nx],
                   list(BOX if per == "nat" else per))
    u = segpu.Field("u", m, 1, segpu.BCs(*walls, m))
    ls = segpu.HelmholtzEqn(u, None, -3.0, -1.0, 0.5, 0, segpu.solver_opts(mode=segpu.MODE_EXACT))
    n = ls.vecSize
    gx, gw, D = m.gll()
    Kh = np.abs(D.T @ np.diag(gw) @ D)
    hx = 1.0 / nx
    for dt, prec in ((torch.bfloat16, segpu.PREC_BF16), (torch.float16, segpu.PREC_FP16)):
        xl = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(case)).to(dt)
        x = xl.double()
        y, r, zero = (torch.zeros(n, device="cuda", dtype=torch.float64) for _ in range(3))
        y.fill_(float("nan"))
        yf = torch.full((n + 2,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        ls.residual(x.data_ptr(), zero.data_ptr(), r.data_ptr())
        ls.apply(x.data_ptr(), y.data_ptr())
        ls.apply_low(xl.data_ptr(), yf.data_ptr() + 4, prec)
        segpu.synchronize()
        scale = float(x.abs().max()) * 4.0 * (3.0 * (gw.max() * hx) ** 2 / 4 + Kh.sum(1).max() * gw.max())
        assert float((y + r).abs().max()) <= 64 * 2.0 ** -53 * scale
        assert bool(yf[0].isnan()) and bool(yf[-1].isnan())
        assert float((yf[1:-1].double() + r).abs().max()) <= 64 * 2.0 ** -24 * scale
