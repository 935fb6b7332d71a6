"""The on-chip CG (patches of elements, one block each) at the edges of its
range: single elements, two elements around a periodic direction, element
counts that no cut divides, the largest patch of each kernel form and the
first size beyond it, every norm and null-space mode, and batches whose teams
need several launches.

Tolerances: iteration counts within 2 of the oracle's and solutions at rtol
1e-12 within 1e-8 of its magnitude, as for every CG solve of the suite; where
the oracle's matrix would be too large, against the fast-diagonalization
solution of the same system; batched against single solves 1e-10.
"""
import numpy as np
import pytest

from test_gpu_linsys import build

pytestmark = pytest.mark.gpu

P, CH, BOX = (True, True), (True, False), (False, False)
NONE, TB, ALL = (False,) * 4, (True, True, False, False), (True,) * 4

SMALL = [
    (1, 1, 12, (0.0, 0.0), (1.0, 2.0), BOX, ALL),
    (1, 1, 3, (0.0, 0.0), (1.0, 1.0), BOX, NONE),
    (2, 2, 2, (-1.0, 0.0), (1.0, 1.0), P, NONE),
    (2, 5, 9, (0.0, 0.0), (1.0, 1.0), CH, TB),
    (31, 1, 5, (0.0, 0.0), (7.0, 1.0), BOX, NONE),
    (13, 11, 8, (0.0, 0.0), (1.0, 1.0), CH, TB),
    (19, 17, 6, (0.0, -1.0), (2.0, 1.0), P, NONE),
    (7, 9, 11, (0.0, 0.0), (1.0, 1.0), BOX, ALL),
]


@pytest.mark.parametrize("case", range(len(SMALL)))
@pytest.mark.parametrize("norm", [0, 1, 2])
def test_matches_oracle(segpu, oracle, case, norm):
    om, m, fs, fr, ls, A, f2v, v2f, sol, rhs = build(segpu, oracle, SMALL[case], -3.0, -1.0, 1.0,
                                                     True, seed=case + 40)
    ref, st = oracle.helmholtz_solve(om, sol, rhs, -3.0, -1.0, 1.0, bcs=SMALL[case][6], quirk=True,
                                     rtol=1e-12, norm_type=norm)
    ls.set_opts(segpu.solver_opts(rtol=1e-12, norm_type=norm))
    out = ls.Solve("helm_")
    assert st["reason"] == out["reason"] == 2
    assert abs(out["its"] - st["its"]) <= 2, (out, st)
    got = fs.vals
    assert np.abs(got - ref).max() <= 1e-8 * np.abs(ref).max()
    assert np.array_equal(got[f2v < 0], sol[f2v < 0])


def smooth(S, ne, p, lam, method, rtol=1e-11):
    m = S.Mesh("m", list(ne), "legendre", p, [0, 0], [1, 1], [True, True])
    b = S.BCs(False, False, False, False, m)
    X = m.verts
    u, f = S.Field("u", m, 1, b), S.Field("f", m, 1, b)
    f.vals = np.cos(2 * np.pi * X[:, 0]) * np.sin(4 * np.pi * X[:, 1]) + 0.2
    ls = S.HelmholtzEqn(u, f, -lam, -1.0, 1.0, 0,
                        S.solver_opts(rtol=rtol, mode=S.MODE_EXACT, method=method))
    return m, u, f, ls


# 148 patches of at most 2048 nodes (all state in registers), of at most 4096,
# and beyond (the streaming kernel)
@pytest.mark.parametrize("ne,p", [((64, 64), 8), ((70, 72), 8), ((81, 80), 8), ((100, 104), 8),
                                  ((150, 3), 12), ((3, 260), 4)])
def test_large_matches_fast_diagonalization(segpu, ne, p):
    out = {}
    for method in (segpu.METHOD_CG, segpu.METHOD_FDM):
        m, u, f, ls = smooth(segpu, ne, p, 20.0, method)
        assert ls.Solve()["reason"] == 2
        out[method] = u.vals
    ref = out[segpu.METHOD_FDM]
    assert np.abs(out[segpu.METHOD_CG] - ref).max() <= 1e-8 * np.abs(ref).max()


def test_batch_over_several_launches(segpu):
    """Four large systems beside 60 small ones: more blocks than one launch
    holds, teams of one block and of many."""
    sizes = [(40, 44), (52, 30), (36, 36), (48, 41)] + [(2 + k % 7, 3 + k % 5) for k in range(60)]
    systems = [smooth(segpu, s, 8, 1.0 + k, segpu.METHOD_CG) for k, s in enumerate(sizes)]
    singles = []
    for m, u, f, ls in systems:
        st = ls.Solve()
        singles.append((u.vals, st))
        u.vals = 0.0
    stats = segpu.solve_batch([s[3] for s in systems])
    for (m, u, f, ls), (ref, rst), st in zip(systems, singles, stats):
        assert st["reason"] == rst["reason"] == 2
        assert abs(st["its"] - rst["its"]) <= 2
        assert np.abs(u.vals - ref).max() <= 1e-10 * np.abs(ref).max()


def test_iteration_limits_and_zero_rhs(segpu):
    m, u, f, ls = smooth(segpu, (9, 8), 6, 1.0, segpu.METHOD_CG)
    ls.set_opts(segpu.solver_opts(rtol=1e-12, mode=segpu.MODE_EXACT, max_it=5))
    st = ls.Solve()
    assert (st["reason"], st["its"]) == (-3, 5)
    ls.set_opts(segpu.solver_opts(rtol=1e-12, mode=segpu.MODE_EXACT, max_it=0))
    assert ls.Solve()["its"] == 0
    f.vals = 0.0
    ls.set_opts(segpu.solver_opts(rtol=1e-12, mode=segpu.MODE_EXACT))
    st = ls.Solve()
    assert st["its"] == 0 and st["reason"] in (2, 3)
    assert not np.any(u.vals)


@pytest.mark.parametrize("case", [3, 5])
@pytest.mark.parametrize("batched", [False, True])
def test_subnormal_inner_products(segpu, oracle, case, batched):
    """Data so small that the inner products are subnormal: the solve ends as
    the oracle's does (the product of successive p . A p underflows, reason
    -10 after one step) and leaves finite values, not those of an overflowed
    1 / beta. Single solves run as a cluster, batches through packets."""
    e = 1e-156
    om, m, fs, fr, ls, A, f2v, v2f, sol, rhs = build(segpu, oracle, SMALL[case], -3.0, -1.0, 1.0,
                                                     True, seed=case + 40)
    fs.vals, fr.vals = sol * e, rhs * e
    ls.Assemble()
    ref, st = oracle.helmholtz_solve(om, sol * e, rhs * e, -3.0, -1.0, 1.0, bcs=SMALL[case][6],
                                     quirk=True, rtol=1e-10, atol=0.0)
    ls.set_opts(segpu.solver_opts(rtol=1e-10, atol=0.0))
    out = segpu.solve_batch([ls])[0] if batched else ls.Solve("helm_")
    assert (out["reason"], out["its"]) == (st["reason"], st["its"]) == (-10, 1)
    assert np.isfinite(fs.vals).all() and np.isfinite(out["rnorm"])


# every form of the kernel: one cluster and a grid, each with all of a block's
# state in registers (at most 2048 nodes) and in shared memory (at most 4096)
FORMS = [
    ((9, 7), 6, P, NONE), ((14, 16), 5, CH, TB),                              # cluster, registers
    ((20, 20), 9, P, NONE), ((16, 16), 12, CH, TB), ((16, 29), 8, BOX, ALL),  # cluster, shared
    ((20, 31), 7, P, NONE), ((31, 15), 8, BOX, NONE),
    ((40, 36), 8, P, NONE), ((35, 44), 7, CH, TB), ((52, 29), 8, BOX, ALL),   # grid, registers
    ((70, 72), 8, P, NONE), ((66, 61), 9, CH, TB), ((90, 71), 7, BOX, ALL),   # grid, shared
]


def form_system(S, form, method, poisson=False, off=0.0, **kw):
    ne, p, per, walls = form
    m = S.Mesh("m", list(ne), "legendre", p, [0, 0], [1, 1], list(per))
    b = S.BCs(*walls, m)
    X = m.verts
    u, f = S.Field("u", m, 1, b), S.Field("f", m, 1, b)
    f.vals = (np.cos(2 * np.pi * X[:, 0]) * np.sin(4 * np.pi * X[:, 1])
              + np.cos(6 * np.pi * X[:, 1]) + off)
    o = S.solver_opts(rtol=1e-11, mode=S.MODE_EXACT, method=method, **kw)
    ls = S.PoissonEqn(u, f, 1.0, o) if poisson else S.HelmholtzEqn(u, f, -20.0, -1.0, 1.0, 0, o)
    return m, u, f, ls


@pytest.mark.parametrize("form", range(len(FORMS)))
@pytest.mark.parametrize("norm", [0, 1, 2])
def test_every_form_and_norm(segpu, form, norm):
    _, u, _, ls = form_system(segpu, FORMS[form], segpu.METHOD_CG, norm_type=norm)
    assert ls.Solve()["reason"] == 2
    _, r, _, lr = form_system(segpu, FORMS[form], segpu.METHOD_FDM)
    assert lr.Solve()["reason"] == 2
    assert np.abs(u.vals - r.vals).max() <= 1e-8 * np.abs(r.vals).max()


PERIODIC = [0, 2, 5, 7, 10]


@pytest.mark.parametrize("form", PERIODIC)
@pytest.mark.parametrize("project", [False, True])
def test_null_space_in_every_form(segpu, form, project):
    """Periodic Poisson: the mean of z as a third reduction, and a right-hand
    side off the operator's range projected onto it first."""
    off = 0.3 if project else 0.0
    out = []
    for method in (segpu.METHOD_CG, segpu.METHOD_FDM):
        _, u, _, ls = form_system(segpu, FORMS[form], method, poisson=True, off=off)
        st = ls.Solve(removeNullSpace=True, projectRHS=project)
        assert st["reason"] == 2, st
        out.append(u.vals - u.vals.mean())
    assert np.abs(out[0] - out[1]).max() <= 1e-8 * np.abs(out[1]).max()


def test_batch_with_null_space(segpu):
    """Teams of one block to many, the constant removed in each."""
    sizes = [(40, 36), (9, 8), (2, 2), (25, 14), (5, 6), (50, 41)]
    systems = [form_system(segpu, (s, 8, P, NONE), segpu.METHOD_CG, poisson=True) for s in sizes]
    stats = segpu.solve_batch([s[3] for s in systems], removeNullSpace=True)
    for (m, u, f, ls), s, st in zip(systems, sizes, stats):
        assert st["reason"] == 2
        _, r, _, lr = form_system(segpu, (s, 8, P, NONE), segpu.METHOD_FDM, poisson=True)
        assert lr.Solve(removeNullSpace=True)["reason"] == 2
        got, ref = u.vals - u.vals.mean(), r.vals - r.vals.mean()
        assert np.abs(got - ref).max() <= 1e-8 * np.abs(ref).max()


def test_solves_with_no_memory_left(segpu):
    """A system created before the rest of the program took all device memory
    still solves, alone and in a batch: without room for its packets the
    streaming kernel runs on the vectors the system has."""
    import ctypes
    import torch

    def make(ne, svv=0):
        m, u, f, ls = smooth(segpu, ne, 5, 7.0, segpu.METHOD_CG)
        if svv:
            ls = segpu.HelmholtzEqn(u, f, -7.0, -1.0, 1.0, svv,
                                    segpu.solver_opts(rtol=1e-11, mode=segpu.MODE_EXACT))
        return m, u, f, ls

    # both streaming kernels' code on the device, and the answers
    warm = [make((9, 8), 2), make((8, 8), 2)]
    for w in warm:
        assert w[3].Solve()["reason"] == 2
    segpu.solve_batch([w[3] for w in warm])
    ref = [make((9, 8)), make((6, 7))]
    for r in ref:
        assert r[3].Solve()["reason"] == 2
    ref = [r[1].vals for r in ref]
    systems = [make((9, 8)), make((6, 7))]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    rt.cudaFree.argtypes = [ctypes.c_void_p]
    held = []
    size = torch.cuda.mem_get_info()[0]
    while size >= 256:
        p = ctypes.c_void_p()
        if rt.cudaMalloc(ctypes.byref(p), size) == 0:
            held.append(p)
        else:
            rt.cudaGetLastError()
            size //= 2
    try:
        got = []
        for s in systems:
            assert s[3].Solve()["reason"] == 2
            got.append(s[1].vals)
            s[1].vals = 0.0
        assert all(st["reason"] == 2 for st in segpu.solve_batch([s[3] for s in systems]))
        got += [s[1].vals for s in systems]
    finally:
        for p in held:
            rt.cudaFree(p)
    for a, b in zip(got, ref + ref):
        assert np.abs(a - b).max() <= 1e-8 * np.abs(b).max()
