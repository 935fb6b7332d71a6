"""SL advection where the element search and the kernel forms change over:
points on and beside element boundaries, domains far from the origin, tiny and
huge ones, and the second-order advection on both sides of the size from which
its half-level velocities are formed once per vertex.

The element search is compared bit for bit with the oracle's on the GPU's own
departure points, values with the accurate oracle at the suite's tolerance
(1e-12 of the field's magnitude), widened where the domain's offset itself
rounds coordinates: a coordinate c is known to |c| 2^-53, which moves a value
by that times the field's gradient.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACC_TOL = 1e-12


def make(S, nx, ny, N, lo, hi, per):
    return S.Mesh("m", [nx, ny], "legendre", N, list(lo), list(hi), list(per))


DOMAINS = [((0.0, 0.0), (1.0, 1.0)), ((1000.0, -500.0), (1001.0, -499.0)), ((-1e-7, 0.0), (1e-7, 3e-7)),
           ((-4e5, 1e6), (6e5, 3e6)), ((1e9, 0.0), (1e9 + 4.0, 1.0))]


@pytest.mark.parametrize("domain", range(len(DOMAINS)))
@pytest.mark.parametrize("N", [4, 7])
@pytest.mark.parametrize("per", [(True, True), (False, False)])
def test_points_on_element_boundaries(segpu, oracle, domain, N, per):
    """A uniform velocity whose displacement is a whole, half or hair's breadth
    over a whole number of elements puts departure points on boundaries."""
    lo, hi = DOMAINS[domain]
    nx, ny = 6, 5
    L = np.array(hi) - np.array(lo)
    om = oracle.Mesh(nx, ny, N, lo, hi, per)
    oa = oracle.Mesh(nx, ny, N, lo, hi, per, accurate=True)
    X = (om.verts() - np.array(lo)) / L
    phi = om.periodic_update(np.sin(2 * np.pi * X[:, 0]) * np.cos(2 * np.pi * X[:, 1]))
    m = make(segpu, nx, ny, N, lo, hi, per)
    f, v = segpu.Field("phi", m, 1, None), segpu.Field("vel", m, 2, None)
    f.vals = phi
    adv = segpu.Advector(f, v)
    adv.record_departures()
    slack = np.abs([*lo, *hi]).max() / L.min() * 2.0 ** -53 * 4 * np.pi * 4
    for cx, cy in ((1.0, 1.0), (2.0, 0.5), (0.5, 0.0), (1.0 + 1e-11, 1.0 - 1e-11), (1e-10, 3.0)):
        vel = np.tile([cx * L[0] / nx, cy * L[1] / ny], (om.nv, 1))
        v.vals = vel
        adv.Advect(1.0)
        out = adv.fieldSL.vals
        el, xy = adv.departures()
        oel, _ = om.global_to_local(xy)
        assert np.array_equal(oel, el)
        acc = oa.advect(phi, vel, 1.0)
        assert np.abs(out - acc).max() <= ACC_TOL + slack


@pytest.mark.parametrize("nx,ny,N,per", [(5, 4, 6, (True, False)), (28, 19, 9, (True, False)),
                                         (24, 30, 10, (False, False)), (41, 37, 7, (True, True))])
def test_second_order_both_forms(segpu, oracle, nx, ny, N, per):
    rng = np.random.default_rng(nx)
    om = oracle.Mesh(nx, ny, N, (0.0, 0.0), (1.0, 1.0), per, accurate=True)
    X = om.verts()
    x, y = X[:, 0], X[:, 1]
    u = np.stack([-np.sin(np.pi * x) ** 2 * np.sin(2 * np.pi * y),
                  np.sin(np.pi * y) ** 2 * np.sin(2 * np.pi * x)], 1)
    up = om.periodic_update(u * (1 + 0.02 * rng.standard_normal((om.nv, 1))), 2)
    u = om.periodic_update(u, 2)
    psi = om.periodic_update(np.cos(2 * np.pi * x) * np.sin(2 * np.pi * y))
    psip = om.periodic_update(psi + 0.01 * rng.standard_normal(om.nv))
    dt = 1.5 / max(nx, ny) / np.abs(u).max()
    m = make(segpu, nx, ny, N, (0.0, 0.0), (1.0, 1.0), per)
    f, fp = segpu.Field("psi", m, 1, None), segpu.Field("psiPrev", m, 1, None)
    v, vp = segpu.Field("vel", m, 2, None), segpu.Field("velPrev", m, 2, None)
    f.vals, fp.vals, v.vals, vp.vals = psi, psip, u, up
    adv = segpu.Advector(f, v, fp, vp)
    adv.record_departures()
    adv.Advect(dt)
    acc = om.advect(psi, u, dt, field_prev=psip, vel_prev=up, nthreads=8)
    assert np.abs(adv.fieldSL.vals - acc).max() <= ACC_TOL * np.abs(acc).max()
    el, xy = adv.departures()
    assert np.array_equal(om.global_to_local(xy[:om.nv])[0], el[:om.nv])
    assert np.array_equal(om.global_to_local(xy[om.nv:])[0], el[om.nv:])
    # two components, velocity advecting itself
    adv2 = segpu.Advector(v, v, vp, vp)
    adv2.Advect(dt)
    acc2 = om.advect(u, u, dt, field_prev=up, vel_prev=up, nthreads=8)
    assert np.abs(adv2.fieldSL.vals - acc2).max() <= ACC_TOL * np.abs(acc2).max()


@pytest.mark.parametrize("N", [4, 7])
@pytest.mark.parametrize("far", [2.0 ** 19 + 3.25, 2.0 ** 31 + 3.25, 2.0 ** 32 - 2.25, 2.0 ** 32 + 3.25,
                                 2.0 ** 33 - 1.75, 2.0 ** 40 + 4.5, 2.0 ** 50 + 2.25])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("side", [-1.0, 1.0])
def test_points_far_outside(segpu, N, far, axis, side):
    """A point billions of elements outside the mesh takes the value of the
    mesh's edge, as the reference's search clamped to the mesh gives it, and
    not that of the element its index is congruent to modulo 2^32. (The
    spacing is a power of two, so both coordinates are exact; the field is
    linear and the local coordinate clamped to an end node, so is the value.)"""
    nE = 8
    m = make(segpu, nE, nE, N, (0.0, 0.0), (2.0, 2.0), (False, False))
    X = m.verts
    f = segpu.Field("f", m, 1, None)
    f.vals = X[:, axis] + 1.0
    p = np.array([[0.3, 0.3]])
    p[0, axis] = side * far * 0.25
    got = f.InterpGlobal(p)[0, 0]
    el, lc = m.GlobalToLocal(p)
    end = nE - 1 if side > 0 else 0
    assert (el[0] % nE, el[0] // nE)[axis] == end and lc[0, axis] == side
    assert abs(got - (3.0 if side > 0 else 1.0)) <= 1e-12


def test_departures_far_outside_are_refused(segpu):
    """A flow of 2^33 elements a step is an error, not a gather at the element
    its departure points are congruent to."""
    m = make(segpu, 8, 8, 5, (0.0, 0.0), (1.1, 0.9), (True, True))
    f, v = segpu.Field("f", m, 1, None), segpu.Field("v", m, 2, None)
    f.vals = np.cos(m.verts[:, 0])
    for c in (2.0 ** 33 + 8, 2.0 ** 33 + 11.3, -(2.0 ** 33) - 9.1):
        v.vals = np.tile([c * 1.1 / 8, 0.0], (m.nVertsTotal, 1))
        adv = segpu.Advector(f, v)
        adv.record_departures()
        adv.Advect(1.0)
        with pytest.raises(segpu.SEError) as e:
            adv.departures()
        assert e.value.code == segpu.SE_ERR_DOMAIN


@pytest.mark.parametrize("order", [1, 2])
def test_tallest_meshes(segpu, order):
    """More rows of vertices than a grid's y dimension of blocks covers (65535
    blocks of 16): 349,526 elements of order 3 are 1,048,579. A field linear
    in y under a uniform flow is moved by the displacement, cut off at the
    walls; coordinates near 3.5e5 are known to 6e-11."""
    ny = 349526
    m = make(segpu, 1, ny, 3, (0.0, 0.0), (1.0, float(ny)), (False, False))
    y = m.verts[:, 1]
    f, v = segpu.Field("f", m, 1, None), segpu.Field("v", m, 2, None)
    f.vals = y
    v.vals = np.tile([0.0, 0.7], (m.nVertsTotal, 1))
    if order == 1:
        adv, want = segpu.Advector(f, v), np.maximum(y - 0.7, 0.0)
    else:  # 2 f(x1) - f(x2) / 2 with both levels of the field equal
        adv = segpu.Advector(f, v, f, v)
        want = 2.0 * np.maximum(y - 0.7, 0.0) - 0.5 * np.maximum(y - 1.4, 0.0)
    adv.Advect(1.0)
    assert np.abs(adv.fieldSL.vals - want).max() <= 1e-9
