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
