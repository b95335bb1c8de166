"""The wet elements' right-hand side held node by node, each to its own terms:
elements whose depth or current varies strongly keep FP64's precision at their
shallow and slow nodes, whichever of the two paths takes them."""

import numpy as np
import pytest

from dgcom_gb300 import abi
from dgcom_gb300.device import DeviceRun, SWEPhysics2D
from dgcom_gb300.mesh import TAG_WALL, uniform_rectangle
from dgcom_gb300.physics import SWEDeviceForm2D, WallBoundary
from oracle_lib import oracle

pytestmark = pytest.mark.gpu

SIDE = 100.0


def rectangle(order, ratio, shear, nx=2, ny=3, aspect=1.0):
    """Depths falling by ``ratio`` over each element along x, currents along x
    falling by ``shear`` over each element along y; continuous, so that a face's
    flux is its nodes' own."""
    dy = SIDE / aspect
    mesh = uniform_rectangle(0.0, nx * SIDE, 0.0, ny * dy, nx, ny)
    form = SWEDeviceForm2D(mesh=mesh, order=order)
    x, y = form.positions()
    h = 20.0 * np.power(float(ratio), -x / SIDE)
    form.bathymetry = -h
    form.boundaries = {TAG_WALL: WallBoundary()}
    hu = 0.3 * h * np.power(float(shear), -y / dy)
    return form, (h.reshape(-1), hu.reshape(-1), 1e-3 * hu.reshape(-1))


def derivative(order):
    p = np.polynomial.legendre
    c = np.zeros(order + 1)
    c[-1] = 1.0
    x = np.concatenate([[-1.0], np.sort(p.legroots(p.legder(c)).real), [1.0]]) if order > 1 \
        else np.array([-1.0, 1.0])
    at = p.legval(x, c)
    with np.errstate(divide="ignore"):
        d = at[:, None] / at[None, :] / (x[:, None] - x[None, :])
    np.fill_diagonal(d, 0.0)  # a node's pair with itself is no pair
    return np.abs(d)


def own_terms(form, q, dy):
    """Each node's largest pair terms: of mass, and of the two momenta's pressure."""
    n1 = form.order + 1
    h, hu, hv = (a.reshape(-1, n1, n1) for a in q)
    d = derivative(form.order)

    def along_x(pair):
        return (d[None, None] * np.abs(pair)).max(axis=3) * 2.0 / SIDE

    def along_y(pair):
        return np.swapaxes((d[None, None] * np.abs(pair)).max(axis=3), 1, 2) * 2.0 / dy

    def plus(a):
        return a[:, :, :, None] + a[:, :, None, :]

    def times(a):
        return a[:, :, :, None] * a[:, :, None, :]

    t = lambda a: np.swapaxes(a, 1, 2)
    mass = np.maximum(along_x(plus(hu)), along_y(plus(t(hv))))
    return [m.reshape(-1) for m in (mass, 9.81 * along_x(times(h)), 9.81 * along_y(times(t(h))))]


def check_nodes(form, q, own):
    """Device and oracle both round a node's some thirty operations at 2^-53 of
    terms of this size: together 64 of these."""
    dev, ref = SWEPhysics2D(form, 0), oracle(form)
    try:
        for s in (dev, ref):
            s.upload(*q)
        for name, g, w, o in zip(("h", "hu", "hv"), dev.compute_rhs_into(0.0),
                                 ref.compute_rhs_into(0.0), own):
            err = (np.abs(g - w) / o).max()
            assert err <= 64.0 * 2.0 ** -53, f"{name}: {err:.3e} of a node's own terms"
    finally:
        dev.close()
        ref.close()


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("ratio, shear, aspect", [
    (1.05, 1.0, 1.0), (1.5, 1.0, 1.0), (2.0, 1.0, 1.0), (2.5, 1.0, 1.0), (4.0, 1.0, 1.0),
    (30.0, 1.0, 1.0), (1.05, 8.0, 1.0), (1.05, 64.0, 1.0), (1.05, 1.0, 30.0),
    (8.0, 100.0, 4.0)])
def test_every_node_to_its_own_terms(order, ratio, shear, aspect):
    form, q = rectangle(order, ratio, shear, aspect=aspect)
    check_nodes(form, q, own_terms(form, q, SIDE / aspect))


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("shear", [1e4, 1e6])
def test_currents_far_below_the_waves(order, shear):
    """Faces whose currents are 1e-13 to 1e-19 of the wave's speed."""
    form, q = rectangle(order, 1.05, shear)
    check_nodes(form, q, own_terms(form, q, SIDE))


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("shelf", [5.0, 0.1])
def test_a_shelf_beside_deep_water(order, shelf):
    """A step of the bed along an element edge, one surface over it: the shelf's
    nodes to their own depth's terms."""
    form, _ = rectangle(order, 1.0, 1.0)
    x, _ = form.positions()
    column = (x.mean(axis=1) > SIDE)[:, None] & np.ones_like(x, dtype=bool)
    form.bathymetry = np.where(column, 0.137 - shelf, 0.137 - 20.0)
    h = 0.137 - form.bathymetry
    q = (h.reshape(-1), 0.01 * h.reshape(-1), 0.02 * h.reshape(-1))
    check_nodes(form, q, own_terms(form, q, SIDE))


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("ratio, shear", [(2.5, 1.0), (1.05, 1e3)])
def test_a_sum_into_the_stage_s_input(order, ratio, shear):
    """The buffer that a stage is summed into may be its input: the same bits as
    into a copy of it, though a slow node reads its element's other nodes."""
    form, q = rectangle(order, ratio, shear, nx=40, ny=9)
    dev = SWEPhysics2D(form, 0)
    try:
        got = []
        for acc in (3, 1):
            for buffer in (abi.STATE, 1, 3):
                dev.upload(*q, buffer=buffer)
            dev.stage_where(base=abi.STATE, input=1, out=2, time=0.0, a=1.0, b=0.0, c=0.01,
                            acc=acc, w=0.5, keep=0.25)
            got.append(dev.download(2) + dev.download(acc))
        for g, w in zip(*got):
            assert np.array_equal(g, w)
    finally:
        dev.close()


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("ratio, shear", [(2.5, 1.0), (1.05, 1e3)])
def test_a_run_over_them_equals_its_calls(order, ratio, shear):
    """Listed before the stage (by their depths) or by it (by their fluxes), and
    taken beside it or behind it: the same bits."""
    form, q = rectangle(order, ratio, shear, nx=5, ny=7)
    dev = SWEPhysics2D(form, 0)
    try:
        dev.upload(*q)
        t = 0.0
        for _ in range(3):
            dt = dev.compute_dt_ssp(0.5)
            dev.step(t, dt, abi.SSP_RK3)
            t += dt
        want = dev.download()
        dev.upload(*q)
        dev.run_with_callback(DeviceRun(span=(0.0, 1e9), cfl=0.5, max_steps=3))
        for g, w in zip(dev.download(), want):
            assert np.array_equal(g, w)
    finally:
        dev.close()
