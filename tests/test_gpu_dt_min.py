"""The smallest step's own kernel while its bound moves: every element's step
is below all before it, so that each block lowers the bound that the others
read."""

import numpy as np
import pytest

from dgcom_gb300 import abi
from dgcom_gb300.device import DeviceRun, SWEPhysics2D
from dgcom_gb300.mesh import TAG_WALL, uniform_rectangle
from dgcom_gb300.physics import SWEDeviceForm2D, WallBoundary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numerics", [abi.NUMERICS_FAST, abi.NUMERICS_EXACT])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_the_smallest_of_falling_steps(numerics, order):
    mesh = uniform_rectangle(0.0, 200.0, 0.0, 150.0, 200, 150)
    form = SWEDeviceForm2D(mesh=mesh, order=order, numerics=numerics)
    form.boundaries = {TAG_WALL: WallBoundary()}
    nn = (order + 1) ** 2
    k = np.arange(mesh.n_elements)
    # 5e-5 an element, above the float filter's 2^-16, and one node the fastest
    h = np.repeat((1.0 + 1e-4 * k)[:, None], nn, axis=1)
    u = np.zeros_like(h)
    u[k, k % nn] = 0.5
    dev = SWEPhysics2D(form, 0)
    try:
        for way in (1, -1):
            q = h[::way].reshape(-1), (h * u)[::way].reshape(-1), np.zeros(h.size)
            for _ in range(5):
                dev.upload(*q)
                want = dev.element_dt(0.5).min()
                report = dev.run_with_callback(DeviceRun(span=(0.0, 1e9), cfl=0.5, max_steps=1))
                assert report.n_steps == 1 and report.dt_min == want
    finally:
        dev.close()
