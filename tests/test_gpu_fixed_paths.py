"""The dispatches around the fixed-point stage: what each path gives where
its rule draws the line, against the oracle, and the smallest step's own
kernel against the element steps.

A stage state is held to 1e-12 of its field's largest value, as every stage
is; a right-hand side to 1e-10 (test_gpu_parity.py has the reasons)."""

import numpy as np
import pytest

from dgcom_gb300 import abi, cases
from dgcom_gb300.device import DeviceRun, SWEPhysics2D
from oracle_lib import oracle
from test_gpu_parity import TOL, TOL_RHS, rel_err

pytestmark = pytest.mark.gpu

# depth spreads within an element (2^9 is the fixed point's limit), Froude
# numbers above one, films below the subcells' depth and dry land beside
# water. (At rest the right-hand side is rounding alone, which no relative
# comparison can judge: test_a_lake_at_rest below.)
STATES = ["spread", "fast", "film", "shore"]


def state(form, kind, seed=5):
    rng = np.random.default_rng(seed)
    x, _ = form.positions()
    b = form.bathymetry.reshape(-1)
    n = b.size
    h = np.maximum(0.3 - b, 0.0)
    if kind == "shore":
        h = np.maximum(-0.2 - b, 0.0)
    elif kind == "spread":
        h = 0.02 * np.exp2(rng.uniform(0.0, 12.0, n))
    elif kind == "film":
        h = np.where(rng.random(n) < 0.3, 1e-4 * rng.random(n), 0.5 + rng.random(n))
    speed = {"rest": 0.0, "fast": 2.0 * np.sqrt(9.81 * h)}.get(kind, 0.4)
    u = speed * (0.6 + 0.4 * np.cos(x.reshape(-1) / 3000.0))
    wet = h > 1e-3
    return h, np.where(wet, h * u, 0.0), np.where(wet, -0.5 * h * u, 0.0)


@pytest.mark.parametrize("kind", STATES)
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("curved", [False, True])
def test_stage_paths_match_the_oracle(kind, order, curved):
    form = cases.shoreline_setup(order, False, False, curved=curved, wet_dry=True)
    form.manning_n = 0.02
    dev, ref = SWEPhysics2D(form, 0), oracle(form)
    try:
        q = state(form, kind)
        for s in (dev, ref):
            s.upload(*q)
        err = rel_err(dev.compute_rhs_into(0.0), ref.compute_rhs_into(0.0))
        assert err <= TOL_RHS, f"relative RHS difference {err:.3e}"
        dt = ref.compute_dt_ssp(0.5)
        for s in (dev, ref):
            s.step(0.0, dt, abi.SSP_RK3)
        err = rel_err(dev.download(), ref.download())
        assert err <= TOL, f"relative step difference {err:.3e}"
    finally:
        dev.close()
        ref.close()


@pytest.mark.parametrize("speed", [0.0, 1e-30])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_a_lake_at_rest(order, speed):
    """Still water over a bed (and a current far below its rounding): the
    momentum's right-hand side is rounding, and no larger than the oracle's;
    the depth's is zero or of the current's size."""
    form = cases.split_form_setup(order, False, "smooth", curved=True)
    dev, ref = SWEPhysics2D(form, 0), oracle(form)
    try:
        q = cases.split_form_state(form, speed)
        for s in (dev, ref):
            s.upload(*q)
        got, want = dev.compute_rhs_into(0.0), ref.compute_rhs_into(0.0)
        for g, w in zip(got[1:], want[1:]):
            assert np.abs(g).max() <= np.abs(w).max()
        assert np.abs(got[0]).max() <= 2.0 * np.abs(want[0]).max()
    finally:
        dev.close()
        ref.close()


@pytest.mark.parametrize("numerics", [abi.NUMERICS_FAST, abi.NUMERICS_EXACT])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["rest", "fast", "film", "shore"])
def test_a_runs_step_is_the_smallest_element_step(numerics, order, kind):
    """A run takes the smallest step by its own kernel: the element steps'
    minimum, bit for bit."""
    form = cases.shoreline_setup(order, False, True, curved=True, wet_dry=True, numerics=numerics)
    dev = SWEPhysics2D(form, 0)
    try:
        dev.upload(*state(form, kind))
        want = dev.element_dt(0.5).min()
        report = dev.run_with_callback(DeviceRun(span=(0.0, 1e9), cfl=0.5, max_steps=1))
        assert report.n_steps == 1 and report.dt_min == want
    finally:
        dev.close()


@pytest.mark.parametrize("nx, ny, shallow", [(37, 5, 0), (37, 5, 1), (37, 5, 107), (37, 5, 108),
                                             (37, 5, 109), (37, 5, 185), (400, 20, 1216),
                                             (400, 20, 1217)])
def test_subcell_lists_of_any_length(nx, ny, shallow):
    """At order 2 a short list of subcell elements has a warp for each (up to
    four a block of the launch, and 1216 in all), a longer one packs them."""
    form = cases.tidal_channel(nx=nx, ny=ny, order=2).form
    dev, ref = SWEPhysics2D(form, 0), oracle(form)
    try:
        rng = np.random.default_rng(11)
        h = 0.5 + rng.random((nx * ny, 9))
        h[rng.permutation(nx * ny)[:shallow], 4] = 1e-4
        h = h.reshape(-1)
        for s in (dev, ref):
            s.upload(h, 0.4 * h, -0.2 * h)
        err = rel_err(dev.compute_rhs_into(0.0), ref.compute_rhs_into(0.0))
        assert err <= TOL_RHS, f"relative RHS difference {err:.3e}"
    finally:
        dev.close()
        ref.close()


@pytest.mark.parametrize("members", [1, 3])
@pytest.mark.parametrize("order", [2, 3])
def test_a_run_equals_its_calls(order, members):
    """The step graph (subcell elements listed beside the face pass and taken
    beside the others) gives what the calls one by one give, bit for bit,
    and an ensemble's members theirs."""
    from dgcom_gb300.ensemble import Ensemble

    forms = [cases.tidal_channel(nx=37 + m, ny=5, order=order).form for m in range(members)]
    states = [cases.with_flow(cases.Case(f, None, 0.5, abi.SSP_RK3, 0.0)) for f in forms]
    want = []
    for f, q in zip(forms, states):
        dev = SWEPhysics2D(f, 0)
        dev.upload(*q)
        t = 0.0
        for _ in range(5):
            dt = dev.compute_dt_ssp(0.5)
            dev.step(t, dt, abi.SSP_RK3)
            t += dt
        want.append(dev.download())
        dev.upload(*q)
        dev.run_with_callback(DeviceRun(span=(0.0, 1e9), cfl=0.5, max_steps=5))
        for g, w in zip(dev.download(), want[-1]):
            assert np.array_equal(g, w)
        dev.close()
    with Ensemble(forms) as ens:
        for m, q in enumerate(states):
            ens.upload(m, *q)
        ens.run(5, 0.5)
        for m in range(members):
            for g, w in zip(ens.download(m), want[m]):
                assert np.array_equal(g, w)
