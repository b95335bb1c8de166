"""dgswe_step_host where the state is cut into several element chunks (8 MiB of
state each, eight at most): the upload, dt and face passes as the chunks arrive,
and the last stage and its copies back chunk by chunk, against the same steps
taken call by call; the same bits. The meshes of test_gpu_step_host.py are one
chunk each."""

import numpy as np
import pytest

from dgcom_gb300 import abi, cases
from dgcom_gb300.device import SWEPhysics2D
from test_gpu_step_host import pinned

pytestmark = pytest.mark.gpu

CHUNK = 8 << 20


def steps_equal_the_calls(case, chunks, held, scheme=abi.SSP_RK3, steps=2):
    q0 = cases.with_flow(case)
    assert 3 * q0[0].nbytes // CHUNK >= chunks if chunks == 8 else 3 * q0[0].nbytes // CHUNK == chunks
    a, b = SWEPhysics2D(case.form, 0), SWEPhysics2D(case.form, 0)
    try:
        host = [held(x) for x in q0]
        b.upload(*q0)
        t = 7200.0
        for _ in range(steps):
            dt = a.step_host(t, case.cfl, *host, scheme=scheme)
            want_dt = b.compute_dt_ssp(case.cfl, scheme)
            assert dt == want_dt
            b.step(t, want_dt, scheme)
            want = b.download()
            for g, w in zip(host, want):
                assert np.array_equal(g, w)
            for g, w in zip(a.download(), want):
                assert np.array_equal(g, w)
            t += dt
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("held", [pinned, np.array])
@pytest.mark.parametrize("nx, ny, order, chunks", [
    (200, 141, 4, 2),   # the fewest elements that make two
    (257, 256, 3, 3),   # a last chunk that is shorter
    (400, 280, 4, 8),   # just eight
    (500, 352, 1, 2),   # the most elements a chunk
])
def test_chunks_of_a_channel(held, nx, ny, order, chunks):
    steps_equal_the_calls(cases.tidal_channel(nx, ny, order), chunks, held)


@pytest.mark.parametrize("numerics", [abi.NUMERICS_FAST, abi.NUMERICS_EXACT])
@pytest.mark.parametrize("scheme", [abi.SSP_RK3, abi.SSP_RK43])
def test_chunks_of_an_unstructured_box(numerics, scheme):
    """Faces and dt neighbours across chunks, islands with drying shores."""
    case = cases.coastal_box(90_000, 3, lx=60_000.0, ly=45_000.0, n_islands=3, numerics=numerics)
    steps_equal_the_calls(case, 4, pinned, scheme)
