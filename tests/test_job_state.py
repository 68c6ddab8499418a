"""State that a job keeps on both sides of a call: checkpoint buffers the caller
may reuse, and the two field sets of the block-step kernels when a call fails
part way."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems

pytestmark = pytest.mark.gpu

FIELDS_TM = (abi.EZ, abi.HX, abi.HY)


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


def state_of(J, comps):
    return [J.get_field(c) for c in comps] + [x for q in range(len(J.spec.monitors)) for x in J.get_monitor(q)]


def test_load_state_leaves_the_callers_buffer_free(gpu):
    """A page-locked checkpoint buffer is read by the device itself: when
    fdtd_load_state returns, the caller may already refill it."""
    torch = pytest.importorskip("torch")
    spec, _ = problems.config_2d_tmz(precision=abi.F32, n=2048, ncyl=4, nfreq=100)
    J = gpu.Job(spec)
    J.step(1, 40)
    want = J.save_state()
    pinned = torch.empty(want.size, dtype=torch.uint8, pin_memory=True).numpy()
    tail = want.size // 2
    for _ in range(5):
        pinned[:] = want
        J.step(41, 3)
        J.load_state(pinned)
        pinned[tail:] = 0x3f
        np.testing.assert_array_equal(J.save_state(), want)
    J.close()
