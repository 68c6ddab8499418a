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


def test_refused_load_state_leaves_the_state(gpu):
    """A checkpoint whose probe records do not fit in device memory is refused;
    the job, whose fields are in the second set, goes on with its own."""
    spec, _ = problems.config_2d_tmz(precision=abi.F32, n=192, ncyl=2, nfreq=8, npml=16)
    spec.add_probe((96, 96, 0), (abi.EZ,))
    A = gpu.Job(spec, tile=4)
    A.step(1, 1500)  # more probe records than a new job's buffer holds
    long = A.save_state()
    A.close()
    J = gpu.Job(spec, tile=4)
    J.step(1, 8)
    rng = np.random.default_rng(1).standard_normal((1, 192, 192))
    rng[:, :16] = rng[:, -16:] = rng[:, :, :16] = rng[:, :, -16:] = 0
    J.set_field(abi.EZ, rng)
    J.step(9, 8)  # one launch: the current fields are in the second set
    K = gpu.Job(spec, tile=4)
    K.load_state(J.save_state())
    J.step(17, 8)
    K.step(17, 8)
    try:
        gpu.fail_alloc_after(0)
        with pytest.raises(gpu.FdtdError) as e:
            J.load_state(long)
        assert e.value.code == abi.FDTD_ENOMEM
    finally:
        gpu.fail_alloc_after(-1)
    J.step(25, 40)
    K.step(25, 40)
    for a, b in zip(state_of(J, FIELDS_TM), state_of(K, FIELDS_TM)):
        np.testing.assert_array_equal(a, b)
    assert np.any(J.get_field(abi.EZ))
    J.close()
    K.close()
