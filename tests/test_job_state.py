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


@pytest.mark.parametrize("dim", [1, 2, 3])
def test_failed_launch_is_an_error_and_no_step(gpu, monkeypatch, dim):
    """The first launch of a step fails: the step reports it, and the same call
    again takes the step from the state before it."""
    monkeypatch.setenv("FDTD_TUNE", "block")
    if dim == 1:
        spec, _ = problems.config_1d_gold(precision=abi.F32)
        comps = (abi.EX, abi.HZ)
    elif dim == 2:
        spec, _ = problems.config_2d_tmz(precision=abi.F32, n=192, ncyl=2, nfreq=8, npml=16)
        comps = FIELDS_TM
    else:
        spec, _ = problems.config_3d_sphere(precision=abi.F32, n=48, nfreq=4, npml=8)
        comps = range(6)
    outs = []
    for fail in (False, True):
        J = gpu.Job(spec)
        J.step(1, 6)
        if fail:
            try:
                gpu.fail_launch_after(0)
                with pytest.raises(gpu.FdtdError) as e:
                    J.step(7, 8)
                assert e.value.code == abi.FDTD_ECUDA
            finally:
                gpu.fail_launch_after(-1)
        J.step(7, 8)
        J.step(15, 300)
        outs.append(state_of(J, comps))
        J.close()
    assert any(np.any(a) for a in outs[0])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


def test_kernel_that_fails_in_the_tuner_is_left_out(gpu):
    spec, _ = problems.config_2d_tmz(precision=abi.F32, n=163, ncyl=1, nfreq=6, npml=12)
    spec.materials = spec.materials[:1]  # odd rows of vacuum: a kind of grid that no other test has timed in this process
    try:
        gpu.fail_launch_after(0)
        J = gpu.Job(spec)
    finally:
        gpu.fail_launch_after(-1)
    assert J.tile() in (1, 2, 3)
    J.step(1, 200)
    K = gpu.Job(spec)  # the failure is not kept: the kernel is a candidate again
    assert K.tile() == 4
    K.step(1, 200)
    for a, b in zip(state_of(J, FIELDS_TM), state_of(K, FIELDS_TM)):
        np.testing.assert_array_equal(a, b)
    J.close()
    K.close()


@pytest.mark.parametrize("dim,tile", [(2, 0), (3, 0), (3, 9)])
@pytest.mark.parametrize("after", [1, 2])
def test_failed_capture_leaves_the_state(gpu, monkeypatch, dim, tile, after):
    """The capture of a ring of steps stops after an odd or even number of
    recorded launches: nothing has run, so the job's fields are where they were."""
    monkeypatch.setenv("FDTD_TUNE", "block")
    if dim == 2:
        spec, _ = problems.config_2d_tmz(precision=abi.F32, n=192, ncyl=2, nfreq=8, npml=16)
        comps = FIELDS_TM
    else:
        spec, _ = problems.config_3d_sphere(precision=abi.F32, n=64, nfreq=4, npml=8)
        comps = range(6)
    outs = []
    for fail in (False, True):
        J = gpu.Job(spec, tile=tile)
        if fail:
            try:
                gpu.fail_launch_after(after)
                with pytest.raises(gpu.FdtdError) as e:
                    J.step(1, 320)
                assert e.value.code == abi.FDTD_ECUDA
            finally:
                gpu.fail_launch_after(-1)
            assert all(not np.any(J.get_field(c)) for c in comps)
        J.step(1, 320)
        outs.append(state_of(J, comps))
        J.close()
    assert any(np.any(a) for a in outs[0])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("after", [1, 5])
def test_failed_pack_capture_leaves_the_members(gpu, monkeypatch, after):
    """The capture of a pack's ring stops part way in its first or second job: the
    members go on alone, from their own fields."""
    from fdtd_gpu import serve
    monkeypatch.setenv("FDTD_TUNE", "block")
    specs = [problems.config_2d_tmz(precision=abi.F32, n=n, ncyl=2, nfreq=8, npml=16, seed=n)[0] for n in (160, 192)]
    alone = []
    for s in specs:
        J = gpu.Job(s)
        J.step(1, 900)
        alone.append(state_of(J, FIELDS_TM))
        J.close()
    S = serve.Server(max_active=4, chunk_steps=64)
    try:
        gpu.fail_launch_after(after)
        tickets = [S.submit(s, 900) for s in specs]
        for tk, want in zip(tickets, alone):
            assert S.wait(tk) == abi.REQ_DONE
            got = state_of(S.job(tk), FIELDS_TM)
            assert any(np.any(a) for a in want)
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
            S.release(tk)
    finally:
        gpu.fail_launch_after(-1)
        S.close()


def test_line_without_room_for_a_second_set(gpu):
    """A 1D job whose second set of buffers cannot be had runs in the kernel that
    needs none, with the same results; other allocations of set-up still fail it."""
    spec, _ = problems.config_1d_gold(precision=abi.F64)
    ref = gpu.Job(spec)
    full = ref.device_bytes()
    ref.step(1, 700)
    want = state_of(ref, (abi.EX, abi.HZ))
    ref.close()
    refused = without = 0
    try:
        for k in range(200):
            gpu.fail_alloc_after(k)
            try:
                J = gpu.Job(spec)
            except gpu.FdtdError as e:
                assert e.code == abi.FDTD_ENOMEM
                refused += 1
                continue
            gpu.fail_alloc_after(-1)
            if J.device_bytes() == full:
                J.close()
                break
            without += 1
            J.step(1, 700)
            for a, b in zip(state_of(J, (abi.EX, abi.HZ)), want):
                np.testing.assert_array_equal(a, b)
            J.close()
    finally:
        gpu.fail_alloc_after(-1)
    assert refused > 10 and without >= 4
