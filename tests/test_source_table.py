"""The sources' values are computed in pieces of 256 steps: a job stepped one
step or one procedure at a time across their ends takes the same values as one
stepped in a single call."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [1, 254])
@pytest.mark.parametrize("precision", [abi.F32, abi.F64])
def test_steps_one_by_one_equal_one_call(precision, first):
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    spec, _ = problems.config_2d_tmz(precision=precision, n=64, ncyl=1, nfreq=4, npml=8)
    outs = []
    for way in range(3):
        J = job.Job(spec)
        if first > 1:
            J.step(1, first - 1)
        if way == 0:
            J.step(first, 520)
        for n in range(first, first + 520):
            if way == 1:
                J.step(n, 1)
            elif way == 2:
                J.step_procedures(n)
        outs.append([J.get_field(c) for c in (abi.EZ, abi.HX, abi.HY)] + list(J.get_monitor(0)))
        J.close()
    assert np.any(outs[0][0])
    for got in outs[1:]:
        for a, b in zip(got, outs[0]):
            np.testing.assert_array_equal(a, b)
