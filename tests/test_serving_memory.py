"""Admission under a short budget: the second sets of buffers that the block-step
kernels hold must not keep a job waiting for the end of another one that it fits
beside without them."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems, serve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


def estimate(gpu, spec):
    J = gpu.Job(spec, commit=False)
    n = J.estimate_bytes()
    J.close()
    return n


@pytest.mark.parametrize("kind", ["te", "sphere"])
def test_short_job_runs_beside_a_long_one(gpu, kind):
    if kind == "te":
        long, short = (problems.as_te(problems.config_2d_tmz(precision=abi.F32, n=n, ncyl=4, nfreq=8)[0]) for n in (1024, 768))
    else:
        long, short = (problems.config_3d_sphere(precision=abi.F32, n=n, nfreq=4, npml=12)[0] for n in (208, 200))
    J = gpu.Job(short)
    J.step(1, 96)
    want = [J.get_monitor(q) for q in range(len(short.monitors))]
    J.close()
    # the long job and four fifths of the short one's footprint
    S = serve.Server(hbm_budget=int(estimate(gpu, long) + 0.8 * estimate(gpu, short)), max_active=4, chunk_steps=64,
                     pack_cells=-1)
    a = S.submit(long, 2000000)
    b = S.submit(short, 96)
    assert S.wait(b, 20000) == abi.REQ_DONE
    assert S.wait(a, 0) == abi.REQ_RUNNING
    for (x, y), (p, q) in zip(want, (S.job(b).get_monitor(q) for q in range(len(short.monitors)))):
        np.testing.assert_array_equal(x, p)
        np.testing.assert_array_equal(y, q)
    assert S.stats()["held_bytes_max"] <= S.stats()["budget_bytes"]
    S.close()
