"""The commit-time choice of the step kernel: what is kept for one kind of grid
must not be taken for another."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems
from fdtd_gpu.spec import mask

pytestmark = pytest.mark.gpu

BLOCK3 = 10


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


def test_mixed_materials_are_a_kind_of_their_own(gpu):
    """A grid whose rows all mix two materials takes the 3D block-step kernel's
    general rows everywhere, 1.6 times the split step at 320^3, and must not
    inherit the choice of a plain grid committed before it."""
    spec, _ = problems.config_3d_sphere(precision=abi.F32, n=320, nfreq=2, npml=12)
    spec.materials = spec.materials[:1]
    J = gpu.Job(spec)
    J.close()
    spec.add_dielectric(mask(np.random.default_rng(1).random((320, 320, 320)) < 0.5), 2.25)
    J = gpu.Job(spec)
    used = J.tile()
    J.close()
    assert used != BLOCK3


def test_a_line_of_sources_is_a_kind_of_its_own(gpu):
    """A line of sources along z puts a row of general rounds into every plane of a
    tile, 1.6 times the split step at 400^3; the grid without it takes the 3D
    block-step kernel."""
    spec, _ = problems.config_3d_sphere(precision=abi.F32, n=400, nfreq=2, npml=12)
    spec.monitors = []
    J = gpu.Job(spec)
    J.close()
    spec.sources.append(dict(spec.sources[0], lo=(200, 200, 0), hi=(200, 200, 399)))
    J = gpu.Job(spec)
    used = J.tile()
    J.close()
    assert used != BLOCK3
