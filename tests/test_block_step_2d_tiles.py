"""Both tile shapes of the 2D block-step kernel against the half-step kernels, bit
for bit, with the kernel chosen by environment, so that no timing decides what
is compared: the tall shape (taken once its tiles outnumber the SMs) with odd
rows, periodic axes, several materials, many sampled rows and tiles whose
dispersive state goes past shared memory; the low shape where it cannot be
pinned."""
import numpy as np
import pytest

from fdtd_gpu import abi
from test_block_step_2d import BLOCK, gpu, make, result  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("te", [False, True])
@pytest.mark.parametrize("nx,ny,kw", [
    # 112 x 48 cells owned: 13 x 14 tiles and more
    (1344, 672, {}), (1345, 673, dict(sub=True, lorentz=True)), (1347, 625, dict(vertical=True, lorentz=True)),
    (1348, 630, dict(per=(1, 0), sub=True)), (1401, 671, dict(pml=0, per=(1, 1), lorentz=True)),
    (1920, 1200, dict(sub=True, vertical=True)),
    # 112 x 16 cells owned
    (227, 81, dict(vertical=True, lorentz=True)), (231, 90, dict(pml=0, per=(1, 1), vertical=True)),
])
def test_block_step_equals_half_steps(gpu, monkeypatch, te, nx, ny, kw):  # noqa: F811
    monkeypatch.setenv("FDTD_TUNE", "block")
    spec = make(nx, ny, te, **kw)
    calls = (1, 2, 5, 8, 9, 64, 31)
    used, got = result(gpu, spec, calls)
    assert used == BLOCK
    split, ref = result(gpu, spec, (sum(calls),), tile=2)
    assert split == 2 and any(np.any(r) for r in ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("te", [False, True])
def test_single_steps_of_a_large_grid_run_split(gpu, te):  # noqa: F811
    """One step from the canonical field set takes the half-step kernels where the
    block-step kernel's halo costs more (2048^2: 22 us against 55), and few
    steps after an odd number of launches still come from the current set."""
    spec = make(2048, 2048, te)
    J = gpu.Job(spec)
    if J.tile() == BLOCK:
        J.profile()
        for n in range(1, 9):
            J.step(n, 1)
        J.sync()
        assert J.kernel_time(abi.KERNEL_E)[0] == 8 and J.kernel_time(abi.KERNEL_STEP)[0] == 0
    J.close()
    calls = (1, 1, 8, 1, 1, 2, 8, 3, 64, 1)
    got, ref = result(gpu, spec, calls)[1], result(gpu, spec, (sum(calls),), tile=2)[1]
    assert any(np.any(r) for r in ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("te", [False, True])
@pytest.mark.parametrize("nx,ny,kw", [
    (1345, 673, {}), (560, 300, {}), (449, 131, dict(pml=0, per=(1, 1), lorentz=True)), (225, 96, dict(per=(1, 0))),
])
def test_columns_of_samples_and_sources(gpu, monkeypatch, te, nx, ny, kw):  # noqa: F811
    """Line monitors and sources along y and probes, on and beside the first and
    last column that a tile owns (112 of them) and at the ends of the grid."""
    monkeypatch.setenv("FDTD_TUNE", "block")
    spec = make(nx, ny, te, **kw)
    e, h = (abi.EX, abi.HZ) if te else (abi.EZ, abi.HX)
    om = spec.monitors[0].omega
    for x in (0, 111, 112, 223, nx - 1):
        spec.add_monitor((x, 3, 0), (x, ny - 4, 0), (e, h), om)
        spec.add_probe((x, ny // 2, 0), (e, h))
    spec.add_monitor((100, 20, 0), (130, 40, 0), (h, e), om)
    spec.add_monitor((0, 0, 0), (nx - 1, ny - 1, 0), (e, abi.EY if te else abi.HY, h), om[:1])
    for x in (lo for lo in (spec.main_lo[0], 105, 112) if lo <= spec.main_hi[0]):
        spec.sources.append(dict(component=e, lo=(x, 5, 0), hi=(x, ny - 6, 0), amp=0.3, t0=1e-16, st=2e-16, w0=3e15))
    calls = (3, 8, 64, 17, 31)
    used, got = result(gpu, spec, calls)
    assert used == BLOCK
    ref = result(gpu, spec, (sum(calls),), tile=2)[1]
    for a, b in zip(got, ref):
        assert np.any(b)
        np.testing.assert_array_equal(a, b)
