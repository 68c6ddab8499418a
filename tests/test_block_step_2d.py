"""The 2D block-step kernel (several steps of a tile per launch, FP32) against
the half-step kernels, bit for bit, where its tiles end: grids a cell short of,
at and past a tile's 112 columns and 16 or 48 rows, odd row lengths, periodic
axes, every length of a launch, materials, sources and samples on the seams."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems
from fdtd_gpu.spec import JobSpec, box, spheres

pytestmark = pytest.mark.gpu

BLOCK = 4  # the tile number of the block-step kernel


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


def make(nx, ny, te, pml=8, per=(0, 0), gold=True, lorentz=False, sub=False, vertical=False):
    ds = 1e-9
    lo = [0 if p else pml for p in per]
    spec = JobSpec(layout=abi.LAYOUT_2D_TE if te else abi.LAYOUT_2D_TM, n=(nx, ny, 1), ku=0.5, dt=0.5 * ds / problems.C0,
                   ds=ds, periodic=(per[0], per[1], 0), precision=abi.F32, main_lo=(lo[0], lo[1], 0),
                   main_hi=(nx - 1 - lo[0], ny - 1 - lo[1], 0))
    spec.add_dielectric(box((0, 0, 0), (nx - 1, ny - 1, 0)), 1.0)
    if sub:
        spec.add_dielectric(box((lo[0], ny // 2, 0), (nx - 1 - lo[0], ny - 1 - lo[1], 0)), 2.25)
    if gold:
        spec.add_gold(spheres([(nx / 2, ny / 2, 0, min(nx, ny) / 5)]), problems.GOLD_CONFIG)
    if lorentz:
        spec.add_lorentz(box((lo[0] + 3, lo[1] + 2, 0), (lo[0] + 12, lo[1] + 9, 0)), problems.GOLD_JP)
    if pml:
        spec.pml = dict(mode=abi.PML_SPLIT, npml=((pml, pml), (pml, pml), (0, 0)), eps_lo=1.0,
                        sigma_max=problems.pml_sigma_max(3.0, np.exp(-16.0), pml, ds), order=3.0)
    e, h = (abi.EX, abi.HZ) if te else (abi.EZ, abi.HX)
    p = dict(t0=1e-16, st=2e-16, w0=3e15)
    spec.sources.append(dict(component=e, lo=(0, ny // 2, 0), hi=(nx - 1, ny // 2, 0), amp=1.0, **p))
    om = problems.dft_omegas(500e-9, 800e-9, 3)
    y = min(48, ny - 2)
    spec.add_monitor((0, y, 0), (nx - 1, y, 0), (e, h), om)
    if vertical:  # a column of samples and a second, overlapping source
        spec.add_monitor((nx // 2, 0, 0), (nx // 2, ny - 1, 0), (e, h), om)
        spec.sources.append(dict(component=e, lo=(4, ny // 2, 0), hi=(nx - 5, ny // 2 + 1, 0), amp=0.5, **p))
    spec.add_probe((nx // 2, y, 0), (e, h))
    return spec


def result(gpu, spec, calls, tile=0):
    J = gpu.Job(spec, tile=tile)
    rng = np.random.default_rng(7)
    te = spec.layout == abi.LAYOUT_2D_TE
    lo, hi = spec.main_lo, spec.main_hi
    x = np.zeros((1, spec.n[1], spec.n[0]))
    x[0, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1] = rng.standard_normal((hi[1] - lo[1] + 1, hi[0] - lo[0] + 1))
    J.set_field(abi.EX if te else abi.EZ, x)
    n = 1
    for k in calls:
        J.step(n, k)
        n += k
    out = [J.get_field(c) for c in ((abi.EX, abi.EY, abi.HZ) if te else (abi.EZ, abi.HX, abi.HY))]
    for q in range(len(spec.monitors)):
        out += list(J.get_monitor(q))
    out.append(J.get_probe(0))
    used = J.tile()
    J.close()
    return used, out


@pytest.mark.parametrize("te", [False, True])
@pytest.mark.parametrize("nx,ny,kw", [
    (112, 48, {}), (111, 47, {}), (113, 49, {}), (224, 96, {}), (228, 100, dict(sub=True)),
    (225, 65, dict(sub=True, lorentz=True)), (160, 144, dict(pml=0, per=(1, 1))),
    (125, 97, dict(pml=0, per=(1, 1), lorentz=True)), (64, 60, dict(pml=0, per=(1, 1))),
    (300, 130, dict(per=(1, 0))), (130, 300, dict(vertical=True)), (1920, 1200, dict(sub=True)),
])
def test_block_step_equals_half_steps(gpu, te, nx, ny, kw):
    spec = make(nx, ny, te, **kw)
    calls = (1, 2, 3, 5, 7, 8, 9, 64, 31, 33)
    # pinned where it can be; elsewhere the tuner keeps it for the small grids
    pin = BLOCK if not te and nx % 4 == 0 and not any(spec.periodic) else 0
    used, got = result(gpu, spec, calls, pin)
    assert used == BLOCK or nx > 1000, f"the tuner kept tile {used}"
    split, ref = result(gpu, spec, (sum(calls),), tile=2)
    assert split == 2 and any(np.any(r) for r in ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_block_step_state_through_every_entry_point(gpu):
    """After an odd number of launches the fields are in the second set of
    buffers: a field written, a checkpoint, the per-procedure step and the
    count of non-finite values have to find and leave the current one."""
    spec = make(200, 120, False)
    outs = []
    for tile in (BLOCK, 2):
        J = gpu.Job(spec, tile=tile)
        J.step(1, 3)
        J.set_field(abi.HX, J.get_field(abi.HX) + 0.25)
        J.step(4, 1)
        state = J.save_state()
        J.step(5, 8)
        J.load_state(state)
        J.step(5, 2)
        J.step_procedures(7)
        J.step(8, 5)
        assert J.count_nonfinite() == 0
        outs.append([J.get_field(c) for c in (abi.EZ, abi.HX, abi.HY)])
        J.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
