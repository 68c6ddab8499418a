"""The 1D block-step kernel (several steps of a stretch per launch) and the fold
of many rings against the step-at-a-time line kernel, bit for bit: lines a cell
short of, at and past a block's stretch (64 or 96 cells; 192 or 224 past the
SMs), both halves of odd step counts, slabs, the incident line, materials, and
more samples in a stretch and a monitor than are staged or folded together."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems
from fdtd_gpu.spec import JobSpec, box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


def make(n, precision, pml=6, tfsf=False, mat=None, wide=0):
    ds, ku = 1e-9, 0.99
    spec = JobSpec(layout=abi.LAYOUT_1D, n=(1, n, 1), ku=ku, dt=ku * ds / problems.C0, ds=ds, precision=precision,
                   main_lo=(0, pml, 0), main_hi=(0, n - pml - 1, 0))
    spec.add_dielectric(box((0, pml, 0), (0, n - pml - 1, 0)), 1.0)
    spec.add_dielectric(box((0, n // 2, 0), (0, n - pml - 1, 0)), 2.25)
    m = box((0, n // 2 - 5, 0), (0, n // 2 + 4, 0))
    if mat == "gold":
        spec.add_gold(m, problems.GOLD_CONFIG)
    elif mat == "lorentz":
        spec.add_lorentz(m, problems.GOLD_JP)
    elif mat == "both":
        spec.add_gold(m, problems.GOLD_CONFIG)
        spec.add_lorentz(box((0, n // 4, 0), (0, n // 4 + 2, 0)), problems.GOLD_JP)
    if pml:
        spec.pml = dict(mode=abi.PML_REFERENCE, npml=((0, 0), (pml, pml), (0, 0)), eps_lo=1.0, eps_hi=2.25,
                        sigma_max=problems.pml_sigma_max(3.0, np.exp(-16.0), pml, ds), order=3.0)
    p = dict(t0=1e-16, st=2e-16, w0=3e15)
    if tfsf:
        spec.tfsf = dict(boundary=pml + 9, eps_lo=1.0, eps_hi=1.0)
        spec.sources.append(dict(component=abi.EX_INC, lo=(0, pml + 3, 0), hi=(0, pml + 3, 0), amp=1.0, **p))
    spec.sources.append(dict(component=abi.EX, lo=(0, n // 3, 0), hi=(0, n // 3 + 2, 0), amp=0.5, **p))
    om = problems.dft_omegas(500e-9, 800e-9, 5)
    comps = (abi.EX, abi.HZ) + ((abi.EX_INC, abi.HZ_INC) if tfsf else ())
    spec.add_monitor((0, n // 2, 0), (0, n // 2, 0), comps, om, 20, 130)
    if wide:
        spec.add_monitor((0, n // 2 - 1, 0), (0, n // 2 + wide - 2, 0), comps[:2], om)
    spec.add_probe((0, n // 2, 0), comps)
    return spec


def result(gpu, spec, calls):
    J = gpu.Job(spec)
    n = spec.n[1]
    x = np.zeros((1, n, 1))
    lo, hi = spec.main_lo[1], spec.main_hi[1]
    x[0, lo:hi + 1, 0] = np.random.default_rng(3).standard_normal(hi - lo + 1)
    J.set_field(abi.EX, x)
    at = 1
    for k in calls:
        J.step(at, k)
        at += k
    out = [J.get_field(c) for c in (abi.EX, abi.HZ) + ((abi.EX_INC, abi.HZ_INC) if spec.tfsf else ())]
    for q in range(len(spec.monitors)):
        out += list(J.get_monitor(q))
    out.append(J.get_probe(0))
    J.close()
    return out


@pytest.mark.parametrize("precision", [abi.F32, abi.F64])
@pytest.mark.parametrize("n,kw", [
    (40, dict(pml=0)), (63, {}), (64, dict(tfsf=True)), (65, dict(mat="gold")), (96, dict(mat="both", tfsf=True)),
    (97, dict(pml=0, mat="gold")), (192, dict(mat="lorentz", wide=7)), (193, dict(tfsf=True, wide=8)),
    (449, dict(mat="both", wide=40)), (45001, dict(mat="gold", tfsf=True)),
])
def test_block_step_equals_steps(gpu, precision, n, kw):
    spec = make(n, precision, **kw)
    calls = (2, 3, 31, 33, 64, 17, 90)
    got = result(gpu, spec, calls)
    ref = result(gpu, spec, (1,) * sum(calls))
    assert any(np.any(r) for r in ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_full_stage_is_folded_ring_by_ring(gpu):
    spec = make(100, abi.F64)
    got, ref = result(gpu, spec, (4200,)), result(gpu, spec, (32,) * 131 + (8,))
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_block_step_state_through_a_checkpoint(gpu):
    spec = make(130, abi.F32, tfsf=True, mat="gold")
    outs = []
    for steps in ((5, 40, 7), (1,) * 52):
        J = gpu.Job(spec)
        at = 1
        for i, k in enumerate(steps):
            J.step(at, k)
            at += k
            if at == 6:
                state = J.save_state()
                J.step(6, 3)
                J.load_state(state)
        outs.append([J.get_field(c) for c in (abi.EX, abi.HZ, abi.EX_INC, abi.HZ_INC)] + list(J.get_monitor(0)))
        J.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
