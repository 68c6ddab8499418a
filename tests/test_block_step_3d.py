"""The 3D block-step kernel (two steps of a tile per launch, FP32) against the
half-step kernels, bit for bit, where its tiles end: grids a cell short of, at
and past a tile's 60 columns and 13 rows, every PML face on its own and
together, periodic axes shorter than a tile, materials (dispersive cells on the
seams), sources, and samples after either step."""
import numpy as np
import pytest

from fdtd_gpu import abi, problems
from fdtd_gpu.spec import JobSpec, box, spheres

pytestmark = pytest.mark.gpu

BLOCK = 10  # the tile number of the 3D block-step kernel


@pytest.fixture(scope="module")
def gpu():
    from fdtd_gpu import build, job
    build.build()
    if job.device_count() < 1:
        pytest.skip("no sm_103a device")
    return job


GRAPHENE = dict(fermi_ev=0.4, tau=0.1e-12, temperature=300.0, chi3=1e-18, raman_frac=0.3, raman_freq=47.4e12,
                raman_tau=1e-12, thickness=2e-9, e_scale=1.0)


def make(n, per=(0, 0, 0), pml=4, mat=None, sub=False, mean=False):
    ds = 1e-9
    lo = [0 if q else pml for q in per]
    hi = [n[a] - 1 - lo[a] for a in range(3)]
    spec = JobSpec(layout=abi.LAYOUT_3D, n=n, ku=0.5, dt=0.5 * ds / problems.C0, ds=ds, precision=abi.F32, periodic=per,
                   main_lo=tuple(lo), main_hi=tuple(hi))
    spec.add_dielectric(box((0, 0, 0), tuple(x - 1 for x in n)), 1.0)
    if sub:
        spec.add_dielectric(box((lo[0], lo[1], n[2] // 2), tuple(hi)), 2.25)
    ball = spheres([(n[0] / 2, n[1] / 2, n[2] / 2, min(n) / 4)])
    if mat in ("gold", "both"):
        spec.add_gold(ball, problems.GOLD_CONFIG)
    if mat in ("lorentz", "both"):
        spec.add_lorentz(box((lo[0] + 1, lo[1] + 1, lo[2] + 1), (lo[0] + 4, lo[1] + 3, lo[2] + 5)), problems.GOLD_JP)
    if mat == "graphene":
        spec.add_graphene(box((0, 0, n[2] // 2), (n[0] - 1, n[1] - 1, n[2] // 2)), GRAPHENE)
    if pml and not all(per):
        spec.pml = dict(mode=abi.PML_SPLIT, npml=tuple((0, 0) if q else (pml, pml) for q in per), eps_lo=1.0,
                        sigma_max=problems.pml_sigma_max(3.0, np.exp(-16.0), pml, ds), order=3.0)
    p = dict(t0=1e-16, st=2e-16, w0=3e15)
    spec.sources.append(dict(component=abi.EX, lo=(0, 0, lo[2] + 3), hi=(n[0] - 1, n[1] - 1, lo[2] + 3), amp=1.0, **p))
    spec.sources.append(dict(component=abi.EZ, lo=(n[0] // 2 - 3, 0, n[2] // 2 - 2), hi=(n[0] // 2 + 2, n[1] - 1, n[2] // 2 + 1),
                             amp=0.7, **p))
    om = problems.dft_omegas(500e-9, 800e-9, 3)
    spec.add_monitor((0, 0, n[2] // 2 + 1), (n[0] - 1, n[1] - 1, n[2] // 2 + 1), (abi.EX, abi.EY, abi.HX, abi.HY), om, mean=mean)
    spec.add_monitor((n[0] // 2, 0, 0), (n[0] // 2, n[1] - 1, n[2] - 1), (abi.EZ, abi.HZ), om)
    spec.add_probe((n[0] // 2 + 1, n[1] // 2, n[2] // 2), (abi.EX, abi.EZ, abi.HY))
    return spec


def start(spec):
    x = np.zeros(spec.n[::-1])
    lo, hi = spec.main_lo, spec.main_hi
    part = tuple(slice(lo[a], hi[a] + 1) for a in (2, 1, 0))
    x[part] = np.random.default_rng(5).standard_normal(x[part].shape)
    return x


def state(J, spec):
    out = [J.get_field(c) for c in range(6)]
    for q in range(len(spec.monitors)):
        out += list(J.get_monitor(q))
    return out + [J.get_probe(0)]


def result(gpu, spec, calls, tile=0):
    J = gpu.Job(spec, tile=tile)
    J.set_field(abi.EX, start(spec))
    at = 1
    for k in calls:
        J.step(at, k)
        at += k
    out, used = state(J, spec), J.tile()
    J.close()
    return used, out


@pytest.mark.parametrize("n,kw", [
    ((60, 13, 20), dict(pml=0)), ((56, 12, 9), dict(pml=0, sub=True)), ((64, 14, 33), {}),
    ((120, 26, 24), dict(mat="gold")), ((124, 27, 40), dict(mat="both", sub=True, mean=True)),
    ((180, 39, 21), dict(per=(0, 1, 1))), ((64, 40, 30), dict(per=(1, 0, 1), mat="gold")),
    ((68, 30, 50), dict(per=(1, 1, 0), mat="lorentz")), ((8, 8, 64), dict(per=(1, 1, 0), mat="graphene", mean=True)),
    ((48, 40, 2), dict(per=(1, 1, 1))), ((72, 72, 72), dict(pml=8, mat="gold", sub=True)),
])
def test_block_step_equals_half_steps(gpu, monkeypatch, n, kw):
    if n[2] == 2:  # two planes: no room for the ball and the sheet of sources
        spec = make((n[0], n[1], 8), **kw)
        spec.n, spec.main_hi = n, (n[0] - 1, n[1] - 1, 1)
        spec.sources, spec.monitors, spec.probes = [], [], []
        spec.add_monitor((0, 0, 1), (n[0] - 1, n[1] - 1, 1), (abi.EX, abi.HZ), problems.dft_omegas(500e-9, 800e-9, 3))
        spec.add_probe((5, 5, 0), (abi.EX,))
    else:
        spec = make(n, **kw)
    calls = (1, 2, 3, 7, 64, 20, 33)
    monkeypatch.setenv("FDTD_TUNE", "block")
    used, got = result(gpu, spec, calls)
    assert used == BLOCK
    split, ref = result(gpu, spec, (sum(calls),), tile=2)
    assert split == 2 and any(np.any(r) for r in ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_block_step_state_through_every_entry_point(gpu, monkeypatch):
    """A field written, a checkpoint, the per-procedure step and the count of
    non-finite values, after odd and even numbers of launches."""
    spec = make((80, 30, 28), mat="gold")
    outs = []
    for tile in (0, 2):
        monkeypatch.setenv("FDTD_TUNE", "block")
        J = gpu.Job(spec, tile=tile)
        assert J.tile() == (tile or BLOCK)
        J.step(1, 3)
        J.set_field(abi.HX, J.get_field(abi.HX) + 0.25)
        J.step(4, 1)
        saved = J.save_state()
        J.step(5, 8)
        J.load_state(saved)
        J.step(5, 2)
        J.step_procedures(7)
        J.step(8, 5)
        assert J.count_nonfinite() == 0
        outs.append(state(J, spec))
        J.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
