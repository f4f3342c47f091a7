"""Fields that one row could hold but that run as two short levels by default
(complex128 2^12 and 2^13, complex64 to 2^14): the transfer function per
sample with the reference's own roundings, propagate without state in the
plan (several streams, a first call under capture), lockstep batches.

Tolerances: complex128 against the oracle's FP64 propagation, two transforms
on either side at 0.87 u sqrt(log2 N) each (u = 2^-53) and the product:
2 x 4.9e-16 and 2.2e-16, so 1.2e-15; complex64 1e-6 as in test_gpu_radix32.py."""

import numpy as np
import pytest

from conftest import rel_l2
from oracle import bigwave_np as bw

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200 import _lib as L  # noqa: E402
from rave_sim_b200 import workloads  # noqa: E402
from rave_sim_b200.autotune import plan_tuning  # noqa: E402
from rave_sim_b200.engine import Simulation  # noqa: E402

CASES = [("c16", 12), ("c16", 13), ("c8", 12), ("c8", 13), ("c8", 14)]
TOL = {"c16": 1.2e-15, "c8": 1e-6}
DX, WL, DZ = 2e-9, 2.7e-11, 1e-4


def _field(n, dt, seed):
    rng = np.random.default_rng(seed)
    u = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return u if dt == "c16" else u.astype(np.complex64).astype(np.complex128)


@pytest.mark.parametrize("dt,lg", CASES)
@pytest.mark.parametrize("cut", [1e300, 1.1e8])
def test_reference_rounding(dt, lg, cut):
    n = 1 << lg
    sim = bw.Sim(N=n, dx=DX, z_detector=1, detector_size=1e-6, psx=1e-7, psy=1, wl=WL, chunk_size=n)
    u = _field(n, dt, lg)
    U0 = np.fft.fft(u)
    ref, Uref = bw.propagate(u, U0, sim, DZ, cut)
    p = rsw.Plan(n, dt)
    assert p.info()["log_rows"] > 0
    d = torch.from_numpy(u).cuda().to(p.dtype)
    args = dict(dx=DX, wl=WL, dz=DZ, cutoff_freq=cut)
    assert rel_l2(p.propagate(d.clone(), None, **args).cpu().numpy(), ref) < TOL[dt]
    v, U = d.clone(), torch.empty_like(d)
    p.propagate(v, U, **args)
    assert rel_l2(v.cpu().numpy(), ref) < TOL[dt] and rel_l2(U.cpu().numpy(), Uref) < TOL[dt]
    v, U = torch.full_like(d, float("nan")), torch.from_numpy(U0).cuda().to(p.dtype)
    p.propagate(v, U, skip_fft=True, **args)
    assert rel_l2(v.cpu().numpy(), ref) < TOL[dt] and rel_l2(U.cpu().numpy(), Uref) < TOL[dt]


@pytest.mark.parametrize("dt,lg", CASES)
def test_two_streams_share_a_plan(dt, lg):
    p = rsw.Plan(1 << lg, dt)
    d = torch.from_numpy(_field(1 << lg, dt, 1)).cuda().to(p.dtype)
    fields, streams = [d.clone(), d.clone()], [torch.cuda.Stream(), torch.cuda.Stream()]
    want = [d.clone(), d.clone()]
    for _ in range(40):
        for k in range(2):
            p.propagate(want[k], None, dx=DX, wl=WL, dz=DZ * (k + 1), cutoff_freq=1e300)
    torch.cuda.synchronize()
    for _ in range(40):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                p.propagate(fields[k], None, dx=DX, wl=WL, dz=DZ * (k + 1), cutoff_freq=1e300)
    torch.cuda.synchronize()
    assert torch.equal(fields[0], want[0]) and torch.equal(fields[1], want[1])


@pytest.mark.parametrize("dt,lg", CASES)
def test_first_call_under_capture(dt, lg):
    p, q = rsw.Plan(1 << lg, dt), rsw.Plan(1 << lg, dt)
    d = torch.from_numpy(_field(1 << lg, dt, 2)).cuda().to(p.dtype)
    want = q.propagate(d.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    u = d.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.propagate(u, None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(u, want)


@pytest.mark.parametrize("dt,lg", CASES)
def test_tuning_round_trip(dt, lg):
    p = rsw.Plan(1 << lg, dt)
    q = rsw.Plan(1 << lg, dt, tuning=plan_tuning(p))
    assert plan_tuning(q) == plan_tuning(p)
    d = torch.from_numpy(_field(1 << lg, dt, 3)).cuda().to(p.dtype)
    a = p.propagate(d.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert torch.equal(a, q.propagate(d.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300))


@pytest.mark.parametrize("dt,lg", CASES)
@pytest.mark.parametrize("count", [2, 9])
def test_batches(dt, lg, count):
    n, dx = 1 << lg, 100e-9
    case = workloads.talbot_lau(n=n, dx=dx, dtype=dt, nr_steps=2, phase_steps=2)
    case["sim_params"].update(detector_size=0.5 * n * dx, detector_pixel_size_x=n * dx / 64)
    energies = [30000.0 + 4000.0 * k for k in range(count)]
    # a cutoff that is active for the lower energies only
    ang = float(np.arcsin(workloads.wavelength_from_energy(sum(energies) / count) / (2 * dx)))
    sim = Simulation(case, dtype=dt, cutoff_angles=[ang] * (len(case["elements"]) + 1))
    runs = [{"energy": e, "db_table": workloads.db_table(e), "weight": 1.0 / (k + 1)} for k, e in enumerate(energies)]
    launches = L.load().rsw_launch_count
    try:
        a = launches()
        for r in runs:
            sim.run_source(energy=r["energy"], db_table=r["db_table"], source=case["source"], weight=r["weight"])
        b = launches()
        one = sim.detected()
        sim.reset()
        c = launches()
        sim.run_sources(runs, source=case["source"])
        # the sources share every pass; only their transfer functions are built one by one
        assert launches() - c < 0.75 * (b - a)
        assert np.abs(one).max() > 0 and rel_l2(sim.detected(), one) < 1e-12
    finally:
        sim.close()
