"""set_propagator on plans whose rows default to 32 samples per thread (the
exact kernel has rows of 16): exact and back, with the Fresnel schedule as it
was; on a plan made from the default's own tuning and beside an RSW_ROW_E that
such rows have no kernel for; in a stream capture. Oracle and tolerance as in
test_gpu_radix32.py."""

import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200 import _lib as L  # noqa: E402
from rave_sim_b200.autotune import plan_tuning  # noqa: E402

N, DX, WL, DZ = 1 << 25, 2e-9, 2.7e-11, 1e-5


def _check(p, exact):
    g = torch.Generator(device="cuda").manual_seed(5)
    u = torch.randn(N, dtype=torch.complex64, device="cuda", generator=g)
    k = torch.arange(N, device="cuda", dtype=torch.float64)
    f = torch.where(k < N // 2, k, k - N) / (N * DX)
    ph = 2 * math.pi * DZ * f * f / (1 / WL + torch.sqrt(1 / WL ** 2 - f * f)) if exact else math.pi * WL * DZ * f * f
    h = torch.polar(torch.ones_like(f), ph) * complex(math.cos(-2 * math.pi / WL * DZ), math.sin(-2 * math.pi / WL * DZ))
    ref = torch.fft.ifft(torch.fft.fft(u.to(torch.complex128)) * h)
    got = p.propagate(u.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert float((got.to(torch.complex128) - ref).norm() / ref.norm()) < 1e-6


def test_exact_and_back():
    p = rsw.Plan(N, "c8")
    before = plan_tuning(p)
    assert before["row_e"] == 32
    _check(p, False)
    for _ in range(2):
        p.set_propagator("exact")
        p.set_propagator("exact")
        _check(p, True)
        p.set_propagator("fresnel")
        assert plan_tuning(p) == before
        _check(p, False)


def test_default_tuning_round_trip():
    p = rsw.Plan(N, "c8", tuning=plan_tuning(rsw.Plan(N, "c8")))
    p.set_propagator("exact")
    _check(p, True)


def test_unavailable_override(monkeypatch):
    monkeypatch.setenv("RSW_ROW_E", "8")  # rows of 2^14 have no such kernel
    p = rsw.Plan(N, "c8")
    p.set_propagator("exact")
    _check(p, True)


def test_counts_asked_for_stay(monkeypatch):
    with pytest.raises(L.RswError):
        rsw.Plan(1 << 20, "c16", tuning={"levels": 2, "log_rows": 8, "row_e": 8}).set_propagator("exact")
    monkeypatch.setenv("RSW_ROW_E", "32")
    with pytest.raises(L.RswError):
        rsw.Plan(N, "c8").set_propagator("exact")


def test_in_a_capture():
    p = rsw.Plan(N, "c8")
    u = torch.ones(N, dtype=torch.complex64, device="cuda")
    p.scale(u, 1.0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.set_propagator("exact")
        p.propagate(u, None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    graph.replay()
    torch.cuda.synchronize()
    # a constant field only takes the constant phase
    want = complex(math.cos(-2 * math.pi / WL * DZ), math.sin(-2 * math.pi / WL * DZ))
    assert float((u - want).abs().max()) < 1e-5
