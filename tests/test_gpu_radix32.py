"""Radix-32 kernels (32 samples per thread): propagation over every row and
column length they are built for, remainders of one to five bits, against an
FP64 torch transform; and the exact propagator on a plan whose rows default to
them. Tolerances (rel-L2): complex128 1e-13 times the phase's rounding (the
phase is below 1e2 rad), so 1e-12; complex64 1e-6 (about 2.5e-7 measured for
the radix-16 kernels at these lengths)."""

import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200.autotune import plan_tuning  # noqa: E402

DX, WL, DZ = 2e-9, 2.7e-11, 1e-5


def _reference(u, exact=False):
    n = u.numel()
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    f = torch.where(k < n // 2, k, k - n) / (n * DX)
    ph = math.pi * WL * DZ * f * f
    if exact:
        ph = 2 * math.pi * DZ * f * f / (1 / WL + torch.sqrt(1 / WL ** 2 - f * f))
    h = torch.polar(torch.ones_like(f), ph) * complex(math.cos(-2 * math.pi / WL * DZ), math.sin(-2 * math.pi / WL * DZ))
    return torch.fft.ifft(torch.fft.fft(u.to(torch.complex128)) * h)


def _rel(a, b):
    return float((a.to(torch.complex128) - b).norm() / b.norm())


def _field(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, dtype=torch.complex128, device="cuda", generator=g).to(dtype)


@pytest.mark.parametrize("dt,rows,cols", [("c8", 9, 9), ("c8", 10, 10), ("c8", 11, 11), ("c8", 12, 9), ("c8", 13, 10),
                                          ("c8", 14, 9), ("c16", 9, 9), ("c16", 10, 10), ("c16", 11, 11),
                                          ("c16", 12, 9), ("c16", 13, 9)])
def test_propagate(dt, rows, cols):
    n = 1 << (rows + cols)
    p = rsw.Plan(n, dt, tuning={"levels": 2, "log_rows": cols, "row_e": 32, "col_e": 32})
    u = _field(n, p.dtype, rows)
    ref = _reference(u)
    got = p.propagate(u.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert _rel(got, ref) < (1e-12 if dt == "c16" else 1e-6)
    U = torch.empty_like(u)
    got = p.propagate(u.clone(), U, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert _rel(got, ref) < (1e-12 if dt == "c16" else 1e-6)
    assert _rel(U, torch.fft.fft(ref)) < (1e-12 if dt == "c16" else 1e-6)


def test_exact_propagator_on_default_rows():
    n = 1 << 25
    p = rsw.Plan(n, "c8")
    assert plan_tuning(p)["row_e"] == 32
    u = _field(n, p.dtype, 1)
    got = p.propagate(u.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert _rel(got, _reference(u)) < 1e-6
    p.set_propagator("exact")
    got = p.propagate(u.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    assert _rel(got, _reference(u, exact=True)) < 1e-6
