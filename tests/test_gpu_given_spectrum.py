"""propagate from a given spectrum where a CTA of the row pass takes several
rows (more rows than resident CTAs), two and three levels: the row's chirp
factors, which some of its warps fill, meet the samples without a transform
in between. Oracle: torch's FP64 transform; tolerances as for the other
propagations (rel-L2 complex128 1e-12, complex64 1e-6 times the three
roundings of spectrum, product and transform: 3e-6)."""

import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402

TOL = {"c16": 1e-12, "c8": 3e-6}
DX, WL, DZ = 2e-9, 2.7e-11, 1e-5


@pytest.mark.parametrize("dt", ["c16", "c8"])
# two levels: default and short rows (128 to 2^12 samples); three levels
@pytest.mark.parametrize("lg,split", [(22, None), (22, "RSW_SPLIT=11"), (18, "RSW_SPLIT=11"), (22, "RSW_SPLIT3=5,6,11")])
def test_skip_fft(monkeypatch, dt, lg, split):
    n = 1 << lg
    if split:
        monkeypatch.setenv(*split.split("="))
    p = rsw.Plan(n, dt)
    g = torch.Generator(device="cuda").manual_seed(lg)
    U = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g).to(p.dtype)
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    f = torch.where(k < n // 2, k, k - n) / (n * DX)
    h = torch.polar(torch.ones_like(f), math.pi * WL * DZ * f * f)
    h = h * complex(math.cos(-2 * math.pi / WL * DZ), math.sin(-2 * math.pi / WL * DZ))
    ref = U.to(torch.complex128) * h
    err = lambda a, b: float((a.to(torch.complex128) - b).norm() / b.norm())  # noqa: E731
    for _ in range(3):  # a field left from before must not matter
        u, V = torch.full_like(U, float("nan")), U.clone()
        p.propagate(u, V, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300, skip_fft=True)
        assert err(V, ref) < TOL[dt]
        assert err(u, torch.fft.ifft(ref)) < TOL[dt]
