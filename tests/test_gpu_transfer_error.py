"""Rounding error of the complex128 transfer function in its chirp form: the
spectrum of a propagated unit sample is H itself (the transform of the sample
is exactly 1 everywhere). Against long double, from 2^14 (the shortest default
lengths in chirp form) up. Tolerance: three factors (thread, register, table),
each rounded once, and their two products, rms at most 0.6 u apiece (u =
2^-53): sqrt(5) 0.6 u = 1.34 u, a quarter on top for sincospi's own error."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402

DX, WL, DZ = 2e-9, 2.7e-11, 1e-4


@pytest.mark.parametrize("lg", [14, 15, 16, 18, 19, 20])
def test_chirp_form(lg):
    n = 1 << lg
    p = rsw.Plan(n, "c16")
    assert p.info()["log_rows"] > 0
    u = torch.zeros(n, dtype=torch.complex128, device="cuda")
    u[0] = 1
    U = torch.empty_like(u)
    p.propagate(u, U, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300)
    ld = np.longdouble
    ks = np.fft.fftfreq(n, 1.0 / n).astype(ld)
    f = ks / (ld(n) * ld(DX))
    th = ld((math.pi * WL) * DZ) * f * f
    phi = ((-2 * math.pi) / WL) * DZ
    ref = (np.cos(th) + 1j * np.sin(th)) * np.clongdouble(complex(math.cos(phi), math.sin(phi)))
    d = np.abs(U.cpu().numpy() - ref)
    assert float(np.sqrt((d * d).mean())) < 1.25 * math.sqrt(5) * 0.6 * 2.0 ** -53
