"""The samples-per-thread overrides (RSW_ROW_E, RSW_COL_E) over the lengths at
the ends of what the kernels are built for: taken where a kernel exists, the
default elsewhere, and the transforms right in both cases. Tolerances as for
the other transforms (rel-L2 against numpy in FP64: complex128 1e-12,
complex64 2e-6; propagations complex64 5e-6)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200.autotune import plan_tuning  # noqa: E402

FFT = {"c16": 1e-12, "c8": 2e-6}
PROP = {"c16": 1e-12, "c8": 5e-6}
DX, WL, DZ = 2e-9, 2.7e-11, 1e-5


def _check(p, n, dt):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g).to(p.dtype)
    X = torch.fft.fft(x.to(torch.complex128))
    err = lambda a, b: float((a.to(torch.complex128) - b).norm() / b.norm())  # noqa: E731
    assert err(p.fft(x.clone()), X) < FFT[dt]
    assert err(p.ifft(X.to(p.dtype, copy=True)), x.to(torch.complex128)) < FFT[dt]
    f = torch.from_numpy(np.fft.fftfreq(n) / DX).cuda()
    h = torch.polar(torch.ones_like(f), np.pi * WL * DZ * f * f) * np.exp(-2j * np.pi / WL * DZ)
    ref = torch.fft.ifft(X * h)
    assert err(p.propagate(x.clone(), None, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300), ref) < PROP[dt]
    U = torch.empty_like(x)
    assert err(p.propagate(x.clone(), U, dx=DX, wl=WL, dz=DZ, cutoff_freq=1e300), ref) < PROP[dt]
    assert err(U, X * h) < PROP[dt]


# single rows (no 32-per-thread kernel), multi-level rows of 2^7 and 2^8 (none), of 2^9 and more, and
# Bluestein lengths over a single row and over multi-level rows
@pytest.mark.parametrize("dt", ["c16", "c8"])
@pytest.mark.parametrize("n,row_e", [(1 << 8, 16), (1 << 9, 16), (1 << 10, 16), (1 << 11, 16), (1 << 14, 16),
                                     (1 << 18, 32), (1 << 22, 32), (200, 16), (1001, 16), (300001, 32)])
def test_rows_of_32(monkeypatch, dt, n, row_e):
    monkeypatch.setenv("RSW_ROW_E", "32")
    p = rsw.Plan(n, dt)
    assert plan_tuning(p)["row_e"] == row_e
    _check(p, n, dt)


# complex128 columns of 2^12 have no 32-per-thread kernel, shorter and complex64 ones do
@pytest.mark.parametrize("dt,lg,cols,col_e", [("c16", 24, 12, 8), ("c16", 20, 9, 32), ("c8", 26, 12, 32), ("c8", 15, 8, 16)])
def test_columns_of_32(monkeypatch, dt, lg, cols, col_e):
    monkeypatch.setenv("RSW_COL_E", "32")
    monkeypatch.setenv("RSW_SPLIT", str(cols))
    p = rsw.Plan(1 << lg, dt)
    t = plan_tuning(p)
    assert (t["log_rows"], t["col_e"]) == (cols, col_e)
    _check(p, 1 << lg, dt)


# 8 per thread: rows of 2^11 to 2^13 only
@pytest.mark.parametrize("dt,lg,cols,row_e", [("c16", 21, 9, 8), ("c16", 20, 10, 16), ("c8", 25, 11, 32), ("c8", 11, 0, 16)])
def test_rows_of_8(monkeypatch, dt, lg, cols, row_e):
    monkeypatch.setenv("RSW_ROW_E", "8")
    if cols:
        monkeypatch.setenv("RSW_SPLIT", str(cols))
    p = rsw.Plan(1 << lg, dt)
    assert plan_tuning(p)["row_e"] == row_e
    _check(p, 1 << lg, dt)
