"""Bluestein plans over every form of the power-of-two passes under them: one,
two and three levels, and rows whose kernel has no table product (8 samples
per thread by a registered tuning). propagate with a spectrum buffer, without
and from a given spectrum, against numpy in FP64; tolerances as in
test_gpu_bluestein.py (complex128 1e-12, complex64 5e-6)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200 import autotune  # noqa: E402

TOL = {"c16": 1e-12, "c8": 5e-6}
FORMS = {"single": (1001, None), "two": (40001, None), "three": (40001, "RSW_SPLIT3=4,4,9"), "rows_of_8": (100003, 8)}


@pytest.mark.parametrize("dt", ["c16", "c8"])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_propagate_over_every_schedule(monkeypatch, dt, form):
    n, how = FORMS[form]
    m = 1 << (2 * n - 2).bit_length()
    if isinstance(how, str):
        monkeypatch.setenv(*how.split("="))
    if how == 8:
        autotune.register(m, dt, {"levels": 2, "log_rows": 7, "row_e": 8, "col_e": 16})
    try:
        p = rsw.Plan(n, dt)
    finally:
        autotune.register(m, dt, None)
    t = autotune.plan_tuning(p)
    assert t["levels"] == {"single": 1, "three": 3}.get(form, 2) and (how != 8 or t["row_e"] == 8)
    rng = np.random.default_rng(n)
    u = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if dt == "c8":
        u = u.astype(np.complex64).astype(np.complex128)
    dx, wl, dz, cut = 2e-9, 2.7e-11, 1e-3, 1.1e8
    f = np.fft.fftfreq(n) / dx
    H = np.exp(1j * ((np.pi * wl) * dz) * f * f) * np.exp(1j * ((-2 * np.pi) / wl) * dz)
    H[int(np.ceil(n * (cut * dx))):n - int(np.ceil(n * (cut * dx))) + 1] = 0
    U = np.fft.fft(u)
    ref = np.fft.ifft(U * H)
    ud = torch.from_numpy(u).cuda().to(p.dtype)
    assert rel_l2(p.fft(ud.clone()).cpu().numpy(), U) < TOL[dt]
    given = torch.from_numpy(U).cuda().to(p.dtype)
    for Ud, skip in ((None, False), (torch.empty_like(ud), False), (given, True)):
        v = ud.clone()
        p.propagate(v, Ud, dx=dx, wl=wl, dz=dz, cutoff_freq=cut, skip_fft=skip)
        assert rel_l2(v.cpu().numpy(), ref) < TOL[dt]
        if Ud is not None:
            assert rel_l2(Ud.cpu().numpy(), U * H) < TOL[dt]
