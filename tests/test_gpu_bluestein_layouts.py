"""The chirp spectrum of Bluestein plans in the layout of their inner plan:
complex64 inner plans whose level structure complex128 has too, and rows of
2^14, which it has not (the spectrum then goes through natural order). Oracle
and tolerance as in test_gpu_bluestein.py (complex64 5e-6)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200 import autotune  # noqa: E402


@pytest.mark.parametrize("tuning", [
    {"levels": 2, "log_rows": 4, "row_e": 16}, {"levels": 2, "log_rows": 4, "row_e": 32},
    {"levels": 2, "log_rows": 9, "row_e": 16, "col_e": 8}, {"levels": 2, "log_rows": 9, "row_e": 32, "col_e": 32},
    {"levels": 3, "log_rows": 4, "log_mid": 4, "row_e": 16}])
def test_inner_layouts(tuning):
    n, m = 100003, 1 << 18
    autotune.register(m, "c8", tuning)
    try:
        p = rsw.Plan(n, "c8")
    finally:
        autotune.register(m, "c8", None)
    t = autotune.plan_tuning(p)
    assert all(t[k] == v for k, v in tuning.items())
    rng = np.random.default_rng(4)
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    X = p.fft(torch.from_numpy(x).cuda())
    assert rel_l2(X.cpu().numpy(), np.fft.fft(x.astype(np.complex128))) < 5e-6
    assert rel_l2(p.ifft(X).cpu().numpy(), x) < 5e-6
