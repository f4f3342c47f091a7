"""Rounding error of the complex128 transforms over the stages whose twiddles
are products of looked-up powers (rows of 2^12 and 2^13 with 16 and 32 samples
per thread, columns from 2^10 with 8), against numpy's transform in long
double. Tolerance: each of the log2 N levels rounds once, rms u / sqrt(3) =
0.58 u (u = 2^-53), times 1.5 for the twiddles' own rounding and the products:
0.87 u sqrt(log2 N)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402


def _two(cols, row_e=16, col_e=16):
    return {"levels": 2, "log_rows": cols, "row_e": row_e, "col_e": col_e}


@pytest.mark.parametrize("lg,tuning", [(10, None), (13, None), (16, _two(4)), (17, _two(4)), (16, _two(4, 32)),
                                       (17, _two(4, 32)), (17, _two(10, 16, 8)), (18, _two(11, 16, 8)),
                                       (19, _two(12, 16, 8)), (19, _two(12)), (20, None), (21, None), (22, None)])
def test_error_against_long_double(lg, tuning):
    n = 1 << lg
    p = rsw.Plan(n, "c16", tuning=tuning)
    rng = np.random.default_rng(lg)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    xl = x.astype(np.clongdouble)
    tol = 0.87 * 2.0 ** -53 * np.sqrt(lg)
    for got, ref in ((p.fft, np.fft.fft), (p.ifft, np.fft.ifft)):
        r = ref(xl)
        d = np.abs(got(torch.from_numpy(x).cuda()).cpu().numpy() - r)
        assert float(np.sqrt((d * d).sum() / (np.abs(r) ** 2).sum())) < tol
