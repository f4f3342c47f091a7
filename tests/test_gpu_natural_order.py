"""Natural-order transforms over the level structures whose reordering runs
through shared-memory tiles (from 2^18 samples; gathers below): column
levels of 16, 32, 64 and more, short and long rows, a middle level. Oracle: numpy's FP64 transform;
tolerances as for the other transforms (rel-L2: complex128 1e-12, complex64
2e-6). The transforms of a unit sample at an odd place pin every index."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402

TOL = {"c16": 1e-12, "c8": 2e-6}


@pytest.mark.parametrize("dt", ["c16", "c8"])
@pytest.mark.parametrize("lg,split", [(11, (4,)), (17, (6,)), (18, (5,)), (18, (6,)), (18, (11,)), (19, (7,)),
                                      (18, (4, 4)), (18, (5, 4)), (20, (7, 6))])
def test_natural_order(monkeypatch, dt, lg, split):
    n = 1 << lg
    if len(split) == 1:
        monkeypatch.setenv("RSW_SPLIT", str(split[0]))
    else:
        monkeypatch.setenv("RSW_SPLIT3", "%d,%d,%d" % (*split, lg - sum(split)))
    p = rsw.Plan(n, dt)
    assert p.info()["log_rows"] == split[0]
    rng = np.random.default_rng(lg)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    xd = torch.from_numpy(x).to("cuda").to(p.dtype)
    x = xd.cpu().numpy().astype(np.complex128)
    X = p.fft(xd, torch.empty_like(xd))
    assert rel_l2(X.cpu().numpy(), np.fft.fft(x)) < TOL[dt]
    assert rel_l2(p.ifft(X, torch.empty_like(X)).cpu().numpy(), x) < TOL[dt]
    e = torch.zeros_like(xd)
    e[n // 3] = 1
    k = np.arange(n, dtype=np.int64) * (n // 3) % n
    assert np.abs(p.fft(e).cpu().numpy() - np.exp(-2j * np.pi * k / n)).max() < 10 * TOL[dt]
