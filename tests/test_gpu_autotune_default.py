"""The autotuner times the untuned plan's own schedule among its candidates,
at every level structure: a registered result is then never slower than no
tuning by more than the timing's noise."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import rave_sim_b200 as rsw  # noqa: E402
from rave_sim_b200 import autotune  # noqa: E402


@pytest.mark.parametrize("dt,lg", [("c16", 11), ("c16", 13), ("c16", 16), ("c16", 20), ("c16", 24), ("c16", 26), ("c8", 11), ("c8", 14),
                                   ("c8", 16), ("c8", 20), ("c8", 25), ("c8", 26), ("c8", 27)])
def test_default_is_tried(monkeypatch, dt, lg):
    for v in ("RSW_SPLIT", "RSW_SPLIT3", "RSW_ROW_E", "RSW_COL_E"):
        monkeypatch.delenv(v, raising=False)
    p = rsw.Plan(1 << lg, dt)
    default = autotune.plan_tuning(p)
    p.close()
    tried = autotune.tune(1 << lg, dt, reps=1, save=False, register_result=False)["tried"]
    assert default in [t for t, _ in tried]


# the fastest splits by measurement (complex64 outer columns of 2^8 run a
# split step 18 % and 22 % slower at 2^27 and 2^28, complex128 ones of 2^9
# and 2^10 4 % and 9 % slower at 2^26 and 2^27)
@pytest.mark.parametrize("dt,lg,split", [("c8", 27, (9, 4)), ("c8", 28, (10, 4)), ("c16", 26, (8, 5)), ("c16", 27, (8, 6))])
def test_default_three_level_split(monkeypatch, dt, lg, split):
    for v in ("RSW_SPLIT", "RSW_SPLIT3", "RSW_ROW_E", "RSW_COL_E"):
        monkeypatch.delenv(v, raising=False)
    t = autotune.plan_tuning(rsw.Plan(1 << lg, dt))
    assert (t["levels"], t["log_rows"], t["log_mid"]) == (3, *split)
