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


@pytest.mark.parametrize("dt,lg", [("c16", 11), ("c16", 16), ("c16", 20), ("c16", 24), ("c16", 26), ("c8", 11),
                                   ("c8", 16), ("c8", 20), ("c8", 25), ("c8", 26), ("c8", 27)])
def test_default_is_tried(monkeypatch, dt, lg):
    for v in ("RSW_SPLIT", "RSW_SPLIT3", "RSW_ROW_E", "RSW_COL_E"):
        monkeypatch.delenv(v, raising=False)
    p = rsw.Plan(1 << lg, dt)
    default = autotune.plan_tuning(p)
    p.close()
    tried = autotune.tune(1 << lg, dt, reps=1, save=False, register_result=False)["tried"]
    assert default in [t for t, _ in tried]
