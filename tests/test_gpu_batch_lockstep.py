"""Batches run in lockstep (one launch per pass for all sources) at every
level structure and kernel form, the outer columns of 256 threads of
three-level complex128 plans and lengths on both sides of the two-CTA column
kernels among them."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from conftest import rel_l2  # noqa: E402
from rave_sim_b200 import _lib as L  # noqa: E402
from rave_sim_b200 import workloads  # noqa: E402
from rave_sim_b200.engine import Simulation  # noqa: E402


@pytest.mark.parametrize("dtype,lg,split", [("c16", 20, "7,4,9"), ("c16", 20, None), ("c16", 21, None), ("c16", 22, None),
                                            ("c8", 20, "7,4,9"), ("c8", 20, None)])
def test_one_launch_per_pass(monkeypatch, dtype, lg, split):
    if split:
        monkeypatch.setenv("RSW_SPLIT3", split)
    case = workloads.talbot_lau(n=1 << lg, dx=8e-9, dtype=dtype, nr_steps=2, phase_steps=2)
    runs = [{"energy": e, "db_table": workloads.db_table(e), "weight": w} for e, w in ((30000.0, 1.0), (41000.0, 0.5))]
    sim = Simulation(case, dtype=dtype)
    count = L.load().rsw_launch_count
    try:
        a = count()
        for r in runs:
            sim.run_source(energy=r["energy"], db_table=r["db_table"], source=case["source"], weight=r["weight"])
        b = count()
        one = sim.detected()
        sim.reset()
        c = count()
        sim.run_sources(runs, source=case["source"])
        d = count()
        # the sources share every pass; only their chirp tables are built one by one
        assert d - c < 0.75 * (b - a)
        assert rel_l2(sim.detected(), one) < 1e-12
    finally:
        sim.close()
