"""The autotuner's report where the eigensolver reads neither the team nor the start (FP64, up to 16
orbitals): the plan's own settings, and no times that differ by noise alone."""
import pytest

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.model import synthetic_orthogonal_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [3, 10, 16])
def test_nothing_to_choose(nw):
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(nw, 1, seed=nw, full_position=True)
    task = _abi.TaskArrays([(_abi.BERRY_CURVATURE, ["xy"]), (_abi.QUANTUM_METRIC, ["xx", "yz"])])
    with ResponseEngine(model, task, max_batch=4096) as eng:
        rep = eng.autotune((16, 16, 16), 0, 4096)
    assert rep["eigh_team"] == 32 and rep["warm_start"] == 1
    times = set(rep["eigh_ms"].values()) | set(rep["start_ms"].values())
    assert len(times) == 1 and times.pop() > 0
