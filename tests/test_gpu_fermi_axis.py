"""Fermi-axis responses against the oracle where the kernel's splits change: one and several warps per
CTA, orbital counts around the warp width and above shared memory's reach, fewer and more Fermi
levels than warps, two components of one and of different curvature planes, and the same components
beside a frequency response in one pass."""
import numpy as np
import pytest

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.model import synthetic_orthogonal_model

pytestmark = pytest.mark.gpu


def rel_err(got, ref):
    scale = np.max(np.abs(ref))
    return np.max(np.abs(got - ref)) / (scale if scale > 0 else 1.0)


@pytest.mark.parametrize("levels", [1, 40])
@pytest.mark.parametrize("nw", [2, 9, 31, 33, 70])
@pytest.mark.parametrize("temperature", [0.0, 300.0])
def test_fermi_axis(oracle_mod, nw, levels, temperature):
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(nw, 1, seed=11 + nw, full_position=True)
    responses = [(_abi.LINEAR_TRANSPORT_BERRY, ["xy", "yz"]), (_abi.BERRY_DIPOLE, ["xyx", "xyz"])]
    if temperature == 0.0:
        responses.append((_abi.INTRINSIC_AHC, ["xy", "zx"]))
    if nw < 33:
        responses.append((_abi.INJECTION_CURRENT, ["xyy"]))
    task = _abi.TaskArrays(responses, fermi_energies=np.linspace(-0.7, 0.8, levels), temperature=temperature,
                           degeneracy_threshold=1e-12, fermi_surface_broadening=0.1,
                           photon_energies=np.linspace(0.1, 2.0, 7), broadening=0.1)
    k = np.random.default_rng(nw).random((5, 3))
    with ResponseEngine(model, task) as eng:
        got = task.split(eng.point_values(k))
        total = task.split(eng.weighted_sum(k, np.full(5, 0.2)))
    ref = oracle_mod.point_values(model, task, k)
    for g, r in zip(got, task.split(ref)):
        assert rel_err(g, r) < 1e-10
    for g, r in zip(total, task.split(ref.mean(axis=0))):
        assert rel_err(g, r) < 1e-10
