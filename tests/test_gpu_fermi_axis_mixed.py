"""Fermi-axis responses on the mixed path, whose passes without a frequency component are kernels of
their own, beside one with a frequency component; and models of one orbital on both paths."""
import numpy as np
import pytest

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.model import synthetic_orthogonal_model

pytestmark = pytest.mark.gpu


def compare(oracle_mod, model, task, k, tol):
    from wanniernlqg_b200.engine import ResponseEngine
    with ResponseEngine(model, task) as eng:
        got = task.split(eng.point_values(k))
        total = task.split(eng.weighted_sum(k, np.full(len(k), 1.0 / len(k))))
    ref = oracle_mod.point_values(model, task, k)
    for g, r in list(zip(got, task.split(ref))) + list(zip(total, task.split(ref.mean(axis=0)))):
        assert np.max(np.abs(g - r)) <= tol * max(np.max(np.abs(r)), 1e-300)


def responses(temperature, with_frequency):
    out = [(_abi.LINEAR_TRANSPORT_BERRY, ["xy", "yz"]), (_abi.BERRY_DIPOLE, ["xyx", "xyz"])]
    if temperature == 0.0:
        out.append((_abi.INTRINSIC_AHC, ["xy", "zx"]))
    if with_frequency:
        out.append((_abi.INJECTION_CURRENT, ["xyy"]))
    return out


@pytest.mark.parametrize("levels", [1, 40])
@pytest.mark.parametrize("nw,with_frequency", [(2, False), (2, True), (9, False), (9, True), (31, False), (31, True),
                                               (70, False)])
@pytest.mark.parametrize("temperature", [0.0, 300.0])
def test_mixed(oracle_mod, nw, levels, temperature, with_frequency):
    """The mixed path's response arithmetic is FP32: 1e-4, as its other comparisons with the oracle."""
    model = synthetic_orthogonal_model(nw, 1, seed=11 + nw, full_position=True)
    task = _abi.TaskArrays(responses(temperature, with_frequency), fermi_energies=np.linspace(-0.7, 0.8, levels),
                           temperature=temperature, degeneracy_threshold=1e-12, fermi_surface_broadening=0.1,
                           photon_energies=np.linspace(0.1, 2.0, 7), broadening=0.1, precision=_abi.PRECISION_MIXED)
    compare(oracle_mod, model, task, np.random.default_rng(nw).random((5, 3)), 1e-4)


@pytest.mark.parametrize("precision,tol", [(_abi.PRECISION_FP64, 1e-10), (_abi.PRECISION_MIXED, 1e-4)])
@pytest.mark.parametrize("temperature", [0.0, 300.0])
@pytest.mark.parametrize("levels", [1, 3, 70])
def test_one_orbital(oracle_mod, levels, temperature, precision, tol):
    model = synthetic_orthogonal_model(1, 1, seed=3, full_position=True)
    task = _abi.TaskArrays(responses(temperature, False), fermi_energies=np.linspace(-0.7, 0.8, levels),
                           temperature=temperature, degeneracy_threshold=1e-12, fermi_surface_broadening=0.1,
                           precision=precision)
    compare(oracle_mod, model, task, np.random.default_rng(1).random((3, 3)), tol)
