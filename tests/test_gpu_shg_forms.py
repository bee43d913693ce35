"""The second-harmonic kernel's forms (one or two CTAs per SM, a global working set) at the edges of the
rule that picks them: orbital counts on both sides of shared memory's reach, components and energies on
both sides of a pass, rounds of points that fill the SMs and that do not."""
import time

import numpy as np
import pytest

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.model import synthetic_orthogonal_model

pytestmark = pytest.mark.gpu

COMPONENTS = ["xxx", "xyz", "zzz", "xyy"]


def make_task(components, energies, kernel=_abi.LORENTZIAN, temperature=0.0):
    return _abi.TaskArrays([(_abi.SECOND_HARMONIC, components)], broadening_type=kernel, broadening=0.05,
                           photon_energies=np.linspace(0.1, 3.0, energies), temperature=temperature)


def by_quantity(task, components, values):
    return values.reshape(values.shape[:-1] + (2, 7, components, -1))


def close(got, ref, tol):
    """Per quantity and term, against the largest of its values."""
    scale = np.max(np.abs(ref), axis=(-1, -2), keepdims=True)
    assert np.all(np.abs(got - ref) <= tol * np.maximum(scale, 1e-300))


@pytest.mark.parametrize("nw", [3, 12, 22, 23, 30, 37])
@pytest.mark.parametrize("components,energies", [(1, 7), (3, 256), (4, 300)])
def test_against_the_oracle(oracle_mod, nw, components, energies):
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(nw, 1, seed=nw, full_position=True)
    task = make_task(COMPONENTS[:components], energies, temperature=300.0 if nw == 12 else 0.0)
    k = np.random.default_rng(nw).random((2, 3))
    ref = oracle_mod.point_values(model, task, k)
    with ResponseEngine(model, task) as eng:
        got = eng.point_values(k)
        total = eng.weighted_sum(k, np.full(2, 0.5))
    for g, r in ((got, ref), (total[None], ref.mean(axis=0)[None])):
        for a, b in zip(g, r):
            close(by_quantity(task, components, a), by_quantity(task, components, b), 1e-9)


@pytest.mark.parametrize("nw", [4, 12, 16, 22])
@pytest.mark.parametrize("components,energies", [(1, 48), (2, 256), (3, 256), (4, 100)])
@pytest.mark.parametrize("kernel", [_abi.LORENTZIAN, _abi.GAUSSIAN])
def test_forms_agree(nw, components, energies, kernel):
    """Batches of 148 points take one CTA per SM; 297 to 1200 points take either form by the rule."""
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(nw, 1, seed=nw, full_position=True)
    task = make_task(COMPONENTS[:components], energies, kernel)
    k = np.random.default_rng(nw).random((1200, 3))
    with ResponseEngine(model, task, max_batch=100) as eng:
        ref = eng.point_values(k)
    with ResponseEngine(model, task, max_batch=1200) as eng:
        for n in (1, 149, 296, 297, 600, 1200):
            total = eng.weighted_sum(k[:n], np.full(n, 1.0 / n))
            close(by_quantity(task, components, total), by_quantity(task, components, ref[:n].mean(axis=0)), 1e-10)
        # The two forms share every step but the order in which a thread meets its components.
        got = eng.point_values(k)
    assert np.max(np.abs(got - ref)) <= 1e-13 * np.max(np.abs(ref))


def test_a_third_component_shares_the_resonances():
    """26 orbitals, 256 energies, Gaussian: three components in one pass of the threads cost about 1.4 times
    one; evaluating the exponentials in a second pass made it 2."""
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(26, 1, seed=5, full_position=True)
    k = np.random.default_rng(1).random((592, 3))
    best = []
    for components in (1, 3):
        with ResponseEngine(model, make_task(COMPONENTS[:components], 256, _abi.GAUSSIAN)) as eng:
            times = []
            for _ in range(7):
                t = time.perf_counter()
                eng.weighted_sum(k, np.ones(592))
                times.append(time.perf_counter() - t)
        best.append(min(times))
    assert best[1] <= 1.7 * best[0]
