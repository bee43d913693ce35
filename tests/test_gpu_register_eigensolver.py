"""The FP64 path's eigensolvers at their edges: every padded order up to 32 (odd counts, one orbital, the
largest order of each group width, the register kernel up to 16 and the one-sided stage from 17), the
CTA form's column blocks and rows per lane above 32, fewer and more points than the groups of a warp
and of the grid, and exactly degenerate levels, against LAPACK's energies and the eigenvector
residual."""
import numpy as np
import pytest

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.model import TightBindingModel, kramers_doubled_model, synthetic_orthogonal_model

pytestmark = pytest.mark.gpu


def bloch(model, k):
    ph = np.exp(2j * np.pi * (model.r_vectors.T @ k)) / model.r_degeneracies
    return np.einsum("ijr,r->ij", model.hamiltonian_r, ph)


def check(model, k, vectors_for):
    from wanniernlqg_b200.engine import ResponseEngine
    task = _abi.TaskArrays([(_abi.QUANTUM_METRIC, ["xx"])])
    with ResponseEngine(model, task, max_batch=max(64, len(k))) as eng:
        e, u = eng.spectrum(k)
    for i in vectors_for:
        h = bloch(model, k[i])
        scale = np.linalg.norm(h)
        assert np.max(np.abs(e[i] - np.linalg.eigvalsh(h))) <= 1e-13 * scale
        assert np.max(np.abs(h @ u[i] - u[i] * e[i])) <= 1e-12 * scale
        assert np.max(np.abs(u[i].conj().T @ u[i] - np.eye(model.num_orbitals))) < 1e-12
        pivot = np.argmax(np.abs(u[i]), axis=0)
        top = u[i][pivot, np.arange(model.num_orbitals)]
        assert np.max(np.abs(top.imag)) < 1e-12 and np.min(top.real) > 0


@pytest.mark.parametrize("nw", [1, 2, 3, 4, 5, 7, 8, 9, 11, 13, 16, 17, 19, 22, 23, 26, 28, 29, 31, 32,
                                33, 36, 37, 40, 41, 48, 63, 64, 65, 72, 95, 96, 97, 112, 128])
def test_every_order(nw):
    model = synthetic_orthogonal_model(nw, 1, seed=100 + nw, full_position=True)
    check(model, np.random.default_rng(nw).random((7, 3)), range(7))


@pytest.mark.parametrize("nw", [4, 6, 16, 20])
@pytest.mark.parametrize("points", [1, 3, 33, 5003])
def test_point_counts(nw, points):
    model = synthetic_orthogonal_model(nw, 1, seed=7 + nw)
    check(model, np.random.default_rng(points).random((points, 3)), {0, points // 2, points - 1})


@pytest.mark.parametrize("nw", [6, 14, 24, 50])
def test_degenerate_levels(nw):
    base = synthetic_orthogonal_model(nw // 2, 1, seed=3, full_position=True)
    check(kramers_doubled_model(base, 0.0), np.random.default_rng(5).random((6, 3)), range(6))


@pytest.mark.parametrize("nw", [5, 21, 39])
@pytest.mark.parametrize("scale", [0.0, 1.0, 1e-9])
def test_diagonal_and_zero_matrices(nw, scale):
    ham = np.zeros((nw, nw, 1), dtype=complex, order="F")
    one = TightBindingModel(np.eye(3), np.zeros((3, 1), int), np.ones(1, int), ham, np.zeros((nw, nw, 3, 1), complex))
    one.hamiltonian_r[:, :, 0] = scale * np.diag(np.r_[3.0, -1.0, 2.0, 2.0, 0.5, np.linspace(-3.0, 1.0, nw - 5)])
    check(one, np.zeros((2, 3)), range(2))


@pytest.mark.parametrize("nw,points", [(3, 5), (13, 2001), (33, 801)])
def test_row_and_column_major_vectors(nw, points):
    """The row-major spectrum (device transposition, pinned chunks: none, several with a remainder, a
    batch boundary inside) is the column-major one transposed, bit for bit."""
    import ctypes
    from wanniernlqg_b200.engine import ResponseEngine
    model = synthetic_orthogonal_model(nw, 1, seed=nw)
    k = np.random.default_rng(nw).random((points, 3))
    dp = ctypes.POINTER(ctypes.c_double)
    with ResponseEngine(model, _abi.TaskArrays([(_abi.QUANTUM_METRIC, ["xx"])]), max_batch=700) as eng:
        e, u = eng.spectrum(k)
        ec, uc = np.zeros_like(e), np.zeros((points, nw, nw), dtype=np.complex128)
        assert eng._L.wnlqg_b200_eval_spectrum(eng._plan, k.ctypes.data_as(dp), points, ec.ctypes.data_as(dp),
                                               uc.ctypes.data_as(dp)) == 0
    assert np.array_equal(e, ec) and np.array_equal(u, uc.transpose(0, 2, 1))
    assert u.flags["C_CONTIGUOUS"]
