"""The FP64 path's two eigensolver stages on chosen matrices (17 orbitals and more): what stage 1 leaves
along a chain of warm starts, and the spectra that stage 2 makes of it and of starts at its bounds."""
import numpy as np
import pytest

import eigensolver_stages as native

pytestmark = pytest.mark.gpu

# Stage 2 orthonormalises stage 1's vectors to second order in D = V^H V - 1, which leaves 5/16 |D|^3:
# 1e-15 of it at |D| = 1.5e-5.  Its first completion asks for ratios |a_ij| / |d_i - d_j| <= 2^-13.
ORTHONORMAL, RATIO = 1.5e-5, 2.0 ** -13


@pytest.fixture(scope="module")
def stages():
    return native.load()


def unitary(rng, nw, angle=None):
    """Haar-like, or exp(i K) with the largest |K_ij| = angle."""
    z = rng.standard_normal((nw, nw)) + 1j * rng.standard_normal((nw, nw))
    if angle is None:
        return np.linalg.qr(z)[0]
    k = z + z.conj().T
    w, q = np.linalg.eigh(k * (angle / np.max(np.abs(k))))
    return (q * np.exp(1j * w)) @ q.conj().T


def stage1_quality(h, v):
    """Spectral norm of V^H V - 1 and the largest ratio of V^H H V."""
    w = v[:h.shape[0], :h.shape[0]].astype(complex)
    a = w.conj().T @ h @ w
    d = a.diagonal().real
    gap = np.abs(d[:, None] - d) + 1e300 * np.eye(len(d))
    return np.linalg.norm(w.conj().T @ w - np.eye(len(d)), 2), np.max(np.abs(a) / gap)


def check_spectrum(h, e, u):
    scale = max(np.linalg.norm(h), 1e-300)
    assert np.max(np.abs(e - np.linalg.eigvalsh(h))) <= 1e-13 * scale
    assert np.max(np.abs(h @ u - u * e)) <= 1e-12 * scale
    assert np.max(np.abs(u.conj().T @ u - np.eye(len(e)))) <= 1e-13


def skewed(rng, nw, scales):
    """One deep level and a band of others, slowly rotating, with the given scales."""
    q, h = unitary(rng, nw), []
    for s in scales:
        h.append(s * (q * np.r_[-1.0, np.linspace(-0.25, 0.25, nw - 1)]) @ q.conj().T)
        q = unitary(rng, nw, 1e-3) @ q
    return np.array([0.5 * (x + x.conj().T) for x in h])


@pytest.mark.parametrize("chain", ["falling", "rising", "jumps"])
@pytest.mark.parametrize("nw", [20, 31, 40, 96])
def test_warm_chain_whose_norm_moves(stages, nw, chain):
    rng = np.random.default_rng(nw)
    if chain == "jumps":
        scales = [1.0, 5.0, 0.1, -1.0, 1.0, 0.0, 2.0, -0.3, -8.0, 1e-20, 1.0, -1e20, 3.0, 0.0, 0.0, 1e-3]
    else:
        scales = 1.5 * 0.98 ** np.arange(150)
        scales = scales if chain == "falling" else scales[::-1]
    h = skewed(rng, nw, scales)
    v, e, u = native.run(stages, h)
    got = np.array([stage1_quality(a, b) for a, b, s in zip(h, v, scales) if s != 0.0])
    assert np.max(got[:, 0]) <= ORTHONORMAL
    assert np.max(got[:, 1]) <= RATIO
    for i in range(0, len(h), 1 if chain == "jumps" else 7):
        check_spectrum(h[i], e[i], u[i])


@pytest.mark.parametrize("nw", [18, 32, 64, 96, 128])
@pytest.mark.parametrize("angle", [1e-2, 9e-4, 4.7e-4, 2.3e-4])
def test_warm_start_from_close_neighbours(stages, nw, angle):
    rng = np.random.default_rng(nw)
    q, h = unitary(rng, nw), []
    for _ in range(12):
        a = (q * np.linspace(-1.0, 1.0, nw)) @ q.conj().T
        h.append(0.5 * (a + a.conj().T))
        q = unitary(rng, nw, angle) @ q
    h = np.array(h)
    v, e, u = native.run(stages, h)
    got = np.array([stage1_quality(a, b) for a, b in zip(h, v)])
    assert np.max(got[:, 0]) <= ORTHONORMAL
    assert np.max(got[:, 1]) <= RATIO
    check_spectrum(h[-1], e[-1], u[-1])


@pytest.mark.parametrize("nw", [17, 32, 64, 96, 128])
@pytest.mark.parametrize("ratio", [1e-6, 1e-5, 3e-5, 7e-5])
@pytest.mark.parametrize("coherent", [True, False])
def test_every_pair_near_the_completion_bound(stages, nw, ratio, coherent):
    """Starts exp(i K) away from the eigenvectors with every |K_ij| = ratio (below 2^-13): the norm of K
    is up to nw times larger."""
    rng = np.random.default_rng(nw)
    q = unitary(rng, nw)
    phase = np.zeros((nw, nw)) if coherent else rng.uniform(0.0, 2.0 * np.pi, (nw, nw))
    k = np.triu(np.exp(1j * phase), 1)
    w, p = np.linalg.eigh(ratio * (k + k.conj().T))
    h = (q * np.linspace(-1.0, 1.0, nw)) @ q.conj().T
    h = 0.5 * (h + h.conj().T)
    start = q @ (p * np.exp(1j * w)) @ p.conj().T
    _, e, u = native.run(stages, h[None], start=start[None])
    check_spectrum(h, e[0], u[0])
