"""The one-CTA FP32 eigensolve over its whole range of matrix sizes: odd sizes (padded to the even
number of indices that the pairing needs), both leading dimensions, matrices that need no rotation,
entries far from 1, and spectra whose kept eigenvectors the FP64 correction finishes."""

import numpy as np
import pytest

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


def _matrix(T, seed):
    """Hermitian, eigenvalues 1, 2, ..., T (gaps of at least 1 / T of the largest)."""
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((T, T)) + 1j * rng.standard_normal((T, T)))
    a = (q * np.arange(1, T + 1)) @ q.conj().T
    return (a + a.conj().T) / 2


def _eigh(a, K):
    T = a.shape[0]
    ev, vec, w = zeros(T * 8), zeros(T * T * 16), zeros(K * T * 8)
    work = zeros(hv.lib().hv_pca_eigh_workspace(T))
    call("hv_pca_eigh", ptr(dev(a.astype(np.complex128))), T, ptr(ev), ptr(vec), T - K, T - 1, ptr(w), ptr(work), None)
    # eigenvectors are columns of a column-major matrix
    return host(ev, np.float64, (T,)), host(vec, np.complex128, (T, T)).T, host(w, np.complex64, (K, T))


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 70, 3e-9])
@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 16, 17, 31, 32, 33, 34, 47, 63, 64])
def test_every_size(cuda, T, scale):
    a = _matrix(T, T) * scale
    K = min(4, T)
    ev, vec, w = _eigh(a, K)
    top = T * scale
    assert np.all(np.diff(ev) >= 0)
    # eigenvalues: FP64 Rayleigh quotients, second order in the FP32 sweeps' error (5e-7 of the
    # Frobenius norm, at most sqrt(T) of the largest)
    assert np.max(np.abs(ev - np.arange(1, T + 1) * scale)) <= 1e-9 * top
    # kept vectors: two first-order FP64 corrections of vectors good to 1e-4 at these gaps
    v = vec[:, T - K:]
    assert np.linalg.norm(a @ v - v * ev[T - K:], axis=0).max() <= 1e-9 * top
    assert np.abs(v.conj().T @ v - np.eye(K)).max() <= 1e-9
    assert np.array_equal(w, v.T.astype(np.complex64))
    # the others: the sweeps' round-off level
    assert np.linalg.norm(a @ vec - vec * ev, axis=0).max() <= 1e-4 * top
    assert np.abs(vec.conj().T @ vec - np.eye(T)).max() <= 1e-4


@pytest.mark.parametrize("T", [3, 32, 33, 64])
def test_no_rotation(cuda, T):
    """A diagonal matrix (no step has a rotation) and the zero matrix."""
    d = np.arange(T, 0, -1.0)
    ev, vec, _ = _eigh(np.diag(d).astype(np.complex128), 1)
    assert np.array_equal(ev, d[::-1])
    assert np.array_equal(vec, np.eye(T)[:, ::-1])
    ev, vec, _ = _eigh(np.zeros((T, T), np.complex128), 1)
    assert np.array_equal(ev, np.zeros(T))


@pytest.mark.parametrize("T", [2, 31, 64])
def test_sparse_rotations(cuda, T):
    """A single coupled pair: every other step of a sweep is looked past."""
    for i, j in ((0, 1), (0, T - 1), (T // 2, T - 1)):
        if i == j:
            continue
        a = np.diag(np.arange(1.0, T + 1)).astype(np.complex128)
        a[i, j] = 0.4 + 0.3j
        a[j, i] = 0.4 - 0.3j
        ev, vec, _ = _eigh(a, min(2, T))
        assert np.max(np.abs(ev - np.linalg.eigvalsh(a))) <= 1e-9 * T
        assert np.linalg.norm(a @ vec - vec * ev, axis=0).max() <= 1e-4 * T
