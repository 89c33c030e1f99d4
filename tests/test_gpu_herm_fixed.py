"""The blocked Hermitian reduction's fixed-point panels at the edges of panels, row passes and scales."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def eng():
    from stablercwa_gb300.engine import Engine
    return Engine()


def hermitian(rng, n):
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    return a + a.conj().T


@pytest.mark.parametrize("n", [64, 65, 66, 96, 97, 98, 113, 128, 129])
def test_fixed_point_panels(eng, n):
    rng = np.random.default_rng(n)
    batch = 48000 // n + 2  # the blocked form
    q = np.linspace(-1.0, 1.0, n)
    kinds = [hermitian(rng, n), hermitian(rng, n).real + 0j, np.diag(rng.normal(size=n)) + 0j,
             np.diag(1e4 * q * q) + hermitian(rng, n), hermitian(rng, n) * 1e-200, hermitian(rng, n) * 1e200,
             np.zeros((n, n), complex), hermitian(rng, n) * 1e-285,
             np.kron(np.eye(2), hermitian(rng, n))[:n, :n] if n % 2 else np.ones((n, n), complex)]
    block = np.diag(np.ones(n - 1), 1) + 0j
    kinds.append(block + block.conj().T)  # tridiagonal already
    a = np.stack([kinds[k % len(kinds)] for k in range(batch)])
    w, v, info = eng.eig_hermitian_batch(a)
    assert not info.any()
    # Householder tridiagonalisation and QL: n eps |A| with a factor of a few; the same for the vectors' orthogonality
    for k in list(range(2 * len(kinds))) + [batch - 1]:
        s = np.abs(a[k]).max() or 1.0
        m = a[k] / s
        assert np.linalg.norm(m @ v[k] - v[k] * (w[k] / s)) <= 8 * n * EPS * max(np.linalg.norm(m), 1.0)
        assert np.linalg.norm(v[k].conj().T @ v[k] - np.eye(n)) <= 8 * n * EPS * np.sqrt(n)


def test_a_matrix_that_is_not_finite_leaves_the_others_alone(eng):
    import torch
    n = 70
    rng = np.random.default_rng(1)
    a = np.stack([hermitian(rng, n) for _ in range(8)] * 90)
    a[3, 5, 6] = a[3, 6, 5] = np.nan
    a[4, 0, 0] = np.inf
    d = torch.tensor(np.ascontiguousarray(a.transpose(0, 2, 1)), device="cuda")
    w = torch.empty((len(a), n), dtype=torch.complex128, device="cuda")
    v = torch.empty_like(d)
    info = torch.full((len(a),), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng.eig_hermitian_batch_device(n, len(a), d.data_ptr(), w.data_ptr(), v.data_ptr(), info.data_ptr())
    eng.synchronize()
    v, w = v.cpu().numpy().transpose(0, 2, 1), w.cpu().numpy()
    for k in (2, 5, 11, 12):
        assert info[k] == 0
        assert np.linalg.norm(a[k] @ v[k] - v[k] * w[k]) <= 8 * n * EPS * np.linalg.norm(a[k])
