"""Divide and conquer (RCWA_GB300_HERM_DC=1) on batches that hold matrices which the fixed-point reduction declines: a
zero matrix beside others gets its own eigenpairs (zeros and an orthonormal basis), whatever earlier calls left in the
workspace. Orders below 64 with few matrices a lane group, and 64 matrices' columns where one lane group is a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(24, 700), (33, 900), (63, 640), (64, 310)])
def test_zero_matrices_by_divide_and_conquer(monkeypatch, n, batch):
    from stablercwa_gb300.engine import Engine
    rng = np.random.default_rng(n)
    few = rng.normal(size=(7, n, n)) + 1j * rng.normal(size=(7, n, n))
    few = few + few.conj().transpose(0, 2, 1)
    a = few[np.arange(batch) % 7]
    eng = Engine()
    monkeypatch.setenv("RCWA_GB300_HERM_DC", "1")
    eng.eig_hermitian_batch(a)  # the workspace the next call gets holds this call's d, e and Q
    zeros = sorted({3, batch // 2, batch - 1})
    a[zeros] = 0.0
    w, v, info = eng.eig_hermitian_batch(a)
    eng.close()
    assert not info.any()
    for k in zeros:
        assert not w[k].any()
        assert np.abs(v[k].conj().T @ v[k] - np.eye(n)).max() <= 1e-14 * n
    for k in (0, 4, batch // 2 + 1):
        assert np.linalg.norm(a[k] @ v[k] - v[k] * w[k]) <= 1e-13 * np.linalg.norm(a[k])
