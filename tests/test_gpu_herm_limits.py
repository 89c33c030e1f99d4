"""The Hermitian solver on both sides of the limits of its fixed-point reduction (csrc/eig.cu herm_fixed_reduce_wanted): n *
batch = 48000 below order 64, 360 matrices from order 64 on. Residual and orthonormality of matrices from both ends and
the middle of the batch, at the bounds of tests/test_gpu_eig_fixed.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(33, 1454), (33, 1455), (40, 1200), (40, 1201), (63, 761), (63, 762), (64, 360), (64, 361),
                                     (121, 360), (121, 361), (161, 298), (161, 299)])
def test_both_sides(n, batch):
    from stablercwa_gb300.engine import Engine
    rng = np.random.default_rng(n)
    few = rng.normal(size=(3, n, n)) + 1j * rng.normal(size=(3, n, n))
    few = few + few.conj().transpose(0, 2, 1)
    few[1] = np.diag(((np.arange(n) - n // 2) * 1.3 + 0.4) ** 2) + 0.1 * few[1]  # a layer's shape
    a = few[np.arange(batch) % 3]
    eng = Engine()
    w, v, info = eng.eig_hermitian_batch(a)
    eng.close()
    assert not info.any()
    for k in (0, 1, 2, batch // 2, batch // 2 + 1, batch - 2, batch - 1):
        assert np.abs(w[k].imag).max() == 0.0
        assert np.linalg.norm(a[k] @ v[k] - v[k] * w[k]) <= 1e-13 * np.linalg.norm(a[k])
        assert np.abs(v[k].conj().T @ v[k] - np.eye(n)).max() <= 1e-13
