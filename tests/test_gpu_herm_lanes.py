"""The Hermitian solver's work split at its edges: matrices per warp of the QL iteration (one up to 152 matrices, two up
to 304, ...), rows per CTA of the rotations' application (16 from order 222 when 32 rows would outnumber the SMs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("n,batch", [(25, 1), (25, 33), (25, 152), (25, 153), (25, 305), (26, 4865), (221, 23), (222, 21), (222, 22),
                                     (301, 16), (430, 11)])
def test_hermitian_eigenpairs(n, batch):
    from stablercwa_gb300.engine import Engine
    rng = np.random.default_rng(n + batch)
    kinds = rng.normal(size=(min(batch, 7), n, n)) + 1j * rng.normal(size=(min(batch, 7), n, n))
    kinds = kinds + kinds.conj().transpose(0, 2, 1)
    a = kinds[np.arange(batch) % len(kinds)]
    eng = Engine()
    w, v, info = eng.eig_hermitian_batch(a)
    eng.close()
    assert not info.any()
    for k in sorted({0, batch // 2, batch - 1}):
        # n eps |A| with a factor of a few, as for the other Hermitian forms
        assert np.linalg.norm(a[k] @ v[k] - v[k] * w[k]) <= 8 * n * EPS * np.linalg.norm(a[k])
        assert np.linalg.norm(v[k].conj().T @ v[k] - np.eye(n)) <= 8 * n * EPS * np.sqrt(n)
    # the same matrix gives the same pairs wherever it lies in the batch
    for k in range(len(kinds), min(batch, 3 * len(kinds))):
        assert np.array_equal(w[k], w[k % len(kinds)]) and np.array_equal(v[k], v[k % len(kinds)])
