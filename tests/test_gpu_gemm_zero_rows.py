"""Tensor-core products that a zero row or column makes zero leave what they are added to as it is (csrc/gemm_tc.cu): solves
with separate diagonal blocks of very different size, whose trailing updates are such products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small_first", [False, True])
@pytest.mark.parametrize("scale", [1e-12, 1e-200])
def test_blocks_of_different_size(small_first, scale):
    from stablercwa_gb300.engine import Engine
    n, batch, h = 96, 64, 48  # enough work for the tensor cores, updates across the blocks' border
    rng = np.random.default_rng(1)
    noise = (rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))) * 0.1 / np.sqrt(n)
    a = np.eye(n) + noise
    a[:, :h, h:] = 0.0
    a[:, h:, :h] = 0.0
    part = slice(0, h) if small_first else slice(h, n)
    a[:, part, part] *= scale
    b = rng.normal(size=(batch, n, 40)) + 1j * rng.normal(size=(batch, n, 40))
    b[:, part] *= scale
    eng = Engine()
    x, singular = eng.solve_batch(a, b)
    eng.close()
    assert not singular.any()
    for p in (slice(0, h), slice(h, n)):
        want = np.linalg.solve(a[:, p, p], b[:, p])
        # conditions below 2: n eps of the largest entry and some
        assert np.abs(x[:, p] - want).max() <= 4 * n * 2.2e-16 * np.abs(want).max()
