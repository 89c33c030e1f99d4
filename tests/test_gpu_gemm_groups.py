"""The tensor-core product's accumulation groups (quads of digits, single pairs) at the edges of their chunks of K: every
count of 64-wide K blocks around one stage, one group of quads (8 blocks) and one of single pairs (16), with ragged
last blocks and tiles, against numpy's product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 7, 8, 9, 15, 16, 17, 25])
def test_accumulation_groups(blocks):
    from stablercwa_gb300.engine import Engine, gemm_info
    rng = np.random.default_rng(blocks)
    eng = Engine()
    for m, n, k in ((65, 129, 32 * blocks), (64, 127, 32 * blocks - 1)):
        a = rng.normal(size=(3, m, k)) + 1j * rng.normal(size=(3, m, k))
        b = rng.normal(size=(3, k, n)) + 1j * rng.normal(size=(3, k, n))
        ra = np.max(np.maximum(np.abs(a.real), np.abs(a.imag)), axis=2)
        cb = np.max(np.maximum(np.abs(b.real), np.abs(b.imag)), axis=1)
        # the FP64 product's own error scale, as in the other product tests
        bound = 4.0 * k * 2.0 ** -53 * ra[:, :, None] * cb[:, None, :]
        assert np.all(np.abs(eng.multiply_batch(a, b) - a @ b) <= bound)
    eng.close()
    assert gemm_info()[2] == 0  # no product kernel gave up on a wait
