"""Batched solves and products where the launch form changes: panels in shared memory or in place, a warp or a
thread per column, a warp per panel, two or eight columns of a product per warp, FP64 or digit products."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def eng():
    from stablercwa_gb300.engine import Engine
    return Engine()


def random(rng, *shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def check(a, x, b):
    # Gaussian elimination with partial pivoting: residual of n eps |A| |X| times a growth of a few units
    n = a.shape[-1]
    for k in range(len(a)):
        bound = 16 * n * EPS * np.linalg.norm(a[k]) * np.linalg.norm(x[k])
        assert np.linalg.norm(a[k] @ x[k] - b[k]) <= bound


@pytest.mark.parametrize("n,nrhs,batch", [(100, 1, 1), (100, 100, 3), (127, 5, 2), (128, 128, 1), (129, 1, 140), (121, 121, 75),
                                          (440, 3, 2), (441, 2, 2), (473, 473, 1), (64, 64, 607), (64, 1, 608),
                                          (65, 2, 608), (33, 33, 700), (32, 32, 200), (15, 15, 3), (16, 16, 3), (16, 4, 650), (41, 1, 300)])
def test_solves_at_the_edges_of_the_launch_forms(eng, n, nrhs, batch):
    rng = np.random.default_rng(n + batch)
    a, b = random(rng, batch, n, n), random(rng, batch, n, nrhs)
    x, singular = eng.solve_batch(a, b)
    assert not singular.any()
    check(a, x, b)


@pytest.mark.parametrize("n,batch", [(111, 3), (450, 1), (51, 610)])
@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_pivots_whose_squares_leave_the_range(eng, n, batch, scale):
    rng = np.random.default_rng(n)
    a, b = random(rng, batch, n, n), random(rng, batch, n, 2)
    x, singular = eng.solve_batch(a * scale, b * scale)
    assert not singular.any()
    check(a, x, b)


@pytest.mark.parametrize("n", [111, 450])
def test_singular_and_nan_systems_leave_their_neighbours_alone(eng, n):
    rng = np.random.default_rng(n)
    a, b = random(rng, 3, n, n), random(rng, 3, n, 4)
    a[0][:, 40] = 0.0
    a[2][:, 35] = np.nan
    x, singular = eng.solve_batch(a, b)
    assert list(singular) == [True, False, False]
    assert np.isnan(x[0]).all() and np.isnan(x[2]).any()
    check(a[1:2], x[1:2], b[1:2])


def test_row_swaps_reach_every_column(eng):
    rng = np.random.default_rng(5)
    n = 140
    p = np.stack([np.eye(n)[rng.permutation(n)] + 0j for _ in range(2)])
    b = random(rng, 2, n, 3)
    x, singular = eng.solve_batch(p, b)
    assert not singular.any()
    np.testing.assert_array_equal(x, p.transpose(0, 2, 1) @ b)


@pytest.mark.parametrize("m,k,n,batch", [(1, 1, 1, 1), (33, 17, 5, 2), (121, 121, 121, 1), (121, 121, 121, 2), (121, 121, 121, 3),
                                         (64, 64, 9, 303), (64, 64, 9, 151), (40, 3, 130, 7),
                                         (9, 32, 50, 300), (9, 32, 50, 4), (25, 5, 33, 700), (1, 33, 1, 700)])
def test_products_at_the_edges_of_the_launch_forms(eng, m, k, n, batch):
    rng = np.random.default_rng(m + batch)
    a, b = random(rng, batch, m, k), random(rng, batch, k, n)
    c = eng.multiply_batch(a, b)
    # each entry: k terms, each off by a few units of its magnitude; a digit product by units of the row and column maxima
    bound = 8 * EPS * k * np.abs(a).max(axis=2, keepdims=True) * np.abs(b).max(axis=1, keepdims=True)
    assert (np.abs(c - a @ b) <= bound).all()
