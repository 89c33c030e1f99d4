"""The general eigensolver's fixed-point form on the GPU: what rcwa_gpu_eig_batch_dev takes when it is asked for no
sweep counts, at the edges of its tiles and of its range of orders. Eigenpair residuals within 1e-13 of ||A||_F (the
bound of the other forms), eigenvalues within 1e-11 ||A||_2 of numpy's, info 0; a matrix it cannot scale (zero, non-finite) gets
the FP64 kernels' answer inside the same batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from stablercwa_gb300.engine import Engine
    e = Engine()
    yield e
    e.close()


def layer(n, rng):
    """Kx^2 - [[eps]] of an absorbing binary grating."""
    f, k, s = rng.uniform(0.3, 0.6), rng.uniform(0.9, 1.2) / 0.574, rng.uniform()
    h = np.subtract.outer(np.arange(n), np.arange(n))
    hs = np.where(h == 0, 1, h)
    c = np.where(h == 0, f, (1 - np.exp(-2j * np.pi * h * f)) / (2j * np.pi * hs))
    return np.diag((s - (np.arange(n) - n // 2) * k) ** 2) - (np.eye(n) + (2.1316 + 0.03j - 1.0) * c)


def solve(eng, a, sweeps):
    import torch
    batch, n = a.shape[:2]
    d = torch.tensor(np.ascontiguousarray(a.transpose(0, 2, 1)), device="cuda")
    w = torch.empty((batch, n), dtype=torch.complex128, device="cuda")
    v = torch.empty((batch, n, n), dtype=torch.complex128, device="cuda")
    info = torch.full((batch,), -1, dtype=torch.int32, device="cuda")
    sw = torch.zeros(batch, dtype=torch.int32, device="cuda") if sweeps else None
    torch.cuda.synchronize()
    eng.eig_batch_device(n, batch, d.data_ptr(), w.data_ptr(), v.data_ptr(), info.data_ptr(), sw.data_ptr() if sweeps else None)
    eng.synchronize()
    return w.cpu().numpy(), v.cpu().numpy().transpose(0, 2, 1), info.cpu().numpy()


@pytest.mark.parametrize("n,batch", [(24, 5), (31, 3), (32, 3), (33, 700), (64, 2), (65, 2), (97, 2), (121, 3), (129, 2), (162, 2),
                                     (353, 1), (440, 1)])
def test_eigenpairs(eng, n, batch):
    rng = np.random.default_rng(n)
    a = np.stack([layer(n, rng) if k % 2 == 0 else rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)) for k in range(batch)])
    w, v, info = solve(eng, a, False)
    assert (info == 0).all()
    for k in range(min(batch, 6)):
        r = np.linalg.norm(a[k] @ v[k] - v[k] * w[k], axis=0) / np.linalg.norm(v[k], axis=0)
        assert r.max() <= 1e-13 * np.linalg.norm(a[k]), (k, r.max())
        assert np.allclose(np.linalg.norm(v[k], axis=0), 1.0, atol=1e-12)
        if k % 2 == 0:  # (random matrices' eigenvalues are less well conditioned than this bound asks)
            ref = np.linalg.eigvals(a[k])
            gap = np.abs(np.subtract.outer(w[k], ref))
            assert gap.min(1).max() <= 1e-11 * np.linalg.norm(a[k], 2) and len(set(gap.argmin(1))) == n


def test_matrices_left_to_the_fp64_kernels(eng):
    rng = np.random.default_rng(1)
    a = np.stack([layer(40, rng) for _ in range(6)])
    a[1] = 0.0
    a[3, 7, 9] = np.nan
    w, v, info = solve(eng, a, False)
    w0, v0, info0 = solve(eng, a, True)  # with sweep counts: the FP64 kernels throughout
    assert np.array_equal(info, info0) and info[1] == 0 and info[3] != 0
    assert np.array_equal(w[1], w0[1]) and np.array_equal(v[1], v0[1])
    for k in (0, 2, 4, 5):
        r = np.linalg.norm(a[k] @ v[k] - v[k] * w[k], axis=0)
        assert r.max() <= 1e-13 * np.linalg.norm(a[k])


@pytest.mark.parametrize("n,batch", [(24, 4), (32, 4), (33, 1400), (65, 3), (121, 396), (121, 397), (301, 2), (440, 1)])
def test_hermitian(eng, n, batch):
    """Both sides of the fixed-point reduction's limit (n * batch = 48000) and of its orders."""
    rng = np.random.default_rng(n + batch)
    few = np.stack([layer(n, rng) for _ in range(min(batch, 4))])
    few = 0.5 * (few + few.conj().transpose(0, 2, 1))
    a = few[np.arange(batch) % len(few)]
    if batch > 4:
        a[5] = 0.0  # left to the FP64 kernels
    w, v, info = eng.eig_hermitian_batch(a)
    assert (info == 0).all()
    for k in range(min(batch, 7)):
        r = np.linalg.norm(a[k] @ v[k] - v[k] * w[k], axis=0)
        assert r.max() <= 1e-13 * np.linalg.norm(a[k])
        assert np.abs(v[k].conj().T @ v[k] - np.eye(n)).max() <= 1e-13
