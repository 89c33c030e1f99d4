"""Matrices whose small eigenvalues FP64 keeps relative to themselves (fix_range_kernel in csrc/eig_fixed.cuh leaves them to
the FP64 kernels): diagonal matrices over twenty decades and blocks of very different size, beside ordinary matrices of the
same batch, through the Hermitian entry and through the general one without sweep counts. Each block's eigenvalues are
held to the block's own norm, every diagonal entry to itself. Orders and batches on both sides of the fixed-point reduction's limits and of its range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def batch_of(n, batch, hermitian, seed):
    rng = np.random.default_rng(seed)
    few = rng.normal(size=(5, n, n)) + 1j * rng.normal(size=(5, n, n))
    if hermitian:
        few = few + few.conj().transpose(0, 2, 1)
    a = few[np.arange(batch) % 5].copy()
    h = n // 2
    blocks = few[0].copy()
    cut = h if hermitian else n - h
    blocks[:cut, cut:] = 0.0
    blocks[cut:, :cut] = 0.0
    # FP64 keeps the small block in either place of a Hermitian matrix; the QR iteration's shifts pass over a first block
    small, large = (slice(0, h), slice(h, n)) if hermitian else (slice(n - h, n), slice(0, n - h))
    blocks[small, small] *= 1e-10
    blocks[large, large] *= 1e10
    diagonal = np.diag(np.logspace(0, -20, n)).astype(complex)
    kinds = {0: diagonal, batch // 2: blocks, batch - 1: diagonal[::-1, ::-1]}
    for k, m in kinds.items():
        a[k] = m
    return a, kinds


def check(a, kinds, w, v):
    n = a.shape[1]
    h = n // 2
    for k, m in kinds.items():
        if np.count_nonzero(m) == n:
            got, want = np.sort(w[k].real), np.sort(np.diag(m).real)
            assert np.all(np.abs(got - want) <= 4 * EPS * np.abs(want))
            continue
        size = np.sort(np.abs(w[k]))
        assert np.all(size[h:] > 1e3 * size[:h].max())
        order = np.argsort(np.abs(w[k]))
        first = np.abs(m[0, 0]) < 1.0  # the small block comes first
        cut = h if first else n - h
        parts = (m[:cut, :cut], m[cut:, cut:]) if first else (m[cut:, cut:], m[:cut, :cut])
        for part, values in zip(parts, (w[k][order[:h]], w[k][order[h:]])):
            # trace and sum of squares of a block, at FP64's backward error of n eps of its norm
            norm = np.linalg.norm(part)
            assert abs(values.sum() - np.trace(part)) <= 16 * n * EPS * norm
            assert abs((values ** 2).sum() - np.trace(part @ part)) <= 16 * n * EPS * norm ** 2
    for k in (1, a.shape[0] // 2 + 1):
        if k in kinds or k >= a.shape[0]:
            continue
        assert np.linalg.norm(a[k] @ v[k] - v[k] * w[k]) <= 1e-13 * np.linalg.norm(a[k]) * np.sqrt(n)


@pytest.mark.parametrize("n,batch", [(2, 5), (23, 40), (30, 3), (41, 1300), (64, 360), (64, 400), (121, 3), (441, 3), (460, 3)])
def test_hermitian(n, batch):
    from stablercwa_gb300.engine import Engine
    a, kinds = batch_of(n, batch, True, n)
    eng = Engine()
    w, v, info = eng.eig_hermitian_batch(a)
    eng.close()
    assert not info.any()
    check(a, kinds, w, v)


@pytest.mark.parametrize("n,batch", [(23, 3), (24, 3), (30, 700), (121, 4), (200, 3)])
def test_general(n, batch):
    import torch
    from stablercwa_gb300.engine import Engine
    a, kinds = batch_of(n, batch, False, n)
    d_a = torch.from_numpy(np.ascontiguousarray(a.transpose(0, 2, 1))).to("cuda")
    w = torch.empty((batch, n), dtype=torch.complex128, device="cuda")
    v = torch.empty((batch, n, n), dtype=torch.complex128, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng = Engine()
    eng.eig_batch_device(n, batch, d_a.data_ptr(), w.data_ptr(), v.data_ptr(), info.data_ptr())
    torch.cuda.synchronize()
    eng.close()
    assert not info.cpu().numpy().any()
    check(a, kinds, w.cpu().numpy(), v.cpu().numpy().transpose(0, 2, 1))
