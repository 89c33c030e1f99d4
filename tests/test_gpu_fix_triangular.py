"""General matrices whose last rows have no entries left of the diagonal: the QR iteration deflates those before it shifts, so a
small block before them, or a small diagonal entry among them, keeps its digits in FP64 (fix_keeps_fp64 in csrc/eig_fixed.cuh
leaves such matrices to the FP64 kernels). The block's eigenvalues are held to its own norm, the diagonal entries to themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def special(n, lead, seed):
    rng = np.random.default_rng(seed)
    g = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    a = np.triu(g)
    a[:lead, :lead] = 1e-10 * g[:lead, :lead]
    a[range(lead, n), range(lead, n)] = 1.0 + np.arange(lead, n)
    a[n - 2, n - 2] = 1e-12
    b = a.copy()
    b[:lead, lead:] = 0.0
    return g, a, b


@pytest.mark.parametrize("n,lead,batch", [(23, 2, 3), (24, 2, 3), (30, 15, 700), (121, 2, 4), (200, 100, 3)])
def test_deflated_rows(n, lead, batch):
    import torch
    from stablercwa_gb300.engine import Engine
    g, a, b = special(n, lead, n)
    m = np.repeat(g[None], batch, axis=0)
    m[0], m[batch - 1] = a, b
    d_a = torch.from_numpy(np.ascontiguousarray(m.transpose(0, 2, 1))).to("cuda")
    w = torch.empty((batch, n), dtype=torch.complex128, device="cuda")
    v = torch.empty((batch, n, n), dtype=torch.complex128, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng = Engine()
    eng.eig_batch_device(n, batch, d_a.data_ptr(), w.data_ptr(), v.data_ptr(), info.data_ptr())
    torch.cuda.synchronize()
    eng.close()
    assert not info.cpu().numpy().any()
    w = w.cpu().numpy()
    for k, x in ((0, a), (batch - 1, b)):
        left = list(w[k])
        for d in np.diag(x)[lead:]:
            i = int(np.argmin(np.abs(np.array(left) - d)))
            assert abs(left.pop(i) - d) <= 4 * EPS * abs(d)
        block, values = x[:lead, :lead], np.array(left)
        norm = np.linalg.norm(block)
        assert abs(values.sum() - np.trace(block)) <= 16 * n * EPS * norm
        assert abs((values ** 2).sum() - np.trace(block @ block)) <= 16 * n * EPS * norm ** 2
