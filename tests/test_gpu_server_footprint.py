"""The serving loop's footprint of a request (what its HBM budget counts) is at least what the solve holds: one request at a
time, against the high-water mark of the device's memory pool. Several gratings, both polarisations, absorbing or not, at
small and large truncations."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
PERIOD = 0.574


def stack(gratings, loss):
    from stablercwa_gb300 import Layer, Stack
    layers = [Layer.grating(0.1, [0.0, 0.2 + 0.05 * g, PERIOD], [complex(1.46 + 0.2 * g, loss), 1.0]) for g in range(gratings)]
    return Stack(nI=1.0, nII=1.46, period=PERIOD, layers=[*layers, Layer.uniform(0.1, 2.1)])


def stack2d(patterned):
    from stablercwa_gb300 import Layer2D, Stack2D, XProfile2D
    layers = [Layer2D.patterned(0.1, [0.0, 0.2, 0.5 + 0.05 * g, 0.8],
                                [XProfile2D([0.0, 0.8], [1.0]), XProfile2D([0.0, 0.2, 0.5, 0.8], [1.0, 2.0, 1.0]), XProfile2D([0.0, 0.8], [1.0])])
              for g in range(patterned)]
    return Stack2D(nI=1.0, nII=1.46, Lx=0.8, Ly=0.8, layers=layers)


class PoolMark:
    """The high-water mark of the default memory pool (CU_MEMPOOL_ATTR_USED_MEM_HIGH)."""

    def __init__(self):
        import torch
        torch.zeros(1, device="cuda")
        self.cu, self.pool = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def reset(self):
        import torch
        torch.cuda.synchronize()
        assert self.cu.cuMemPoolSetAttribute(self.pool, 8, ctypes.byref(ctypes.c_uint64(0))) == 0

    def read(self):
        v = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolGetAttribute(self.pool, 8, ctypes.byref(v)) == 0
        return v.value


def test_footprint_covers_the_solve():
    from stablercwa_gb300.engine import Server
    srv = Server(device=0, slots=1, max_batch=1)
    mark = PoolMark()
    jobs = [(f"1d M {M} gratings {g} loss {loss} pol {pol}", lambda M=M, g=g, loss=loss, pol=pol: srv.submit_1d(stack(g, loss), 1.0, 55.0, M, pol))
            for M in (20, 60, 150) for g in (1, 3) for loss in (0.0, 0.02) for pol in (0, 1)]
    jobs += [(f"conical M {M} gratings {g} loss {loss}", lambda M=M, g=g, loss=loss: srv.submit_conical(stack(g, loss), 1.0, 35.0, 20.0, M))
             for M in (10, 40, 75) for g in (1, 3) for loss in (0.0, 0.02)]
    jobs += [(f"crossed M {M} patterned {g}", lambda M=M, g=g: srv.submit_2d(stack2d(g), 0.7, 10.0, 20.0, M, M, (1.0, 0.0)))
             for M in (2, 6) for g in (1, 3)]
    over = []
    for name, submit in jobs:
        before = None
        for _ in range(2):  # the first request of a kind also loads kernels
            mark.reset()
            before = mark.read()
            reply = srv.wait(submit())[0]
        held = mark.read() - before
        if held > reply["footprint_bytes"]:
            over.append((name, held, reply["footprint_bytes"]))
    srv.close()
    assert not over
