"""RCWA_GB300_AUTOTUNE=auto tunes the keys that the built-in rule gives to FP64 forms and no others: where it takes the
fixed-point reduction (for this batch or a smaller one of the same key) or the general fixed-point solver, solves record
nothing and give the same bits as without a tuner."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import hashlib
import numpy as np
from stablercwa_gb300 import Layer, Stack
from stablercwa_gb300.engine import Engine, autotune_table
eng = Engine()
for index, M, points in ((1.46, 30, 100), (1.46 + 0.01j, 30, 100), (1.46, 60, 400)):
    stack = Stack(nI=1.0, nII=1.46, period=0.574, layers=[Layer.grating(0.4, [0.0, 0.2, 0.574], [index, 1.0])])
    pts = np.stack([np.linspace(0.9, 1.1, points), np.full(points, 55.0)], axis=1)
    r = eng.solve1d_arrays(stack, pts, M, 0)
    print(M, points, hashlib.sha256(r["R"].tobytes()).hexdigest())
print("table:", autotune_table().split())
rng = np.random.default_rng(1)
a = rng.normal(size=(600, 121, 121)) + 0j
eng.eig_hermitian_batch(a)
print("then:", "hermitian 121 512" in autotune_table())
"""


def run(mode):
    env = dict(os.environ, RCWA_GB300_AUTOTUNE=mode)
    env.pop("RCWA_GB300_EIG_GROUP", None)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300, env=env, cwd=root)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip().splitlines()


def test_auto_leaves_fixed_point_keys_alone():
    auto, off = run("auto"), run("0")
    assert auto[:3] == off[:3]
    assert auto[3] == "table: []" and auto[4] == "then: True" and off[4] == "then: False"
