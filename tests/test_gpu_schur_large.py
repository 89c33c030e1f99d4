"""The Schur basis of a conical solve whose order 2N = 446 is beyond the fixed-point solver: the cluster kernel's Schur form
against the one-CTA kernel's (RCWA_GB300_EIG_GROUP=256), at a wavelength where a mode of the layer goes through zero."""
import numpy as np
import pytest

from stablercwa_gb300 import stack_from_json

pytestmark = pytest.mark.gpu
M = 111


def crossing(stack, case):
    """The wavelength at which an eigenvalue of Kx^2 - [[eps]] changes its sign, by bisection."""
    layer = next(L for L in stack.layers if not L.homogeneous)
    theta, phi = np.deg2rad(case["theta"]), np.deg2rad(case["phi"])
    h = np.subtract.outer(np.arange(2 * M + 1), np.arange(2 * M + 1))
    edges, eps = np.asarray(layer.edges), np.asarray(layer.n_values) ** 2
    w = np.exp(-2j * np.pi * h[..., None] * edges / stack.period)
    hs = np.where(h == 0, 1, h)[..., None]
    E = np.where((h == 0)[..., None], np.diff(edges) / stack.period, np.diff(w, axis=-1) / (-2j * np.pi * hs)) @ eps

    def negative(wavelength):
        kx = stack.nI * np.sin(theta) * np.cos(phi) - np.arange(-M, M + 1) * wavelength / stack.period
        return int((np.linalg.eigvalsh(np.diag(kx ** 2) - E) < 0).sum())

    lo, hi = 0.9, 1.05
    below = negative(lo)
    assert negative(hi) != below
    for _ in range(48):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if negative(mid) == below else (lo, mid)
    return 0.5 * (lo + hi)


def test_schur_basis_by_cluster(monkeypatch, conical_cases):
    from stablercwa_gb300.engine import Engine
    case = next(c for c in conical_cases if c["name"] == "schur_at_crossing")
    stack = stack_from_json(case["stack"])
    wavelength = crossing(stack, case)
    eng = Engine()
    monkeypatch.delenv("RCWA_GB300_EIG_GROUP", raising=False)
    cluster = eng.solve_conical(stack, wavelength, case["theta"], case["phi"], M)
    monkeypatch.setenv("RCWA_GB300_EIG_GROUP", "256")
    cta = eng.solve_conical(stack, wavelength, case["theta"], case["phi"], M)
    eng.close()
    assert cluster["status"] == 0 and cta["status"] == 0 and cluster["n_schur"] == cta["n_schur"] == 1
    for key in ("DEr", "DEt"):
        assert np.max(np.abs(cluster[key] - cta[key])) <= 1e-10, key
    assert abs(cluster["DEr"].sum() + cluster["DEt"].sum() - 2.0) <= 1e-9
