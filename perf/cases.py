"""Timed workloads of the solve engine: what they are, how their inputs are made, and what they should give.

Every case goes through the package's public entry points (Engine and Server of stablercwa_gb300.engine):
one solve at a time as in an interactive session, wavelength / angle sweeps of one structure, conical and
crossed gratings, near fields, and a batch of requests to the serving loop. The structures are the ones the
benchmark and the tests use (the grating on a quarter-wave mirror, the README's grating on a film, stacks of
random gratings and absorbing films, rectangular pillars and staircased discs), seeded.

`exact` restates each solve in plain numpy (complex128): the layer operators, numpy's eigensolvers, and the
reflection recursion from the exit medium up.
"""
import math

import numpy as np
import torch

from stablercwa_gb300 import Layer, Layer2D, Stack, Stack2D, XProfile2D, jones_from_angles_2d

PERIOD = 0.574
POLS = {"te": 0, "tm": 1, "both": 2}


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # One small solve: the README's grating on a film at M = 20, as typed in an interactive session or
        # called by an optimiser that moves one parameter at a time. Launches and latency count.
        dict(name="solve_readme_n41", kind="solve", structure="readme", M=20, points=1, pol="te"),
        # One solve at the benchmark's truncation (grating on a 20-film mirror, N = 121): the plain path.
        dict(name="solve_mirror_n121", kind="solve", structure="mirror", M=60, points=1, pol="tm"),
        # The benchmark's headline sweep: 4096 points, both polarisations, device-resident points and results.
        dict(name="sweep_mirror_n121", kind="device", structure="mirror", M=60, points=4096, pol="both"),
        # The same design with an absorbing ridge (every grating matrix non-Hermitian), a spectrum of it.
        dict(name="sweep_lossy_n121", kind="device", structure="lossy", M=60, points=512, pol="both"),
        # A multilayer of absorbing gratings and films at a moderate truncation, host buffers in and out, one of
        # the gratings given by sampled (FFT) coefficients.
        dict(name="sweep_multilayer_n61", kind="solve", structure="multilayer", M=30, points=128, pol="both"),
        # A high-contrast lossless grating near the largest truncation in use (N = 301), a short scan.
        dict(name="scan_contrast_n301", kind="solve", structure="contrast", M=150, points=16, pol="both"),
        # The benchmark's conical sweep: three lossless gratings and an absorbing film, N = 81.
        dict(name="conical_sweep_n81", kind="conical", structure="conical", M=40, points=1024),
        # One conical solve (N = 51), as an ellipsometry fit calls it.
        dict(name="conical_solve_n51", kind="conical", structure="conical", M=25, points=1),
        # Crossed gratings: a spectrum of a rectangular-pillar design at a small truncation (2N = 98) ...
        dict(name="crossed_sweep_n49", kind="crossed", structure="rect", M1=3, M2=3, points=64),
        # ... and one solve of a staircased-disc design at a converged one (2N = 338).
        dict(name="crossed_solve_n169", kind="crossed", structure="disc", M1=6, M2=6, points=1),
        # Near fields of one solve over depth, and their map over one period: the field viewer.
        dict(name="fields_n81", kind="fields", structure="mirror", M=40, points=1, pol="tm", depths=200, nx=256),
        # Requests of different 1-D structures and truncations submitted together to the serving loop.
        dict(name="serve_mixed", kind="serve", structure="multilayer", M=15, M2=50, requests=24),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "device", "device", "conical", "crossed", "fields", "serve"])
    if kind == "serve":
        lo = rng.randint(8, 24)
        return dict(kind=kind, structure="multilayer", M=lo, M2=rng.randint(lo + 4, 52), requests=rng.randint(6, 26))
    if kind == "crossed":
        M1, M2 = rng.randint(1, 6), rng.randint(1, 6)
        N = (2 * M1 + 1) * (2 * M2 + 1)
        return dict(kind=kind, structure=rng.choice(["rect", "disc"]), M1=M1, M2=M2,
                    points=spread(1, max(1, min(200, int(64 * (49 / N) ** 3)))))
    if kind == "conical":
        M = spread(8, 48)
        return dict(kind=kind, structure="conical", M=M, points=spread(1, max(1, min(2000, int(700 * (81 / (2 * M + 1)) ** 3)))))
    if kind == "fields":
        return dict(kind=kind, structure=rng.choice(["readme", "mirror"]), M=spread(10, 60), points=1,
                    pol=rng.choice(["te", "tm"]), depths=spread(20, 400), nx=rng.choice([100, 128, 256, 301]))
    structure = rng.choice(["readme", "mirror", "lossy", "multilayer", "contrast"])
    n_max = 151 if structure in ("lossy", "multilayer") else 301
    M = spread(8, (n_max - 1) // 2)
    n = 2 * M + 1
    if structure in ("readme", "mirror", "contrast"):
        most = 16 if n > 181 else int(3000 * (121 / n) ** 3)
    else:
        most = int((500 if structure == "lossy" else 150) * (121 / n) ** 3)
    if kind == "solve":
        most = min(most, 200)
    return dict(kind=kind, structure=structure, M=M, points=spread(1, max(1, min(4000, most))),
                pol=rng.choice(["te", "tm", "both", "both"]))


def work(case):
    """Bytes in and out, and flops: per grating matrix of order n the eigensolve (about 105 n^3 for the general
    Hessenberg + QR solver, 12 n^3 for a Hermitian matrix) and the interface algebra (about 40 n^3)."""
    kind = case["kind"]
    if kind == "serve":
        ns = [2 * M + 1 for M in _serve_orders(case)]
        return {"bytes": sum(16 + 48 * n for n in ns), "flops": sum(3 * 145 * n ** 3 for n in ns)}
    if kind == "crossed":
        N = (2 * case["M1"] + 1) * (2 * case["M2"] + 1)
        n, mats, c = 2 * N, 2 * case["points"], 145
        return {"bytes": case["points"] * (72 + 210 * N), "flops": mats * c * n ** 3}
    n = 2 * case["M"] + 1
    if kind == "conical":
        return {"bytes": case["points"] * (24 + 216 * n), "flops": case["points"] * 3 * (2 * 12 * n ** 3 + 40 * (2 * n) ** 3)}
    solves = case["points"] * (2 if case["pol"] == "both" else 1)
    gratings = 2 if case["structure"] == "multilayer" else 1
    c = 145 if case["structure"] in ("lossy", "multilayer") else 52
    out = {"bytes": case["points"] * 16 + solves * 48 * n, "flops": solves * gratings * c * n ** 3}
    if kind == "fields":
        out["bytes"] += 96 * case["depths"] * (n + case["nx"])
        out["flops"] += 48 * case["depths"] * n * (n + case["nx"])
    return out


# ------------------------------------------------------------------------------------------- the structures

def _stack(structure, rng):
    """A 1-D structure; its dimensions come from rng, its make-up does not."""
    if structure == "readme":
        w = rng.uniform(0.25, 0.35) * PERIOD
        return Stack(nI=1.0, nII=1.46, period=PERIOD,
                     layers=[Layer.grating(rng.uniform(0.3, 0.45), [0.0, w, PERIOD], [1.46, 1.0]),
                             Layer.uniform(rng.uniform(0.08, 0.15), 1.96)])
    if structure in ("mirror", "lossy"):
        fill, depth = rng.uniform(0.3, 0.5, 2)
        ridge = complex(1.46, 0.01) if structure == "lossy" else 1.46
        layers = [Layer.grating(depth, [0.0, fill * PERIOD, PERIOD], [ridge, 1.0])]
        for _ in range(10):
            layers += [Layer.uniform(1.053 / (4 * 2.1), 2.1), Layer.uniform(1.053 / (4 * 1.46), 1.46)]
        return Stack(nI=1.0, nII=1.46, period=PERIOD, layers=layers)
    if structure == "contrast":
        w = rng.uniform(0.35, 0.65) * PERIOD
        return Stack(nI=1.0, nII=1.46, period=PERIOD,
                     layers=[Layer.grating(rng.uniform(0.1, 0.5), [0.0, w, PERIOD], [rng.uniform(3.3, 4.0), 1.0])])
    if structure == "multilayer":
        period = rng.uniform(0.5, 1.5)

        def index():
            return complex(rng.uniform(1.2, 2.5), rng.uniform(0.005, 0.05))

        def grating(segments, **how):
            inner = period * (np.arange(1, segments) + rng.uniform(-0.3, 0.3, segments - 1)) / segments
            return Layer.grating(rng.uniform(0.05, 0.3), [0.0, *inner, period], [index() for _ in range(segments)], **how)

        def film():
            return Layer.uniform(rng.uniform(0.05, 0.3), index())
        return Stack(nI=1.0, nII=1.46, period=period,
                     layers=[film(), grating(3), film(), film(), grating(2, fourier_method=1, fft_samples=1024), film()])
    assert structure == "conical", structure

    def lossless(segments):
        inner = PERIOD * (np.arange(1, segments) + rng.uniform(-0.3, 0.3, segments - 1)) / segments
        return Layer.grating(rng.uniform(0.05, 0.3), [0.0, *inner, PERIOD], list(rng.uniform(1.0, 2.5, segments)))
    return Stack(nI=1.0, nII=1.46, period=PERIOD,
                 layers=[lossless(2), lossless(3),
                         Layer.uniform(rng.uniform(0.05, 0.3), complex(1.5 + rng.uniform(0, 0.5), rng.uniform(0, 0.1))),
                         lossless(4)])


def _stack2d(structure, rng):
    P = rng.uniform(0.6, 1.0)

    def row(x0, x1):
        return XProfile2D([0.0, x0, x1, P], [1.0, 2.0, 1.0]) if x1 > x0 else XProfile2D([0.0, P], [1.0])

    def patterned():
        d = rng.uniform(0.05, 0.3)
        if structure == "rect":
            w, h = rng.uniform(0.2, 0.7, 2) * P
            return Layer2D.patterned(d, [0.0, 0.5 * (P - h), 0.5 * (P + h), P],
                                     [row(0, 0), row(0.5 * (P - w), 0.5 * (P + w)), row(0, 0)])
        r, K = rng.uniform(0.15, 0.4) * P, 16
        y = [P * k / K for k in range(K + 1)]
        rows = []
        for k in range(K):
            yc = 0.5 * (y[k] + y[k + 1]) - 0.5 * P
            half = np.sqrt(max(r * r - yc * yc, 0.0))
            rows.append(row(0.5 * P - half, 0.5 * P + half))
        return Layer2D.patterned(d, y, rows)

    def film():
        return Layer2D.uniform(rng.uniform(0.05, 0.2), rng.uniform(1.3, 2.2))
    return Stack2D(nI=1.0, nII=1.46, Lx=P, Ly=P, layers=[film(), patterned(), film(), patterned(), film()])


def _serve_orders(case):
    return [int(round(m)) for m in np.linspace(case["M"], case["M2"], case["requests"])]


def _inputs(case, seed):
    """What the case is called with, from the seed alone: a dict of plain host values."""
    rng = np.random.default_rng(seed)
    kind, structure = case["kind"], case["structure"]
    if kind == "serve":
        return {"requests": [(_stack(structure, rng), float(rng.uniform(0.6, 1.4)), float(rng.uniform(0.0, 60.0)), M, k % 2)
                             for k, M in enumerate(_serve_orders(case))]}
    P = case["points"]
    if kind == "crossed":
        es, ep = jones_from_angles_2d(rng.uniform(0.0, 90.0))
        return {"stack": _stack2d(structure, rng),
                "points": [(wl, 5.0 + 20.0 * rng.uniform(), 60.0 * rng.uniform(), es, ep) for wl in rng.uniform(0.4, 1.2, P)]}
    stack = _stack(structure, rng)
    if kind == "conical":
        return {"stack": stack, "points": np.stack([rng.uniform(0.5, 1.6, P), rng.uniform(1.0, 60.0, P),
                                                    rng.uniform(1.0, 89.0, P)], axis=1)}
    theta = (50.0, 70.0) if structure in ("mirror", "lossy", "readme") else (0.5, 60.0)
    out = {"stack": stack, "points": np.stack([rng.uniform(0.9, 1.2, P), rng.uniform(*theta, P)], axis=1)}
    if kind == "fields":
        total = sum(L.d for L in stack.layers)
        out["depths"] = np.linspace(-0.5, total + 0.5, case["depths"]) + rng.uniform(0.0, 1e-3)
    return out


# ------------------------------------------------------------------------------------- running the entry points

_KEPT = {}  # one engine and one serving loop per process, as a program keeps them


def _engine():
    from stablercwa_gb300.engine import Engine
    if "engine" not in _KEPT:
        _KEPT["engine"] = Engine(device=0)
    return _KEPT["engine"]


def _server():
    from stablercwa_gb300.engine import Server
    if "server" not in _KEPT:
        _KEPT["server"] = Server(device=0, slots=8)
    return _KEPT["server"]


def prepare(case, seed):
    state = dict(_inputs(case, seed), case=case)
    if case["kind"] == "serve":
        state["server"] = _server()
        return state
    state["engine"] = _engine()
    if case["kind"] == "device":
        n, P = 2 * case["M"] + 1, case["points"]
        rows = 2 * P if case["pol"] == "both" else P
        state["d_points"] = torch.tensor(state["points"], dtype=torch.float64, device="cuda")
        out = {"R": torch.empty((rows, n), dtype=torch.complex128, device="cuda"),
               "T": torch.empty((rows, n), dtype=torch.complex128, device="cuda"),
               "DEr": torch.empty((rows, n), dtype=torch.float64, device="cuda"),
               "DEt": torch.empty((rows, n), dtype=torch.float64, device="cuda"),
               "status": torch.empty(rows, dtype=torch.int32, device="cuda")}
        state["out"], state["addresses"] = out, {k: v.data_ptr() for k, v in out.items()}
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit_1d(*request) for request in state["requests"]]
        done = [srv.wait(t)[1] for t in tickets]
        return {k: np.concatenate([np.atleast_1d(r[k]) for r in done])
                for k in ("R", "T", "DEr", "DEt", "status", "eig_info", "n_eig", "n_dense_solve")}
    eng = state["engine"]
    if kind == "device":
        eng.solve1d_device(state["stack"], state["d_points"].data_ptr(), case["points"], case["M"], POLS[case["pol"]],
                           state["addresses"])
        return state["out"]
    if kind == "solve":
        return eng.solve1d_arrays(state["stack"], state["points"], case["M"], POLS[case["pol"]])
    if kind == "conical":
        return eng.solve_conical_arrays(state["stack"], state["points"], case["M"])
    if kind == "crossed":
        return eng.solve2d_arrays(state["stack"], state["points"], case["M1"], case["M2"])
    arrays, fields = eng.solve1d_fields(state["stack"], state["points"], case["M"], POLS[case["pol"]], state["depths"])
    wl, theta = state["points"][0]
    kx = 2 * np.pi / wl * _transverse(state["stack"], wl, theta, case["M"])
    return {**arrays, "fields": fields, "map": eng.field_map(fields[0], kx, state["stack"].period, nx=case["nx"])}


def _transverse(stack, wavelength, theta_deg, M):
    """kx / k0 of every order."""
    return stack.nI * np.sin(np.deg2rad(theta_deg)) - np.arange(-M, M + 1) * wavelength / stack.period


# ----------------------------------------------------------------------------------- the same solves in numpy

EXACT_SECONDS = 14.0  # estimated time of the numpy restatement beyond which a case goes without


def exact(case, seed):
    given, kind = _inputs(case, seed), case["kind"]
    if kind == "serve":
        rows = [_solve1d(s, wl, th, M, pol) for s, wl, th, M, pol in given["requests"]]
        return {k: np.concatenate([r[k] for r in rows]) for k in ("R", "T", "DEr", "DEt")}
    if kind == "crossed":
        n = 2 * (2 * case["M1"] + 1) * (2 * case["M2"] + 1)
        if case["points"] * 0.4 * (n / 121) ** 3 > EXACT_SECONDS:
            return None
        return _stacked([_solve2d(given["stack"], p, case["M1"], case["M2"]) for p in given["points"]])
    n = 2 * case["M"] + 1
    if kind == "conical":
        if case["points"] * 0.6 * (2 * n / 121) ** 3 > EXACT_SECONDS:
            return None
        return _stacked([_solve_conical(given["stack"], p, case["M"]) for p in given["points"]])
    pols = (0, 1) if case["pol"] == "both" else (POLS[case["pol"]],)
    per = 0.15 if case["structure"] == "multilayer" else 0.08 if case["structure"] == "lossy" else 0.025
    if len(pols) * case["points"] * per * (n / 121) ** 3 > EXACT_SECONDS:
        return None
    rows = [_solve1d(given["stack"], wl, th, case["M"], pol, given.get("depths")) for pol in pols for wl, th in given["points"]]
    out = _stacked(rows)
    if kind == "fields":
        wl, theta = given["points"][0]
        x = np.arange(case["nx"]) / case["nx"] * given["stack"].period
        wave = np.exp(-1j * 2 * np.pi / wl * np.outer(_transverse(given["stack"], wl, theta, case["M"]), x))
        out["map"] = np.einsum("cjz,jx->czx", out["fields"][0], wave)
    return out


def _stacked(rows):
    return {k: np.stack([r[k] for r in rows]) for k in rows[0]}


def _coefficients(edges, values, period, h):
    """(1 / P) integral of a piecewise-constant profile times exp(-2 pi i h x / P), for an array h."""
    edges, values, h = np.asarray(edges), np.asarray(values), np.asarray(h)
    w = np.exp(-2j * np.pi * np.multiply.outer(h, edges) / period)
    hs = np.where(h == 0, 1, h)[..., None]
    seg = np.where((h == 0)[..., None], np.diff(edges) / period, np.diff(w, axis=-1) / (-2j * np.pi * hs))
    return seg @ values


def _sampled_coefficients(edges, values, period, h, samples):
    """The same from N equidistant samples (the sampled-profile option of a layer)."""
    x = edges[0] + (np.arange(samples) + 0.5) / samples * period
    c = np.fft.fft(np.asarray(values)[np.searchsorted(edges, x, side="right") - 1]) / samples
    return c[h % samples] * np.exp(-2j * np.pi * h * (0.5 / samples + edges[0] / period))


def _toeplitz(layer, values, period, M):
    d = np.arange(2 * M + 1)
    h = d[:, None] - d[None, :]
    if layer.fourier_method == 1:
        return _sampled_coefficients(np.asarray(layer.edges), values, period, h, layer.fft_samples)
    return _coefficients(layer.edges, values, period, h)


def _branch(q):
    """Re q >= 0, and Im q < 0 for a propagating mode."""
    q = np.where(q.real < 0, -q, q)
    return np.where((q.real < 1e-10) & (q.imag > 0), -q, q)


def _times(a, b):
    """a b, where a 1-D array is a diagonal matrix."""
    if a.ndim == 1:
        return a * b if b.ndim == 1 else a[:, None] * b
    return a * b[None, :] if b.ndim == 1 else a @ b


def _inverse_times(a, b):
    if a.ndim == 1:
        return _times(1.0 / a, b)
    return np.linalg.solve(a, np.diag(b) if b.ndim == 1 else b)


def _plus(a, b):
    return a + b if a.ndim == b.ndim else (np.diag(a) if a.ndim == 1 else a) + (np.diag(b) if b.ndim == 1 else b)


def _cascade(regions, depths, k0, incident):
    """Reflected and transmitted amplitudes of a stack of regions (W, V, q): tangential E = W (d + u), H = V (d - u)
    with d ~ exp(-k0 q z) the down-going amplitudes. Also, per layer, the down-going amplitudes at its top and the
    up-going ones at its bottom. incident: (n, columns)."""
    r = np.zeros_like(regions[-1][2])
    below, match = [None] * len(depths), [None] * (len(regions) - 1)
    for j in range(len(regions) - 2, -1, -1):
        (W1, V1, _), (W2, V2, _) = regions[j], regions[j + 1]
        one = np.ones(len(r))
        e, h = _inverse_times(W1, _times(W2, _plus(one, r))), _inverse_times(V1, _times(V2, _plus(one, -r)))
        p, m = 0.5 * _plus(e, h), 0.5 * _plus(e, -h)  # the down- and up-going waves above, per d below
        match[j] = p
        r = m / p if p.ndim == 1 else np.linalg.solve(p.T, m.T).T
        if j > 0:
            below_top = np.exp(-k0 * regions[j][2] * depths[j - 1])
            below[j - 1] = r
            r = _times(_times(below_top, r), below_top)
    R = _times(r, incident) if r.ndim == 2 else r[:, None] * incident
    d, top, bottom = incident, [], []
    for j, p in enumerate(match):
        d = d / p[:, None] if p.ndim == 1 else np.linalg.solve(p, d)
        if j < len(depths):
            top.append(d)
            d = np.exp(-k0 * regions[j + 1][2] * depths[j])[:, None] * d
            bottom.append(_times(below[j], d) if below[j].ndim == 2 else below[j][:, None] * d)
    return R, d, top, bottom


def _modes1d(layer, kx, period, pol, M):
    """(W, V, q, Ez operator) of one layer or medium; Hermitian problems through their Hermitian form."""
    if layer.homogeneous:
        n2 = complex(layer.n) ** 2
        q = _branch(-1j * np.sqrt(n2 - kx ** 2 + 0j))
        return np.ones(len(kx), complex), q / n2 if pol else q, q, np.full(len(kx), 1.0 / n2)
    eps = np.asarray(layer.n_values) ** 2
    lossless = not np.any(eps.imag)
    E = _toeplitz(layer, eps, period, M)
    if not pol:
        A = np.diag(kx ** 2) - E
        lam, W = np.linalg.eigh(A) if lossless else np.linalg.eig(A)
        q = _branch(np.sqrt(lam + 0j))
        return W, W * q, q, None
    C, Ei = _toeplitz(layer, 1.0 / eps, period, M), np.linalg.inv(E)
    B = kx[:, None] * Ei * kx - np.eye(len(kx))
    if lossless:
        L = np.linalg.cholesky(C)
        Y = np.linalg.solve(L, np.linalg.solve(L, 0.5 * (B + B.conj().T)).conj().T)
        lam, Z = np.linalg.eigh(0.5 * (Y + Y.conj().T))
        W = np.linalg.solve(L.conj().T, Z)
    else:
        lam, W = np.linalg.eig(np.linalg.solve(C, B))
    q = _branch(np.sqrt(lam + 0j))
    return W, (C @ W) * q, q, Ei


def _solve1d(stack, wavelength, theta_deg, M, pol, zs=None):
    k0, n = 2 * np.pi / wavelength, 2 * M + 1
    kx = _transverse(stack, wavelength, theta_deg, M)
    media = [Layer.uniform(0.0, stack.nI), *stack.layers, Layer.uniform(0.0, stack.nII)]
    modes = [_modes1d(L, kx, stack.period, pol, M) for L in media]
    depths = [L.d for L in stack.layers]
    R, T, top, bottom = (v for v in _cascade([m[:3] for m in modes], depths, k0, np.eye(n, 1, -M, dtype=complex)))
    R, T = R[:, 0], T[:, 0]
    kI, kII = 1j * modes[0][2], 1j * modes[-1][2]
    if pol:
        kI, kII = kI / complex(stack.nI) ** 2, kII / complex(stack.nII) ** 2
    out = {"R": R, "T": T, "DEr": np.abs(R) ** 2 * (kI / kI[M]).real, "DEt": np.abs(T) ** 2 * (kII / kI[M]).real}
    if zs is None:
        return out
    tops = np.concatenate([[0.0], np.cumsum(depths)])
    F = np.zeros((6, n, len(zs)), complex)
    for i, z in enumerate(zs):
        if z < 0:
            W, V, q, ez = modes[0]
            down, up = np.eye(n, 1, -M, dtype=complex)[:, 0] * np.exp(-k0 * q * z), R * np.exp(k0 * q * z)
        elif z > tops[-1]:
            W, V, q, ez = modes[-1]
            down, up = T * np.exp(-k0 * q * (z - tops[-1])), np.zeros(n)
        else:
            j = int(np.flatnonzero(z <= tops[1:] + 1e-12)[0])
            W, V, q, ez = modes[j + 1]
            zl = min(max(z - tops[j], 0.0), depths[j])
            down, up = np.exp(-k0 * q * zl) * top[j][:, 0], np.exp(-k0 * q * (depths[j] - zl)) * bottom[j][:, 0]
        S, U = (_times(W, down + up) if W.ndim == 1 else W @ (down + up)), (V * (up - down) if V.ndim == 1 else V @ (up - down))
        if pol:
            F[0, :, i], F[2, :, i], F[4, :, i] = -1j * U, ez * (kx * S) if ez.ndim == 1 else ez @ (kx * S), S
        else:
            F[1, :, i], F[3, :, i], F[5, :, i] = S, 1j * U, -kx * S
    return {**out, "fields": F}


def _medium2d(n, Kx, Ky):
    """(W, V, q) of a homogeneous region in Cartesian components, and kz / k0."""
    n2 = complex(n) ** 2
    kz = np.sqrt(n2 - Kx ** 2 - Ky ** 2 + 0j)
    kz = np.where(kz.imag < 0, -kz, kz)
    q = _branch(-1j * kz)
    V = np.block([[np.diag(Kx * Ky / q), np.diag((n2 - Kx ** 2) / q)], [np.diag((Ky ** 2 - n2) / q), np.diag(-Kx * Ky / q)]])
    return (np.ones(2 * len(Kx), complex), V, np.concatenate([q, q])), kz


def _patterned2d(Ei, Cx, Cy, Kx, Ky):
    """(W, V, q) of a structured layer: eigenpairs of P Q with the two inverse-rule operators."""
    one, x, y = np.eye(len(Kx)), Kx[:, None], Ky[:, None]
    P = np.block([[x * Ei * Ky, one - x * Ei * Kx], [y * Ei * Ky - one, -(y * Ei * Kx)]])
    Q = np.block([[np.diag(Kx * Ky), Cy - np.diag(Kx ** 2)], [np.diag(Ky ** 2) - Cx, np.diag(-Kx * Ky)]])
    lam, W = np.linalg.eig(P @ Q)
    q = _branch(np.sqrt(lam))
    return W, (Q @ W) / q, q


def _solve_conical(stack, point, M):
    wavelength, theta, phi = point[0], np.deg2rad(point[1]), np.deg2rad(point[2])
    k0, n = 2 * np.pi / wavelength, 2 * M + 1
    kx = stack.nI * np.sin(theta) * np.cos(phi) - np.arange(-M, M + 1) * wavelength / stack.period
    ky = stack.nI * np.sin(theta) * np.sin(phi)
    Ky = np.full(n, ky)
    first, kzI = _medium2d(stack.nI, kx, Ky)
    last, kzII = _medium2d(stack.nII, kx, Ky)
    regions = [first]
    for L in stack.layers:
        if L.homogeneous:
            regions.append(_medium2d(L.n, kx, Ky)[0])
            continue
        eps = np.asarray(L.n_values) ** 2
        E, C = _toeplitz(L, eps, stack.period, M), _toeplitz(L, 1.0 / eps, stack.period, M)
        regions.append(_patterned2d(np.linalg.inv(E), np.linalg.inv(C), E, kx, Ky))
    kt = np.hypot(kx, ky)
    cs, sn = kx / kt, ky / kt
    incident = np.zeros((2 * n, 2), complex)  # unit s and unit p waves of order 0
    incident[M], incident[n + M] = (-sn[M], cs[M] * np.cos(theta)), (cs[M], sn[M] * np.cos(theta))
    R, T, _, _ = _cascade([*regions, last], [L.d for L in stack.layers], k0, incident)

    def jones(F, kz, index, sign):  # the orders' s and p amplitudes of both incident waves: ss, sp, ps, pp
        s = -sn[:, None] * F[:n] + cs[:, None] * F[n:]
        p = sign * (cs[:, None] * F[:n] + sn[:, None] * F[n:]) * (complex(index) / kz)[:, None]
        return np.concatenate([s, p], axis=1)
    Jr, Jt = jones(R, kzI, stack.nI, -1.0), jones(T, kzII, stack.nII, 1.0)
    unit = stack.nI * np.cos(theta)
    fr, ft = kzI.real / unit, kzII.real / unit
    return {"Jr": Jr, "Jt": Jt, "DEr": fr[:, None] * np.abs(Jr) ** 2, "DEt": ft[:, None] * np.abs(Jt) ** 2,
            "kx": kx, "ky": ky, "flux_r": fr, "flux_t": ft}


def _operators2d(layer, Lx, Ly, M1, M2):
    """(Eps, Cx, Cy): the plain convolution matrix, and Li's rules with the inverse taken along x or along y."""
    n1, n2 = 2 * M1 + 1, 2 * M2 + 1
    dx, dy = np.subtract.outer(np.arange(n1), np.arange(n1)), np.subtract.outer(np.arange(n2), np.arange(n2))
    ye, rows = np.asarray(layer.y_edges), layer.x_profiles
    cuts = np.unique(np.concatenate([np.asarray(p.edges) for p in rows]))
    K = len(rows)
    wy = np.stack([_coefficients(ye, np.eye(K)[k], Ly, dy) for k in range(K)])
    wx = np.stack([_coefficients(cuts, np.eye(len(cuts) - 1)[k], Lx, dx) for k in range(len(cuts) - 1)])
    eps = [np.asarray(p.n_values, complex) ** 2 for p in rows]
    plain = np.stack([_coefficients(p.edges, e, Lx, dx) for p, e in zip(rows, eps)])
    inv_x = np.stack([np.linalg.inv(_coefficients(p.edges, 1.0 / e, Lx, dx)) for p, e in zip(rows, eps)])
    mid = 0.5 * (cuts[1:] + cuts[:-1])
    at = np.stack([e[np.searchsorted(p.edges, mid, side="right") - 1] for p, e in zip(rows, eps)])  # strip, column
    inv_y = np.stack([np.linalg.inv(_coefficients(ye, 1.0 / at[:, c], Ly, dy)) for c in range(len(mid))])
    N = n1 * n2

    def joined(x, y):
        return np.einsum("kac,kbd->abcd", x, y).reshape(N, N)
    return joined(plain, wy), joined(inv_x, wy), joined(wx, inv_y)


def _solve2d(stack, point, M1, M2):
    wavelength, theta, phi, Es, Ep = point[0], np.deg2rad(point[1]), np.deg2rad(point[2]), point[3], point[4]
    k0, nI = 2 * np.pi / wavelength, stack.nI
    m, k = np.repeat(np.arange(-M1, M1 + 1), 2 * M2 + 1), np.tile(np.arange(-M2, M2 + 1), 2 * M1 + 1)
    Kx = nI * np.sin(theta) * np.cos(phi) - m * wavelength / stack.Lx
    Ky = nI * np.sin(theta) * np.sin(phi) - k * wavelength / stack.Ly
    N = len(Kx)
    i0 = N // 2
    first, kzI = _medium2d(nI, Kx, Ky)
    last, kzII = _medium2d(stack.nII, Kx, Ky)
    regions = [first]
    for L in stack.layers:
        if L.homogeneous:
            regions.append(_medium2d(L.n, Kx, Ky)[0])
        else:
            eps, cx, cy = _operators2d(L, stack.Lx, stack.Ly, M1, M2)
            regions.append(_patterned2d(np.linalg.inv(eps), cx, cy, Kx, Ky))
    incident = np.zeros((2 * N, 1), complex)
    incident[i0] = -Es * np.sin(phi) + Ep * np.cos(theta) * np.cos(phi)
    incident[N + i0] = Es * np.cos(phi) + Ep * np.cos(theta) * np.sin(phi)
    R, T, _, _ = _cascade([*regions, last], [L.d for L in stack.layers], k0, incident)
    out = {"Kx": Kx, "Ky": Ky, "kzI": kzI, "kzII": kzII}
    kt = np.hypot(Kx, Ky)
    for F, kz, n, sign, e, de, s, p in ((R[:, 0], kzI, nI, -1.0, "r", "DEr", "Rs", "Rp"),
                                        (T[:, 0], kzII, stack.nII, 1.0, "t", "DEt", "Ts", "Tp")):
        Ex, Ey, on = F[:N], F[N:], kz.real > 1e-12
        Ez = np.where(on, -sign * (Kx * Ex + Ky * Ey) / kz, 0.0)
        out.update({"Ex_" + e: Ex, "Ey_" + e: Ey, "Ez_" + e: Ez})
        out[de] = np.where(on, kz.real * (np.abs(Ex) ** 2 + np.abs(Ey) ** 2 + np.abs(Ez) ** 2) / (nI * np.cos(theta)), 0.0)
        out[s] = (-Ky * Ex + Kx * Ey) / kt
        out[p] = sign * (Kx * Ex + Ky * Ey) / (kt * kz / complex(n))
    return out
