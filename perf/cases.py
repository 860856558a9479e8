"""The calls that a user of this framework spends GPU time in, as measurable cases.

Three kinds:
  call    `TimeEvolutionMexCUDA` on host structs, in place: the drop-in entry
          point, with the upload, the tables and the download in the call;
  prop    `Propagator.propagate` on a handle that the program keeps, then the
          wavepackets, P(E), norms and (if asked) the energies of those steps;
  fit, surface, bkmp2
          the set-up of a potential: training the learned surface, evaluating
          it on a Jacobi grid, evaluating the BKMP2 surface on one.

Inputs are built here (extended-LEPS surfaces, Gaussian packets on DVR
diatomic states, quadratic absorbers) with torch and numpy in FP64; the seed
moves the packet, the energies, the barrier and the absorbers.  The packets
start near the interaction region and the dividing surface lies close to it, so
that a stretch of a hundred steps has what most of a long run has: flux through
the surface.  A complex64 propagation holds complex64 values, so its outputs
are returned in that precision.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "quantum-dynamics_b200"))

EV = 1.0 / 27.211386245988
AMU = 1822.888486209
BOHR = 1.0 / 0.529177210903                     # bohr per angstrom
# (J, K) blocks of a centrifugal-sudden batch, taken from the front
BLOCKS = [(J, K) for J in (0, 5, 10, 15, 20, 25, 30) for K in range(min(J, 4) + 1)]
TRAIN = dict(lr=2e-3, lr_end=1e-5)


# ---- the cases -----------------------------------------------------------------------

def _prop(name, system, n1, n2, nth, steps, f64, kind="prop", runs=1, m=None, points=11,
          ne=241, uniform=True, every=0):
    return dict(name=name, kind=kind, system=system, n1=n1, n2=n2, nth=nth,
                m=nth - 1 if m is None else m, steps=steps, f64=f64, runs=runs, points=points,
                ne=ne, uniform=uniform, every=every)


def listed():
    return [
        # the drop-in call on the smallest grid of the configurations, in its default
        # arithmetic: latency, launches and set-up
        _prop("call_h3_64x64x40_f64", "h+h2", 64, 64, 40, 20, True, kind="call", m=38),
        # the same grid kept on the device in complex64, a stretch between two looks at P(E)
        _prop("h3_64x64x40_f32", "h+h2", 64, 64, 40, 120, False, m=38),
        # F + H2, J = 0: the ordinary single propagation, in both arithmetics; the FP64 one
        # with the energies of every 20th step
        _prop("fh2_128x128x64_f32", "f+h2", 128, 128, 64, 200, False),
        _prop("fh2_128x128x64_f64", "f+h2", 128, 128, 64, 60, True, every=20),
        # batches of centrifugal-sudden blocks (bases of uneven size)
        _prop("cs24_128x96x64_f32", "f+h2", 128, 96, 64, 100, False, runs=24),
        _prop("cs4_256x192x128_f32", "f+h2", 256, 192, 128, 100, False, runs=4),
        # the large grid through the drop-in call in FP64
        _prop("call_256x192x128_f64", "f+h2", 256, 192, 128, 30, True, kind="call"),
        # grids that no configuration names: other factors of 2, 3 and 5, an odd number of
        # angles, a truncated basis, short stencils, energies off a uniform grid
        _prop("odd3_108x90x50_f32", "f+h2", 108, 90, 50, 120, False, runs=3, points=5, ne=150,
              uniform=False),
        _prop("odd_100x54x33_f64", "h+h2", 100, 54, 33, 60, True, m=28, points=3, ne=97,
              uniform=False),
        # the learned surface: minibatch training, and its evaluation on a grid
        dict(name="fit_48k_b4096", kind="fit", n=49152, batch=4096, steps=48),
        dict(name="surface_128x128x64", kind="surface", n1=128, n2=128, nth=64),
        # a real surface on the grid of the H + H2 configuration
        dict(name="bkmp2_64x64x40", kind="bkmp2", n1=64, n2=64, nth=40),
    ]


SMOOTH = [40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192,
          200, 216, 240, 256]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prop"] * 6 + ["call"] * 2 + ["fit", "surface", "bkmp2"])
    if kind == "fit":
        n = _log_int(rng, 4000, 60000)
        return dict(kind=kind, n=n, batch=min(n, _log_int(rng, 256, 8192)), steps=_log_int(rng, 12, 48))
    if kind in ("surface", "bkmp2"):
        n1, n2, nth = rng.randint(32, 180), rng.randint(32, 160), rng.randint(16, 96)
        return dict(kind=kind, n1=n1, n2=n2, nth=nth)
    f64 = rng.random() < 0.5
    # grid points and steps so that the whole costs less than the largest listed case
    n1 = rng.choice(SMOOTH)
    n2 = rng.choice([v for v in SMOOTH if v <= 192])
    nth = _log_int(rng, 24, 128)
    pts = n1 * n2 * nth
    runs = 1
    if kind == "prop" and rng.random() < 0.5:
        runs = max(1, min(24, _log_int(rng, 1, 24), 12_000_000 // pts))
    room = (2.5e8 if f64 else 1.5e9) / (pts * runs)
    steps = min(_log_int(rng, 12, 120) if f64 else _log_int(rng, 80, 150), int(room))
    m = nth - 1 if rng.random() < 0.7 else max(8, nth - 1 - rng.randint(1, nth // 4))
    c = _prop("", rng.choice(["h+h2", "f+h2"]), n1, n2, nth, steps, f64, kind=kind, runs=runs, m=m,
              points=rng.choice([3, 5, 7, 9, 11]), ne=rng.randint(40, 260),
              uniform=rng.random() < 0.7, every=rng.choice([0, 0, 10]) if kind == "prop" else 0)
    del c["name"]
    return c


# ---- inputs --------------------------------------------------------------------------

def _leps(system, g):
    """Three (De, beta, re, sato) of an extended-LEPS surface, in atomic units."""
    hh = (4.7466 * EV, 1.9425 / BOHR, 0.7416 * BOHR)
    fh = (6.12 * EV, 2.2187 / BOHR, 0.9170 * BOHR)
    s = 0.01 * g.uniform(-1.0, 1.0)
    if system == "h+h2":
        return [hh + (0.17 + s,)] * 3
    return [fh + (0.167 + s,), hh + (0.106 + s,), fh + (0.167 + s,)]


def _distances(R, r, x, masses):
    f2 = masses[2] / (masses[1] + masses[2])
    f3 = 1.0 - f2
    r12 = torch.sqrt((f2 * r) ** 2 + R ** 2 - 2 * f2 * r * R * x)
    r13 = torch.sqrt((f3 * r) ** 2 + R ** 2 + 2 * f3 * r * R * x)
    return r12, r.expand_as(r12), r13


def _leps_value(pairs, dist):
    q, j = [], []
    for (de, beta, re, sato), r in zip(pairs, dist):
        pf = 0.5 * de * (1.0 - sato) / (1.0 + sato)
        y = torch.exp(-beta * (r - re))
        q.append(0.5 * (de * (y - 2.0) + pf * (y + 2.0)) * y)
        j.append(0.5 * (de * (y - 2.0) - pf * (y + 2.0)) * y)
    rad = (j[0] * (j[0] - j[1]) + j[1] * (j[1] - j[2]) + j[2] * (j[2] - j[0])).clamp_min(0.0)
    return pairs[1][0] + q[0] + q[1] + q[2] - torch.sqrt(rad)


def _masses(system):
    return np.array([18.9984 if system == "f+h2" else 1.00783, 1.00783, 1.00783]) * AMU


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _potential(R, r, x, masses, pairs, vmax=2.5, rmin=0.4):
    Rt, rt, xt = _dev(R)[None, None, :], _dev(r)[None, :, None], _dev(x)[:, None, None]
    d = _distances(Rt, rt, xt, masses)
    v = _leps_value(pairs, d).clamp_max(vmax)
    ok = (d[0] > rmin) & (d[1] > rmin) & (d[2] > rmin)
    return torch.where(ok, v, torch.full_like(v, vmax))


def _basis(x, K, m):
    """Pbar_{K+l}^K(x_k) / sqrt(l + 1/2), l = 0..m (K = 0: P_l), shape (n, m + 1)."""
    p = np.full(x.size, math.sqrt(0.5))
    for a in range(1, K + 1):
        p = p * math.sqrt((2 * a + 1) / (2 * a)) * np.sqrt(1.0 - x * x)
    v = np.zeros((x.size, m + 1))
    v[:, 0] = p
    if m >= 1:
        v[:, 1] = math.sqrt(2 * K + 3) * x * p
    for l in range(2, m + 1):
        j = K + l
        a = math.sqrt((4 * j * j - 1) / (j * j - K * K))
        b = math.sqrt(((j - 1) ** 2 - K * K) / (4 * (j - 1) ** 2 - 1))
        v[:, l] = a * (x * v[:, l - 1] - b * v[:, l - 2])
    return np.ascontiguousarray(v / np.sqrt(np.arange(m + 1) + 0.5)[None, :])


def _diatom(n, dr, mu, r, v, j0):
    """Levels and vectors of the sinc DVR of the diatom."""
    i = np.arange(1, n + 1, dtype=np.float64)
    d, s = i[:, None] - i[None, :], i[:, None] + i[None, :]
    np.fill_diagonal(d, 1.0)
    h = np.where(np.abs(d) % 2 < 0.5, 1.0, -1.0) * (2.0 / d ** 2 - 2.0 / s ** 2)
    np.fill_diagonal(h, math.pi ** 2 / 3 - 1.0 / (2 * i * i))
    h = h / (2 * mu * dr * dr)
    h[np.diag_indices(n)] += v + j0 * (j0 + 1) / (2 * mu * r ** 2)
    return np.linalg.eigh(h)


def _inputs(case, seed):
    """The shared settings and one dict per run."""
    g = np.random.default_rng([seed, 1])
    masses = _masses(case["system"])
    n1, n2, nth, m = case["n1"], case["n2"], case["nth"], case["m"]
    R, r = np.linspace(0.5, 12.0, n1), np.linspace(0.4, 8.0, n2)
    dR, dr = R[1] - R[0], r[1] - r[0]
    mu_R = masses[0] * (masses[1] + masses[2]) / masses.sum()
    mu_r = masses[1] * masses[2] / (masses[1] + masses[2])
    x, w = np.polynomial.legendre.leggauss(nth)
    pairs = _leps(case["system"], g)
    base = _potential(R, r, x, masses, pairs)
    delta, e0 = g.uniform(0.25, 0.35), g.uniform(0.6, 1.0) * EV
    R0, strength = g.uniform(4.0, 4.6), g.uniform(0.2, 0.4)
    k0 = math.sqrt(2 * mu_R * e0)
    gauss = (math.pi * delta ** 2) ** -0.25 * np.exp(-(R - R0) ** 2 / (2 * delta ** 2) - 1j * k0 * R)
    absorb = lambda q: np.exp(-strength * np.clip((q - (q[-1] - 2.0)) / 2.0, 0.0, None) ** 2)  # noqa: E731
    if case["uniform"]:
        e_coll = np.linspace(0.3, 1.5, case["ne"]) * EV
    else:
        e_coll = np.sort(g.uniform(0.3, 1.5, case["ne"])) * EV
    kE = np.sqrt(2 * mu_R * e_coll)
    eta = math.sqrt(math.pi) * 2 * mu_R * delta / kE * np.exp(-delta ** 2 * (kE - k0) ** 2)
    de, beta, re, _ = pairs[1]
    vd = de * (1.0 - np.exp(-beta * (r - re))) ** 2
    out = dict(R=R, r=r, dR=dR, dr=dr, mu_R=mu_R, mu_r=mu_r, x=x, w=w, dump1=absorb(R),
               dump2=absorb(r), r0=R0, k0=k0, delta=delta, dt=10.0,
               surface=int(math.floor((2.6 - r[0]) / dr + 0.5)), runs=[])
    levels = {}
    for b in range(case["runs"]):
        J, K = BLOCKS[b % len(BLOCKS)] if case["runs"] > 1 else (0, 0)
        j0, v0 = (K + int(g.integers(0, 3)), int(g.integers(0, 2))) if m > 8 else (K, 0)
        if j0 not in levels:
            levels[j0] = _diatom(n2, dr, mu_r, r, vd, j0)
        e, vec = levels[j0]
        phi = vec[:, v0] / math.sqrt(dr) * (1.0 if vec[np.argmax(np.abs(vec[:, v0])), v0] > 0 else -1.0)
        leg = _basis(x, K, m - K)
        ang = leg[:, j0 - K] * math.sqrt(j0 - K + 0.5)
        pot = base if b == 0 else base + _dev((J * (J + 1) - 2 * K * K) / (2 * mu_R * R * R))[None, None, :]
        psi = _dev(ang)[:, None, None] * _dev(phi)[None, :, None] * _dev(gauss)[None, None, :]
        out["runs"].append(dict(J=J, K=K, m=m - K, legendre=leg, pot=pot, psi=psi, e_vj=float(e[v0]),
                                energies=np.ascontiguousarray(e_coll + e[v0]), eta_sq=eta))
    return out


def _geometries(n, seed):
    """n geometries of the F + H2 box with their LEPS energies, all below 8 eV."""
    g = np.random.default_rng([seed, 2])
    masses = _masses("f+h2")
    pairs = _leps("f+h2", g)
    parts, have = [], 0
    while have < n:
        k = 2 * (n - have) + 1024
        d = _distances(_dev(g.uniform(0.5, 12.0, k)), _dev(g.uniform(0.4, 8.0, k)),
                       _dev(g.uniform(-1.0, 1.0, k)), masses)
        v = _leps_value(pairs, d)
        keep = (torch.minimum(torch.minimum(d[0], d[1]), d[2]) > 0.4) & (v < 8 * EV)
        parts.append(torch.stack([d[0], d[1], d[2], v])[:, keep].cpu().numpy())
        have += parts[-1].shape[1]
    a = np.concatenate(parts, axis=1)[:, :n]
    return [np.ascontiguousarray(t) for t in a]


def _weights(seed):
    """He-uniform weights of the surface's network and no biases, in its flat layout."""
    g = np.random.default_rng([seed, 3])
    parts = []
    for k, o in ((3, 64), (64, 64), (64, 64), (64, 64), (64, 1)):
        parts += [g.uniform(-1, 1, o * k) * math.sqrt(6.0 / k), 0.05 * g.standard_normal(o)]
    return np.concatenate(parts).astype(np.float32)


def _norms(geo):
    p = [np.exp(-a / 1.5) for a in geo[:3]]                  # p12, p23, p13
    f = np.stack([p[1], p[0] + p[2], p[0] * p[2]])
    return np.concatenate([f.mean(1), f.std(1), [geo[3].mean(), geo[3].std()]])


def _grid(case):
    return (np.linspace(0.5, 12.0, case["n1"]), np.linspace(0.4, 8.0, case["n2"]),
            np.polynomial.legendre.leggauss(case["nth"])[0])


def _structs(case, seed):
    from qd_b200 import QD_PREC_FP32, QD_PREC_FP64
    from qd_b200.systems import Struct
    q = _inputs(case, seed)
    out = []
    for run in q["runs"]:
        out.append(Struct(
            r1=Struct(n=case["n1"], r=q["R"], dr=q["dR"], mass=q["mu_R"], r0=q["r0"], k0=q["k0"],
                      delta=q["delta"]),
            r2=Struct(n=case["n2"], r=q["r"], dr=q["dr"], mass=q["mu_r"], r0=0.0, k0=0.0, delta=0.0),
            theta=Struct(n=case["nth"], m=run["m"], x=q["x"], w=q["w"], legendre=run["legendre"]),
            pot=run["pot"].cpu().numpy(), psi=run["psi"].cpu().numpy(),
            time=Struct(total_steps=case["steps"], time_step=q["dt"], steps=0),
            options=Struct(wave_to_matlab=None, test_name="",
                           steps_to_copy_psi_from_device_to_host=0,
                           precision=QD_PREC_FP64 if case["f64"] else QD_PREC_FP32),
            dump1=Struct(dump=q["dump1"]), dump2=Struct(dump=q["dump2"]),
            CRP=Struct(eDiatomic=run["e_vj"], n_dividing_surface=q["surface"],
                       n_gradient_points=case["points"], n_energies=case["ne"],
                       energies=run["energies"], eta_sq=run["eta_sq"], CRP=np.zeros(case["ne"]),
                       calculate_CRP=1),
            cs=Struct(J=run["J"], K=run["K"])))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("call", "prop"):
        import qd_b200
        data = _structs(case, seed)
        if kind == "call":
            return dict(case=case, data=data)
        p = qd_b200.Propagator(data)
        if case["every"]:
            p.set_energy_interval(case["every"])
        return dict(case=case, data=data, handle=p)
    if kind == "bkmp2":
        g = np.random.default_rng([seed, 4])
        R, r, x = _grid(case)
        return dict(case=case, R=R + g.uniform(0.0, 0.2), r=r + g.uniform(0.0, 0.1), x=x,
                    masses=_masses("h+h2"))
    from qd_b200.surrogate import Surrogate
    s = Surrogate()
    if kind == "fit":
        s.set_params(_weights(seed))
        return dict(case=case, model=s, geo=_geometries(case["n"], seed))
    s.set_params(_weights(seed), _norms(_geometries(20000, seed)).astype(np.float32))
    R, r, x = _grid(case)
    return dict(case=case, model=s, R=R, r=r, x=x, masses=_masses("f+h2"))


# ---- one pass ------------------------------------------------------------------------

def _as(case, a):
    """An output in the precision the propagation holds it in."""
    t = torch.from_numpy(np.ascontiguousarray(a))
    if case["f64"]:
        return t
    return t.to(torch.complex64 if t.is_complex() else torch.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        from qd_b200 import TimeEvolutionMexCUDA
        data = state["data"]
        TimeEvolutionMexCUDA(data)
        return {"psi": [_as(case, d.psi) for d in data], "crp": [_as(case, d.CRP.CRP) for d in data]}
    if kind == "prop":
        p, n = state["handle"], len(state["data"])
        p.propagate(case["steps"])
        p.download()
        out = {"psi": [_as(case, d.psi) for d in state["data"]],
               "crp": _as(case, np.stack([d.CRP.CRP for d in state["data"]])),
               "norms": _as(case, np.stack([p.norms(case["steps"], k) for k in range(n)]))}
        if case["every"]:
            k = case["steps"] // case["every"]
            out["energies"] = _as(case, np.stack([p.energy_log(b, cap=k)[:, 1:] for b in range(n)]))
        return out
    if kind == "fit":
        s, (r12, r23, r13, v) = state["model"], state["geo"]
        loss = s.fit(r12, r23, r13, v, steps=case["steps"], batch=case["batch"], **TRAIN)
        return {"weights": s.params()[0], "loss": np.float32(loss)}
    if kind == "surface":
        return state["model"].potential(state["R"], state["r"], state["x"],
                                        state["masses"]).astype(np.float32)
    from qd_b200.timeevolution import potential_bkmp2_gpu
    return potential_bkmp2_gpu(state["R"], state["r"], state["x"], state["masses"])


# ---- what a pass cannot do without ---------------------------------------------------

def work(case):
    kind = case["kind"]
    net = 3 * 64 + 3 * 64 * 64 + 64
    if kind == "fit":
        return {"bytes": 32 * case["n"] + 4 * 2 * net,
                "flops": 6 * net * min(case["batch"], case["n"]) * case["steps"]}
    if kind in ("surface", "bkmp2"):
        pts = case["n1"] * case["n2"] * case["nth"]
        return {"bytes": 8 * pts, "flops": (2 * net if kind == "surface" else 600) * pts}
    # a step couples all angles of a grid column, then all columns of an order: two sweeps
    # that read and write the state, one of them reading the potential's phase
    n12, c = case["n1"] * case["n2"], 16 if case["f64"] else 8
    pts, nl = n12 * case["nth"] * case["runs"], case["m"] + 1
    per_col = 8 * case["nth"] * nl                          # both Legendre transforms
    per_slice = 2 * 5 * n12 * math.log2(n12) + 18 * n12     # both DFTs, three phases
    return {"bytes": case["steps"] * pts * 5 * c + pts * 40,
            "flops": case["steps"] * case["runs"] * (n12 * per_col + nl * per_slice)}


# ---- the same in 64 bits -------------------------------------------------------------

def _stencil(points):
    h = (points - 1) // 2
    a = np.array([[float(k) ** (2 * i + 1) for k in range(1, h + 1)] for i in range(h)])
    b = np.zeros(h)
    b[0] = 0.5
    return np.linalg.solve(a, b)


def _exact_run(case, q, run):
    n1, n2, nth, steps, dt = case["n1"], case["n2"], case["nth"], case["steps"], q["dt"]
    nl, z = run["m"] + 1, torch.complex128
    L, w, l = _dev(run["legendre"]), _dev(q["w"]), np.arange(nl)
    back = L.to(z)                                                          # (nth, nl)
    forw = (L * w[:, None] * _dev(l + 0.5)[None, :]).T.contiguous().to(z)     # (nl, nth)
    i1, i2 = 1 / (2 * q["mu_R"] * q["R"] ** 2), 1 / (2 * q["mu_r"] * q["r"] ** 2)
    inertia = _dev(i1)[None, :] + _dev(i2)[:, None]
    jj = _dev((l + run["K"]) * (l + run["K"] + 1.0))
    p1 = 2 * math.pi * np.fft.fftfreq(n1, q["dR"])
    p2 = 2 * math.pi * np.fft.fftfreq(n2, q["dr"])
    T = _dev(p1 ** 2 / (2 * q["mu_R"]))[None, :] + _dev(p2 ** 2 / (2 * q["mu_r"]))[:, None]
    rot = torch.exp(-0.5j * dt * jj[:, None, None] * inertia[None])
    kin = torch.exp(-1j * dt * T)
    V = run["pot"]
    phase = torch.exp(-1j * dt * V)
    dump = _dev(q["dump1"])[None, :] * _dev(q["dump2"])[:, None]
    coef, s = _stencil(case["points"]), q["surface"] - 1
    E = _dev(run["energies"])
    area = q["dR"] * q["dr"]
    psi = run["psi"] * torch.sqrt(phase)
    norms, energies, ps, dps = [], [], [], []
    wk = w[:, None, None]
    lw = _dev(1.0 / (l + 0.5))[:, None, None]
    for t in range(1, steps + 1):
        if t > 1:
            psi = psi * phase
        a = (forw @ psi.reshape(nth, -1)).reshape(nl, n2, n1) * rot
        f = torch.fft.fft2(a)
        log = case["every"] and t % case["every"] == 0
        if log:
            ek = ((f.real ** 2 + f.imag ** 2) * T[None] * lw).sum() / (n1 * n2) * area
        a = torch.fft.ifft2(f * kin[None]) * rot
        if log:
            er = ((a.real ** 2 + a.imag ** 2) * inertia[None] * jj[:, None, None] * lw).sum() * area
        psi = (back @ a.reshape(nl, -1)).reshape(nth, n2, n1)
        if log:
            ep = ((psi.real ** 2 + psi.imag ** 2) * V * wk).sum() * area
            energies.append(torch.stack([ek, er, ep, ek + er + ep]))
        psi = psi * dump[None]
        norms.append(((psi.real ** 2 + psi.imag ** 2) * wk).sum() * area)
        g = sum(c * (psi[:, s + k] - psi[:, s - k]) for k, c in enumerate(coef, 1)) / q["dr"]
        ps.append(psi[:, s].clone())
        dps.append(g)
    t = torch.arange(1, steps + 1, device="cuda", dtype=torch.float64) * dt
    et = dt * torch.exp(1j * E[:, None] * t[None, :])
    phi = (et @ torch.stack(ps).reshape(steps, -1)).reshape(-1, nth, n1)
    dphi = (et @ torch.stack(dps).reshape(steps, -1)).reshape(-1, nth, n1)
    flux = ((phi.conj() * dphi).imag * wk.reshape(1, -1, 1)).sum((1, 2))
    crp = flux / _dev(run["eta_sq"]) * q["dR"] / q["mu_r"]
    return psi, crp, torch.stack(norms), torch.stack(energies) if energies else None


def _net(p, f):
    """The surface's network on standardised features f (n, 3)."""
    o, a = 0, f
    for k in (3, 64, 64, 64):
        W, b = p[o:o + 64 * k].reshape(64, k), p[o + 64 * k:o + 64 * k + 64]
        a = torch.nn.functional.silu(a @ W.T + b)
        o += 64 * k + 64
    return a @ p[o:o + 64] + p[o + 64]


def _features(dist, nm):
    p = [torch.exp(-d / 1.5) for d in dist]
    f = torch.stack([p[1], p[0] + p[2], p[0] * p[2]], dim=-1)
    return (f - nm[:3]) / nm[3:6]


def _exact_fit(case, seed):
    geo = _geometries(case["n"], seed)
    nm = _dev(_norms(geo))
    f, tgt = _features([_dev(a) for a in geo[:3]], nm), (_dev(geo[3]) - nm[6]) / nm[7]
    p = _dev(_weights(seed).astype(np.float64)).requires_grad_(True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    n, B, steps = case["n"], min(case["batch"], case["n"]), case["steps"]
    lr = TRAIN["lr"]
    decay = (TRAIN["lr_end"] / lr) ** (1.0 / (steps - 1)) if steps > 1 else 1.0
    s0, total, seen, loss = 0, 0.0, 0, 0.0
    for t in range(1, steps + 1):
        e = min(n, s0 + B)
        sq = (_net(p, f[s0:e]) - tgt[s0:e]).square().sum()
        (g,) = torch.autograd.grad(sq / (e - s0), p)
        total, seen = total + float(sq.detach()), seen + e - s0
        with torch.no_grad():
            m.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).add_(g * g, alpha=0.001)
            p -= lr * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
        lr *= decay
        s0 = e
        if s0 >= n:
            loss, total, seen, s0 = total / seen, 0.0, 0, 0
    return {"weights": p.detach(), "loss": total / seen if seen else loss}


def exact(case, seed):
    kind = case["kind"]
    if kind == "bkmp2":
        return None
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "surface":
        R, r, x = _grid(case)
        d = _distances(_dev(R)[None, None, :], _dev(r)[None, :, None], _dev(x)[:, None, None],
                       _masses("f+h2"))
        nm = _dev(_norms(_geometries(20000, seed)).astype(np.float32).astype(np.float64))
        p = _dev(_weights(seed).astype(np.float64))
        v = torch.stack([_net(p, _features([a[k] for a in d], nm)) for k in range(x.size)])
        v = (v * nm[7] + nm[6]).clamp_max(2.5)
        ok = (d[0] > 0.4) & (d[1] > 0.4) & (d[2] > 0.4)
        return torch.where(ok, v, torch.full_like(v, 2.5))
    q = _inputs(case, seed)
    psi, crp, norms, energies = [], [], [], []
    for b in q["runs"]:
        a = _exact_run(case, q, b)
        psi.append(a[0].cpu())
        crp.append(a[1])
        norms.append(a[2])
        energies.append(a[3])
    if kind == "call":
        return {"psi": psi, "crp": crp}
    out = {"psi": psi, "crp": torch.stack(crp), "norms": torch.stack(norms)}
    if case["every"] and energies[0] is not None:
        out["energies"] = torch.stack(energies)
    return out
