"""What is timed: the calls that programs using this framework make, at the sizes they make them.

A vortex-filament program holds its filaments either on the host (a list of node arrays, or one flat
array with offsets) or on the device, keeps one cache per set of Biot-Savart parameters, and asks for
the velocity (and sometimes the streamfunction) on all nodes, or for whole RK4 steps, of one system
or of an ensemble.  ``listed`` names twelve such uses; ``draw`` takes others from the same ranges.
``exact`` restates the same quantity in torch in 64 bits: quintic splines by a dense solve, every pair
within the cut-off, and the NUFFT sums with its window, grid and truncation.

Case keys: ``api`` (lists / flat / device / step / ensemble), ``rings`` of about ``nodes`` nodes each
(``ragged``: of different sizes), ``lines`` unclosed periodic lines, ``systems`` of an ensemble;
``split`` (gaussian / kaiser / open), ``beta``, the cut-off L / ``cut``, ``Ns`` (0: from the
splitting's own rule), ``sigma``, ``m``; ``fields`` (1 velocity, 2 streamfunction, 3 both),
``spectra`` (diagnostics of the same evaluation), ``precision``, ``tall`` (period 2 L in z).
"""

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

L = 2 * math.pi
GAMMA, CORE, DELTA, NQUAD = 1.0, 1e-8, 0.25, 3

BASE = {"api": "lists", "rings": 1, "nodes": 200, "ragged": False, "lines": 0, "systems": 1, "split": "gaussian",
        "beta": 3.5, "cut": 8.0, "Ns": 0, "sigma": 1.5, "m": 4, "fields": 1, "spectra": False,
        "precision": "fp64", "tall": False}


def _case(name=None, **kw):
    c = dict(BASE, **kw)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one vortex ring, the call of a first script or of a parameter study: latency only
        _case("ring64_lists_fp64", nodes=64, cut=4.0, Ns=32),
        # isolated vortices without periodicity (ring collisions, knots): the all-pairs sum
        _case("open_4k_lists_fp64", rings=18, nodes=223, ragged=True, split="open", fields=3),
        # lines through the box and rings of all sizes, parameters from the accuracy rule (so an FFT
        # size that is not a multiple of 16), velocity and streamfunction
        _case("lines_rings_6k_lists_fp64", rings=33, nodes=167, ragged=True, lines=4, cut=7.3, beta=3.6, fields=3,
              tall=True),
        # an output step of a simulation: both fields and the spectra
        _case("tangle20k_lists_fp64_spectra", rings=100, Ns=128, fields=3, spectra=True),
        # the right-hand side of a user's own device-side integrator
        _case("tangle20k_device_mixed", api="device", rings=100, Ns=128, precision="mixed"),
        # a small simulation: one RK4 step of a system of a few rings
        _case("step_1k_mixed", api="step", rings=7, cut=4.0, Ns=32, precision="mixed"),
        # statistics over many small systems, one launch per step
        _case("ensemble_24x1k_mixed", api="ensemble", systems=24, rings=7, cut=4.0, Ns=32, precision="mixed"),
        # a production run: one RK4 step of a dense tangle, and the same in FP64 at half the size
        _case("step_200k_mixed", api="step", rings=1000, cut=32.57, Ns=256, precision="mixed"),
        _case("step_100k_fp64", api="step", rings=500, cut=24.17, Ns=190),
        # the largest tangle at the parameters the learned choice takes for 1e-5, on the device and
        # through host arrays
        _case("tangle1m_tuned_device_mixed", api="device", rings=5000, split="kaiser", beta=12.44, cut=45.0, Ns=192,
              m=3, precision="mixed"),
        _case("tangle1m_tuned_flat_mixed", api="flat", rings=5000, split="kaiser", beta=12.44, cut=45.0, Ns=192, m=3,
              precision="mixed"),
        # the same tangle in plain FP64 at the parameters its accuracy is judged at
        _case("tangle1m_device_fp64", api="device", rings=5000, beta=4.0, cut=16.0, Ns=512, m=5),
    ]


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    api = rng.choice(["lists", "lists", "flat", "device", "device", "step", "step", "ensemble"])
    mixed = rng.random() < 0.6
    split = "kaiser" if rng.random() < 0.3 else "gaussian"
    if api == "lists" and not mixed and rng.random() < 0.3:
        split = "open"
    top = {"lists": 4e4, "flat": 8e5, "device": 8e5, "step": 2e5, "ensemble": 2e3}[api]
    low = {"lists": 6e1, "flat": 5e3, "device": 2e3, "step": 5e2, "ensemble": 8e2}[api]
    total = log(low, min(top, 1e4) if split == "open" else top / (1 if mixed else 2))
    nodes = int(min(total, log(40, 400)))
    rings = max(1, round(total / nodes))
    total = rings * nodes
    # a cut-off that leaves some hundreds of pairs per node, as accuracy rules choose it
    cut = min(50.0, max(3.2, (12.57 * total / log(120, 1200)) ** (1 / 3)))
    beta = round(rng.uniform(2.8, 4.0) if split != "kaiser" else rng.uniform(8.0, 14.0), 3)
    while split != "open" and (beta * cut / math.pi if split == "kaiser" else beta * beta * cut * 2 / math.pi) > 300:
        cut *= 0.9  # a Fourier grid that stays below about 450 points a side
    spectra = api == "lists" and split != "open" and rings > 2 and rng.random() < 0.4  # (a plane ring has no helicity)
    return _case(api=api, rings=rings, nodes=nodes, ragged=rng.random() < 0.5,
                 lines=rng.choice([0, 0, 2, 4]) if api == "lists" and split != "open" else 0,
                 systems=rng.randint(4, 24) if api == "ensemble" else 1, split=split, beta=beta, cut=round(cut, 3),
                 sigma=rng.choice([1.25, 1.5, 1.5, 2.0]), m=rng.randint(3, 5) if mixed else rng.randint(4, 6),
                 fields=rng.choice([1, 3] if spectra else [1, 1, 2, 3]) if api in ("lists", "device") else 1, spectra=spectra,
                 precision="mixed" if mixed and split != "open" else "fp64",
                 tall=api != "ensemble" and split != "open" and rng.random() < 0.25)


# ---- inputs ----

def _counts(case, rings):
    """Nodes of every ring: the same, or spread over about a factor of six (fixed by the case)."""
    if not case["ragged"]:
        return [case["nodes"]] * rings
    return [max(5, int(case["nodes"] * (0.3 + 1.4 * ((k * 0.61803398875) % 1.0)))) for k in range(rings)]


def _rings_of(case, k):
    return case["rings"] + (k * 3) % 4 if case["api"] == "ensemble" else case["rings"]


def _periods(case):
    return (L, L, 2 * L) if case["tall"] else (L, L, L)


def _filaments(case, seed, k=0):
    """Random perturbed rings (uniform centres and orientations, radii L/8 .. L/4, radial Fourier modes
    2..8) and, in pairs of opposite orientation, helical lines along z: [(nodes [n, 3], offset [3])]."""
    rng = np.random.default_rng([int(seed), k])
    counts = _counts(case, _rings_of(case, k))
    Ls = np.array(_periods(case))
    B = len(counts)
    R = L / 8 * (1 + rng.random(B))
    centre = rng.random((B, 3)) * Ls
    quat = rng.standard_normal((B, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    w, x, y, z = quat.T
    e1 = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], 1)
    e2 = np.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], 1)
    kk = np.arange(2, 9)
    amp = 0.05 * rng.standard_normal((B, 7)) / kk
    phi = 2 * math.pi * rng.random((B, 7))
    out = [None] * B
    for n in sorted(set(counts)):
        idx = [i for i in range(B) if counts[i] == n]
        t = 2 * math.pi * (np.arange(n) + 0.5) / n
        r = R[idx, None] * (1 + sum(amp[idx, j, None] * np.cos(kk[j] * t + phi[idx, j, None]) for j in range(7)))
        pts = (centre[idx, None] + (r * np.cos(t))[..., None] * e1[idx, None] + (r * np.sin(t))[..., None] * e2[idx, None])
        for j, i in enumerate(idx):
            out[i] = (np.ascontiguousarray(pts[j]), np.zeros(3))
    for j in range(case["lines"]):
        sign, n = 1 - 2 * (j % 2), max(24, case["nodes"])
        t = (np.arange(n) + 0.5) / n - 0.5
        c = rng.random(2) * L
        a = 0.02 * L * (1 + rng.random())
        arg = 4 * math.pi * t + 2 * math.pi * rng.random()
        out.append((np.stack([c[0] + a * np.cos(arg), c[1] + a * np.sin(arg), (0.5 + sign * t) * Ls[2]], 1),
                    np.array([0.0, 0.0, sign * Ls[2]])))
    return out


def _time_step(fils):
    """Half the Kelvin-wave period of the shortest segment (the period is the limit of an explicit step)."""
    d = min(float(np.linalg.norm(np.roll(x, -1, axis=0) - x, axis=1).min()) for x, _ in fils)
    return d * d / GAMMA / (math.log(d / (math.pi * CORE)) + 0.5 - (DELTA + 0.5772156649015329))


# ---- the calls ----

def _package():
    name = "vortexpasta_b200"
    if name not in sys.modules:
        pkg = Path(__file__).resolve().parents[1] / "vortexpasta.jl_b200"
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _params(vp, case):
    Ls = _periods(case)
    if case["split"] == "open":
        sp = vp.NoSplitting()
    elif case["split"] == "kaiser":
        sp = vp.KaiserBesselSplitting(Ls=Ls, beta=case["beta"], rcut=L / case["cut"])
        if case["Ns"]:
            sp.Ns = (case["Ns"],) * 3
    elif case["Ns"]:
        sp = vp.GaussianSplitting(Ls=Ls, alpha=case["beta"] * case["cut"] / L, rcut=L / case["cut"], Ns=case["Ns"])
    else:
        sp = vp.GaussianSplitting(Ls=Ls, beta=case["beta"], rcut=L / case["cut"])
    return vp.ParamsBiotSavart(Gamma=GAMMA, a=CORE, Delta=DELTA, splitting=sp, quadrature=vp.GaussLegendre(NQUAD),
                               backend_long=vp.NonuniformFFTsBackend(case["sigma"], case["m"]),
                               precision=case["precision"])


class _DeviceArray:
    """A device field of the library ([3, Np] float64) as the CUDA array interface shows it.  Tensors made
    from it hold it, and so the cache whose memory it is."""

    def __init__(self, cache, ptr, n):
        self.cache = cache
        self.__cuda_array_interface__ = {"shape": (3, n), "typestr": "<f8", "data": (ptr, False), "version": 3}


_streams = []


def _stream():
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _field(s, bit):
    """The library's output array, wrapped once for as long as it stays where it is."""
    ptr = s["cache"].device_field(bit)[0]
    if s["views"].get(bit, (None,))[0] != ptr:
        s["views"][bit] = (ptr, torch.as_tensor(_DeviceArray(s["cache"], ptr, s["n"]), device="cuda"))
    return s["views"][bit][1]


def prepare(case, seed):
    vp = _package()
    api = case["api"]
    if api == "ensemble":
        systems = []
        for k in range(case["systems"]):
            fils = _filaments(case, seed, k)
            systems.append(([x for x, _ in fils], _params(vp, case), _time_step(fils)))
        ens = vp.timestepping.Ensemble(systems)
        return {"api": api, "ensemble": ens, "start": [x.clone() for x in ens.nodes],
                "stream": torch.cuda.ExternalStream(ens.stream())}
    fils = _filaments(case, seed)
    cache = vp.init_cache(_params(vp, case))
    offsets = np.concatenate([[0], np.cumsum([len(x) for x, _ in fils])]).astype(np.int64)
    nodes = np.concatenate([x for x, _ in fils])
    s = {"api": api, "cache": cache, "n": len(nodes), "offsets": offsets, "fields": case["fields"], "views": {}}
    if api == "lists":
        s["fs"] = [vp.curves.InfiniteFilament(x, o) if o.any() else x for x, o in fils]
        s["out"], s["lists"] = {}, {}
        for name, bit in (("velocity", 1), ("streamfunction", 2)):
            if case["fields"] & bit:
                s["out"][name] = np.zeros((len(nodes), 3))
                s["lists"][name] = [s["out"][name][a:b] for a, b in zip(offsets, offsets[1:])]
        s["spectra"] = case["spectra"]
    elif api == "flat":
        s["nodes"], s["out"] = nodes, np.zeros((len(nodes), 3))
    else:
        cache.set_stream(_stream().cuda_stream)
        s["nodes"] = torch.from_numpy(nodes).cuda()
        torch.cuda.synchronize()
        if api == "step":
            s["dt"], s["work"] = _time_step(fils), s["nodes"].clone()
            torch.cuda.synchronize()
            cache.set_filaments(None, on_device_ptr=s["work"].data_ptr(), offsets=offsets)
    return s


def run(s):
    vp = _package()
    api = s["api"]
    if api == "lists":
        vp.compute_on_nodes_(s["lists"], s["cache"], s["fs"])
        out = dict(s["out"])
        if s["spectra"]:
            out["energy"] = vp.diagnostics.energy_spectrum(s["cache"])[1]
            out["helicity"] = vp.diagnostics.helicity_spectrum(s["cache"])[1]
        return out
    if api == "flat":
        s["cache"].set_filaments_flat(s["nodes"], s["offsets"])
        s["cache"].compute(s["fields"])
        return s["cache"].get(1, s["out"])
    if api == "device":
        s["cache"].set_filaments(None, on_device_ptr=s["nodes"].data_ptr(), offsets=s["offsets"])
        s["cache"].compute(s["fields"])
        return [_field(s, bit) for bit in (1, 2) if s["fields"] & bit]
    if api == "step":  # one step from the same state, so that every pass does the same work
        with torch.cuda.stream(_stream()):
            s["work"].copy_(s["nodes"])
        vp.timestepping.rk4_step(s["cache"], s["work"].data_ptr(), s["dt"])
        return [s["work"], _field(s, 1)]
    stream, common = s["stream"], _stream()  # steps of different ensembles follow one another
    stream.wait_stream(common)
    with torch.cuda.stream(stream):
        torch._foreach_copy_(s["ensemble"].nodes, s["start"])
    s["ensemble"].step(1)
    common.wait_stream(stream)
    return list(s["ensemble"].nodes)


# ---- work and tolerances ----

def _grid(case):
    """(modes, oversampled FFT points) per dimension."""
    Ns, n = [], []
    for Ld in _periods(case):
        kmax = (2 * case["beta"] ** 2 if case["split"] == "gaussian" else case["beta"]) * case["cut"] / L
        N = case["Ns"] or 2 * math.ceil(kmax * Ld / (2 * math.pi)) + 2
        f = max(2, math.ceil(case["sigma"] * N - 1e-9))
        while f % 2 or not _smooth(f):
            f += 1
        Ns.append(N)
        n.append(f)
    return Ns, n


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


def work(case):
    """Per evaluation: 40 operations a pair and field in range (20 more for the second field), the
    window's updates, the FFTs and the splines.  Bytes: nodes in, fields out."""
    flops = total = 0.0
    for k in range(case["systems"]):
        N = sum(_counts(case, _rings_of(case, k))) + case["lines"] * max(24, case["nodes"])
        total += N
        Nq, V = NQUAD * N, np.prod(_periods(case))
        nf = 2 if case["fields"] == 3 else 1
        ops = 400.0 * N
        if case["split"] == "open":
            ops += N * Nq * (20 + 20 * nf)
        else:
            n3 = float(np.prod(_grid(case)[1]))
            ops += N * Nq * min(1.0, 4 / 3 * math.pi * (L / case["cut"]) ** 3 / V) * (20 + 20 * nf)
            ops += 6.0 * (2 * case["m"]) ** 3 * (Nq + nf * N) + (1 + nf) * 3 * 2.5 * n3 * math.log2(n3)
        flops += ops * (4 if case["api"] in ("step", "ensemble") else 1)
    nf = 2 if case["fields"] == 3 else 1
    return {"bytes": 24.0 * total * (1 + nf), "flops": float(flops)}


def tolerance(case):
    """About four times what was measured between the library and ``exact``.  FP64 (rel 2e-11, max 1e-10):
    sums in another order and another solver of the spline system, whose s'' is a second divided
    difference.  Mixed (rel 2.5e-7, max 1.3e-6): 32-bit grids, transforms and pair terms, and the
    run-dependent order of the 32-bit sums; in the velocity of an RK4 step's last stage (1.3e-6, 6e-5) the
    earlier stages' rounding moves the nodes, and s'' with them; helicity spectra cancel (5e-7)."""
    if case["precision"] == "fp64":
        return {"rel": 1e-10, "max": 1e-9}
    if case["api"] == "ensemble":  # positions alone: a step moves a node by a small part of the box
        return {"rel": 3e-10, "max": 5e-8}
    if case["api"] == "step" or case["spectra"]:
        return {"rel": 5e-6, "max": 2.5e-4}
    return {"rel": 1e-6, "max": 5e-6}


# ---- the same quantities in 64 bits ----

def _bspline(K, tx, n, i, x):
    """The K B-splines of order K that are non-zero on segment i at x: a list of K tensors shaped like x."""
    def t(j):
        return torch.gather(tx, 1, (i + j + n).expand(tx.shape[0], -1))[..., None].expand_as(x)
    left = [None] + [x - t(1 - r) for r in range(1, K)]
    right = [None] + [t(r) - x for r in range(1, K)]
    N = [torch.ones_like(x)]
    for r in range(1, K):
        saved, new = torch.zeros_like(x), []
        for s in range(r):
            v = N[s] / (right[s + 1] + left[r - s])
            new.append(saved + right[s + 1] * v)
            saved = left[r - s] * v
        N = new + [saved]
    return N


def _points_of(X, off, knots=None):
    """Point data of [B] filaments of n nodes each (X [B, n, 3], end-to-end offsets [B, 3]): s', s'' on the
    nodes, segment lengths, quadrature points and charges; periodic quintic splines on chordal knots."""
    B, n, _ = X.shape
    dev = X.device
    if knots is None:
        d = torch.roll(X, -1, 1) - X
        d[:, -1] += off
        ls = torch.linalg.norm(d, dim=2)
        knots = (torch.cat([torch.zeros(B, 1, dtype=X.dtype, device=dev), torch.cumsum(ls, 1)], 1))
    t, T = knots[:, :n], knots[:, n:]
    tx = torch.cat([t - T, t, t + T], 1)
    i = torch.arange(n, device=dev)
    N = _bspline(6, tx, n, i, t[..., None])
    A = torch.zeros(B, n, n, dtype=X.dtype, device=dev)
    for s in range(5):
        A[:, i, (i - 5 + s) % n] += N[s][..., 0]
    c = torch.linalg.solve(A, X - (t / T)[..., None] * off[:, None])
    c1 = 5 * (c - torch.roll(c, 1, 1)) / (tx[:, n + 5 + i] - tx[:, n + i])[..., None]
    c2 = 4 * (c1 - torch.roll(c1, 1, 1)) / (tx[:, n + 4 + i] - tx[:, n + i])[..., None]
    zeta, wq = np.polynomial.legendre.leggauss(NQUAD)
    zeta, wq = (torch.tensor(v / 2 + a, dtype=X.dtype, device=dev) for v, a in ((zeta, 0.5), (wq, 0.0)))
    dt = (tx[:, n + 1 + i] - t)[..., None]

    def at(coef, D, z):
        x = t[..., None] + z * dt
        Ns = _bspline(6 - D, tx, n, i, x)
        v = sum(Ns[s][..., None] * coef[:, (i - 5 + D + s) % n, None] for s in range(6 - D))
        if D == 0:
            v = v + (x / T[..., None])[..., None] * off[:, None, None]
        elif D == 1:
            v = v + (off / T)[:, None, None]
        return v

    zero = torch.zeros(1, dtype=X.dtype, device=dev)
    s1, s2 = at(c1, 1, zero)[:, :, 0], at(c2, 2, zero)[:, :, 0]
    pts, der = at(c, 0, zeta), at(c1, 1, zeta)
    length = dt[..., 0] * (wq * torch.linalg.norm(der, dim=3)).sum(2)
    return s1, s2, length, pts, der * (wq * dt)[..., None], knots


def _geometry(fils, dev, knots=None):
    """Point data of all filaments, concatenated in order; `knots`: those of an earlier call, kept."""
    N = sum(len(x) for x, _ in fils)
    f8 = dict(dtype=torch.float64, device=dev)
    G = {"x": torch.empty(N, 3, **f8), "s1": torch.empty(N, 3, **f8), "s2": torch.empty(N, 3, **f8),
         "dp": torch.empty(N, **f8), "p": torch.empty(N, NQUAD, 3, **f8), "q": torch.empty(N, NQUAD, 3, **f8),
         "prev": torch.empty(N, dtype=torch.int64, device=dev), "knots": {}}
    start = np.concatenate([[0], np.cumsum([len(x) for x, _ in fils])])
    for n in sorted({len(x) for x, _ in fils}):
        every = [i for i in range(len(fils)) if len(fils[i][0]) == n]
        for b in range(0, len(every), 512):
            idx = every[b:b + 512]
            X = torch.stack([torch.as_tensor(fils[i][0], **f8) for i in idx])
            off = torch.tensor(np.array([fils[i][1] for i in idx]), **f8)
            rows = torch.tensor(start[idx], device=dev)[:, None] + torch.arange(n, device=dev)
            s1, s2, ln, p, q, kn = _points_of(X, off, None if knots is None else knots[n, b])
            G["knots"][n, b] = kn
            G["x"][rows], G["s1"][rows], G["s2"][rows], G["dp"][rows], G["p"][rows], G["q"][rows] = X, s1, s2, ln, p, q
            G["prev"][rows] = torch.roll(rows, 1, 1)
    return G


def _kaiser_series(beta, rcut, rtol):
    """Chebyshev series (in r / rcut) of the Kaiser-Bessel kernel cut at rtol, and of its integral: the
    short-range weights of that splitting are defined by them."""
    C = np.polynomial.chebyshev
    N = 64
    while True:
        u = np.cos(math.pi * np.arange(N) / (N - 1))
        f = beta / (rcut * math.sinh(beta)) * np.i0(beta * np.sqrt(np.maximum(0, 1 - u * u)))
        w = np.ones(N)
        w[[0, -1]] = 0.5
        T = np.cos(math.pi * (np.outer(np.arange(N), np.arange(N)) % (2 * (N - 1))) / (N - 1))
        c = 2 / (N - 1) * T @ (w * f)
        c[[0, -1]] *= 0.5
        small = np.abs(c) < rtol * np.abs(c).sum()
        cut = next((j for j in range(N - 1) if small[j] and small[j + 1]), None)
        if cut is not None:
            break
        N *= 2
    c = c[:cut]
    c[1::2] = 0.0
    return c, C.chebint(c, lbnd=0) * rcut


def _clenshaw(c, u):
    b1 = b2 = torch.zeros_like(u)
    for v in c[:0:-1]:
        b1, b2 = 2 * u * b1 + float(v) - b2, b1
    return float(c[0]) + u * b1 - b2


def _short_range(case, G, fields):
    """Local term, the pairs within the cut-off, and the removal of the two segments next to each node."""
    x, Ls = G["x"], torch.tensor(_periods(case), dtype=torch.float64, device=G["x"].device)
    is_open = case["split"] == "open"
    p, q = G["p"].reshape(-1, 3), G["q"].reshape(-1, 3)
    rcut, pref = L / case["cut"], GAMMA / (4 * math.pi)
    N = len(x)
    series = None
    if case["split"] == "kaiser":
        series = _kaiser_series(case["beta"], rcut, 10 ** -0.2 * math.exp(-case["beta"]))

    def weights(r):
        if is_open:
            return torch.ones_like(r), torch.ones_like(r)
        if series is not None:
            a = 1 - _clenshaw(series[1], r / rcut)
            return a, a + r * _clenshaw(series[0], r / rcut)
        ar = case["beta"] / rcut * r
        a = torch.erfc(ar)
        return a, a + 2 / math.sqrt(math.pi) * ar * torch.exp(-ar * ar)

    def integrands(d, qs, full):
        r = torch.linalg.norm(d, dim=-1, keepdim=True)
        a, g = (torch.ones_like(r), torch.ones_like(r)) if full else weights(r)
        return (torch.cross(qs, d, dim=-1) * (g / r ** 3) if fields & 1 else None), (qs * (a / r) if fields & 2 else None)

    def add(to, rows, t):
        if t is not None:
            to.index_add_(0, rows, t)

    v, ps = torch.zeros_like(x), torch.zeros_like(x)
    # nodes in order of x; each run of them meets only the sources within the cut-off of it in x
    if is_open:
        order, images = torch.arange(N, device=x.device), [torch.arange(len(p), device=x.device)]
        px = torch.zeros(len(p), dtype=x.dtype, device=x.device)
    else:
        xf, pf = torch.remainder(x[:, 0], Ls[0]), torch.remainder(p[:, 0], Ls[0])
        order, by_x = torch.argsort(xf), torch.argsort(pf)
        xf, images = xf[order], [by_x] * 3
        px = torch.cat([pf[by_x] - Ls[0], pf[by_x], pf[by_x] + Ls[0]])
    images = torch.cat(images)
    a, near = 0, torch.arange(len(p), device=x.device)
    while a < N:
        step = max(1, (1 << 27) // max(1, len(near)))
        mine = order[a:a + step]
        if not is_open:
            ends = torch.stack([xf[a] - rcut, xf[min(a + step, N) - 1] + rcut]) + torch.tensor([-1e-9, 1e-9], device=x.device)
            lo, hi = torch.searchsorted(px, ends).tolist()
            near = images[lo:min(hi, lo + len(p))]
        xs, a = x[mine], a + step
        pn, qn = p[near], q[near]
        r2 = torch.zeros(len(xs), len(pn), device=x.device)  # candidates in 32 bits, with a margin
        for d in range(3):
            e = xs[:, d, None].float() - pn[None, :, d].float()
            if not is_open:
                e -= Ls[d] * torch.round(e / Ls[d])
            r2.addcmul_(e, e)
        i, j = torch.nonzero(r2 <= (math.inf if is_open else rcut * rcut * 1.001 + 1e-5), as_tuple=True)
        for b in range(0, len(i), 1 << 24):
            ii, jj = i[b:b + (1 << 24)], j[b:b + (1 << 24)]
            d = xs[ii] - pn[jj]
            if not is_open:
                d -= Ls * torch.round(d / Ls)
                keep = (d * d).sum(1) <= rcut * rcut
                d, ii, jj = d[keep], ii[keep], jj[keep]
            dv, dp = integrands(d, qn[jj], False)
            add(v, mine[ii], dv)
            add(ps, mine[ii], dp)
    for seg in (torch.arange(N, device=x.device), G["prev"]):
        d = x[:, None] - G["p"][seg]
        if not is_open:
            d -= Ls * torch.round(d / Ls)
        dv, dp = integrands(d, G["q"][seg], True)
        v -= dv.sum(1) if dv is not None else 0.0
        ps -= dp.sum(1) if dp is not None else 0.0
    delta = torch.sqrt(G["dp"] * G["dp"][G["prev"]])[:, None]
    rpsi = math.exp(DELTA - 1) * CORE / 2
    mu = torch.linalg.norm(G["s1"], dim=1, keepdim=True)
    v += torch.log(delta / (rpsi * math.e)) / mu ** 3 * torch.cross(G["s1"], G["s2"], dim=1)
    ps += 2 * torch.log(delta / rpsi) / mu * G["s1"]
    return pref * v, pref * ps


def _long_range(case, G, fields, want_spectra):
    """Windowed spreading, FFT, the Fourier-space operators, inverse FFT and interpolation."""
    dev = G["x"].device
    f8 = dict(dtype=torch.float64, device=dev)
    Ns, n = _grid(case)
    Ls, m = _periods(case), case["m"]
    W = 2 * m
    shape = 0.97 * math.pi * (1 - 1 / (2 * case["sigma"])) * W
    edge = math.exp(-shape)
    gx, gw = np.polynomial.legendre.leggauss(128)

    def hat(xi):  # Fourier transform of the window at xi radians per grid spacing
        th = 0.5 * math.pi * gx
        f = (np.exp(shape * (np.cos(th) - 1)) - edge) * np.cos(th) * 0.5 * math.pi * gw
        return m * (np.cos(np.outer(xi, m * np.sin(th))) @ f)

    def footprint(x):  # flat grid indices and window products of some points: [P, W^3]
        idx, val = [], []
        for d in range(3):
            xh = x[:, d] * (n[d] / Ls[d])
            i0 = torch.floor(xh) - (m - 1)
            s = i0[:, None] + torch.arange(W, **f8)
            z = (xh[:, None] - s) / m
            val.append(torch.where(z.abs() < 1, torch.exp(shape * (torch.sqrt((1 - z * z).clamp_min(0)) - 1)) - edge, 0.0))
            idx.append(torch.remainder(s.long(), n[d]))
        flat = (idx[2][:, :, None, None] * n[1] + idx[1][:, None, :, None]) * n[0] + idx[0][:, None, None, :]
        v = val[2][:, :, None, None] * val[1][:, None, :, None] * val[0][:, None, None, :]
        return flat.reshape(len(x), -1), v.reshape(len(x), -1)

    p, q = G["p"].reshape(-1, 3), G["q"].reshape(-1, 3)
    per = max(1, (1 << 25) // W ** 3)
    grid = torch.zeros(3, n[0] * n[1] * n[2], **f8)
    for a in range(0, len(p), per):
        flat, v = footprint(p[a:a + per])
        for c in range(3):
            grid[c].index_add_(0, flat.reshape(-1), (v * q[a:a + per, c, None]).reshape(-1))
    k = [np.arange(Ns[0] // 2 + 1)] + [np.concatenate([np.arange((N + 1) // 2), np.arange(-(N // 2), 0)]) for N in Ns[1:]]
    F = torch.fft.rfftn(grid.reshape(3, n[2], n[1], n[0]), dim=(1, 2, 3))
    iz, iy = (torch.tensor(k[d] % n[d], device=dev) for d in (2, 1))
    F = F[:, iz][:, :, iy][..., :len(k[0])]
    live = [torch.ones(len(k[d]), dtype=torch.bool, device=dev) for d in range(3)]
    live[0][-1] = False
    for d in (1, 2):
        if Ns[d] % 2 == 0:
            live[d][Ns[d] // 2] = False

    def outer(t, op=torch.mul):
        return op(op(t[2][:, None, None], t[1][None, :, None]), t[0][None, None, :])

    dec = outer([torch.tensor(1 / hat(2 * math.pi * k[d] / n[d]), **f8) for d in range(3)])
    kv = [torch.tensor(2 * math.pi / Ls[d] * k[d], **f8) for d in range(3)]
    k2 = outer([t * t for t in kv], torch.add)
    w = F * dec * outer(live) * (GAMMA / (Ls[0] * Ls[1] * Ls[2]))
    inv = torch.where(k2 > 0, 1 / k2.clamp_min(1e-300), 0.0)
    K = [kv[0][None, None, :], kv[1][None, :, None], kv[2][:, None, None]]

    def curl(u):
        return 1j * torch.stack([K[1] * u[2] - K[2] * u[1], K[2] * u[0] - K[0] * u[2], K[0] * u[1] - K[1] * u[0]])

    if case["split"] == "kaiser":
        s = case["beta"] ** 2 - k2 * (L / case["cut"]) ** 2
        root = torch.sqrt(s.clamp_min(1e-300))
        ewald = torch.where(s > 0, case["beta"] / math.sinh(case["beta"]) * torch.sinh(root) / root, 0.0)
    else:
        ewald = torch.exp(-k2 / (4 * (case["beta"] * case["cut"] / L) ** 2))
    res = {}
    for name, bit, u in (("velocity", 1, lambda: curl(w) * inv), ("streamfunction", 2, lambda: w * inv)):
        if not fields & bit:
            continue
        full = torch.zeros(3, n[2], n[1], n[0] // 2 + 1, dtype=torch.complex128, device=dev)
        full[:, iz[:, None, None], iy[None, :, None], torch.arange(len(k[0]), device=dev)] = u() * ewald * dec
        g = torch.fft.irfftn(full, s=(n[2], n[1], n[0]), dim=(1, 2, 3), norm="forward").reshape(3, -1)
        out = torch.empty_like(G["x"])
        for a in range(0, len(out), per):
            flat, v = footprint(G["x"][a:a + per])
            out[a:a + per] = torch.stack([(g[c][flat] * v).sum(1) for c in range(3)], 1)
        res[name] = out
    if want_spectra:  # of the velocity held after the call, or of the streamfunction's vorticity
        u = curl(w) * inv
        dk = 2 * math.pi / Ls[0]
        bins = (torch.sqrt(k2) / dk + 0.5).long()
        half = torch.where(K[0] == 0, 0.5, 1.0).expand_as(k2) / dk
        V = Ls[0] * Ls[1] * Ls[2]
        for name, val in (("energy", (u.abs() ** 2).sum(0)), ("helicity", 2 * V * (u.conj() * curl(u)).real.sum(0))):
            spec = torch.zeros(len(k[0]), **f8)
            keep = bins < len(spec)
            res[name] = spec.index_add_(0, bins[keep], (val * half)[keep])
    return res


def _evaluate(case, G, fields, spectra=False):
    v, ps = _short_range(case, G, fields)
    res = {"velocity": v, "streamfunction": ps}
    if case["split"] != "open":
        for name, t in _long_range(case, G, fields, spectra).items():
            res[name] = res[name] + t if name in res else t
    return res


def _exact_step(case, fils, dt, dev):
    """One RK4 step (knots of the first stage kept) -> (nodes after it, velocity of its last stage)."""
    G = _geometry(fils, dev)
    x0, knots = G["x"], G["knots"]
    start = np.concatenate([[0], np.cumsum([len(x) for x, _ in fils])])
    total = torch.zeros_like(x0)
    for weight, ahead in ((1, 0.5), (2, 0.5), (2, 1.0), (1, 0.0)):
        v = _evaluate(case, G, 1)["velocity"]
        total += weight * v
        if ahead:
            x = x0 + ahead * dt * v
            G = _geometry([(x[a:b], o) for a, b, (_, o) in zip(start, start[1:], fils)], dev, knots)
    return x0 + dt / 6 * total, v


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["api"] == "ensemble":
        out = []
        for k in range(case["systems"]):
            fils = _filaments(case, seed, k)
            out.append(_exact_step(case, fils, _time_step(fils), dev)[0])
        return out
    fils = _filaments(case, seed)
    if case["api"] == "step":
        x, v = _exact_step(case, fils, _time_step(fils), dev)
        return [x, v.T.contiguous()]
    res = _evaluate(case, _geometry(fils, dev), case["fields"], case["spectra"])
    names = [n for n, bit in (("velocity", 1), ("streamfunction", 2)) if case["fields"] & bit]
    if case["api"] == "lists":
        return {n: res[n].cpu().numpy() for n in names + (["energy", "helicity"] if case["spectra"] else [])}
    if case["api"] == "flat":
        return res["velocity"].cpu().numpy()
    return [res[n].T.contiguous() for n in names]
