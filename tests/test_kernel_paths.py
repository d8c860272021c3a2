"""The kernels and branches that sizes select, at the sizes where they change, against the CPU restatement:
spline solves of filaments around the block counts of the partitioned solve (and its serial form), spreading
and interpolation over kernel widths on grids that bricks do not divide, pair kernels over cell widths and
periodic images, the open-domain pairs around a block of nodes, the interleaved interpolation.

FP64 to 1e-10 as everywhere; mixed to 1e-6 (eight times the 1.2e-7 of the 32-bit pair and grid sums)."""

import math

import numpy as np
import pytest

L = 2 * math.pi
TOL = {"fp64": 1e-10, "mixed": 1e-6}


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def wobbly(vp, n, seed, spread=0.0):
    """A closed curve of n nodes with unequal spacings (by a factor of up to exp(spread))."""
    rng = np.random.default_rng(seed)
    t = np.cumsum(np.exp(spread * (rng.random(n) - 0.5)))
    t = 2 * np.pi * t / t[-1]
    r = 0.9 + 0.1 * np.cos(3 * t)
    return np.stack([3 + r * np.cos(t), 2 + r * np.sin(t), 1 + 0.2 * np.sin(2 * t)], axis=1)


def fields(vp, p, fs, names=("velocity", "streamfunction"), spread_mode=0, entry_bits=0, **kw):
    cache = vp.init_cache(p)
    try:
        assert cache._lib.vpbs_pair_entries(cache.handle, entry_bits) == 0
        assert cache._lib.vpbs_spread_mode(cache.handle, spread_mode) == 0
        out = {n: [np.zeros((len(f), 3)) for f in fs] for n in names}
        vp.compute_on_nodes_(out, cache, fs, **kw)
        counts = cache.pair_counts() if kw.get("shortrange", True) else None
    finally:
        cache.close()
    return {n: np.concatenate(v) for n, v in out.items()}, counts


def params(vp, precision="fp64", rcut=L / 5, Ns=16, m=4, nsubdiv=2, **kw):
    return vp.ParamsBiotSavart(Gamma=1.1, a=1e-8, splitting=vp.GaussianSplitting(Ls=L, alpha=3.4 / rcut, rcut=rcut, Ns=Ns),
                               backend_short=vp.CellListsBackend(nsubdiv), backend_long=vp.NonuniformFFTsBackend(1.5, m),
                               precision=precision, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0.0, 2.0])
def test_spline_solve_sizes(vp, oracle, spread):
    """15 | 16: serial or partitioned; 31 | 32, 63 | 64, 127 | 128: 4, 8, 16, 32 blocks; 600: work space outside
    shared memory."""
    fs = [wobbly(vp, n, n, spread) for n in (5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 331, 600)]
    p = params(vp)
    want = oracle.point_data(p, fs)
    cache = vp.init_cache(p)
    try:
        cache.set_filaments(fs)
        got = cache.pointdata()
    finally:
        cache.close()
    for name, tol in (("d1", 1e-11), ("d2", 1e-9), ("charges", 1e-11), ("dp", 1e-11)):
        start = 0
        for f in fs:
            k = len(f) * (3 if name == "charges" else 1)
            assert rel(got[name][start:start + k], want[name][start:start + k]) <= tol, (name, len(f))
            start += k


@pytest.mark.gpu
def test_spline_solve_extreme_spacings(vp, oracle):
    """Spacings a thousand times shorter here and there: pivots of the partitioned solve fall below its bound and
    the serial form takes over.  Condition number 1e6, so 1e6 eps ~ 2e-10 times some tens."""
    rng = np.random.default_rng(3)
    t = np.cumsum(np.where(rng.random(200) < 0.1, 1e-3, 1.0))
    t = 2 * np.pi * t / t[-1]
    f = np.stack([3 + np.cos(t), 2 + np.sin(t), 1 + 0.1 * np.sin(t)], axis=1)
    p = params(vp)
    want = oracle.point_data(p, [f])
    cache = vp.init_cache(p)
    try:
        cache.set_filaments([f])
        got = cache.pointdata()
    finally:
        cache.close()
    assert rel(got["d1"], want["d1"]) <= 1e-8
    assert rel(got["points"], want["points"]) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 6, 8])
@pytest.mark.parametrize("mode", [0, 1])
def test_window_widths_on_ragged_grids(vp, oracle, m, precision, mode):
    """FFT sizes 18, 30, 36 (bricks of 8 leave 2, 6 and 4 cells over): widths 2 .. 16, wider than a brick too; atomics
    (which so few points take by themselves) and bricks."""
    sp = vp.GaussianSplitting(Ls=(L, L, L), alpha=5.0, rcut=L / 4, Ns=(12, 20, 24))
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, m), precision=precision)
    fs = [wobbly(vp, n, n, 0.5) + np.array([dx, 0.0, dx]) for n, dx in ((40, 0.0), (64, 2.0), (23, 4.5))]
    v, s, _ = oracle.compute_on_nodes(p, fs, velocity=True, streamfunction=True, LIA=False, shortrange=False)
    got, _ = fields(vp, p, fs, LIA=False, shortrange=False, spread_mode=mode)
    # mixed: 32-bit rounding of the transforms, 6e-8 times about four, which the deconvolution multiplies, once per
    # transform, by psi_hat(0) / psi_hat(k): 2.0 (m = 2) to 7 (m = 8) per dimension at the edge of the kept modes,
    # weighted by a filter that leaves e^{-k^2 / 4 alpha^2} = 0.7 there in one dimension (m = 8: 2.2e-6)
    tol = 1e-10 if precision == "fp64" else 2e-6 if m <= 5 else 1e-5
    assert rel(got["velocity"], v) <= tol and rel(got["streamfunction"], s) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("m", [4, 5, 6])
def test_mixed_sums_on_grids_without_whole_bricks(vp, m):
    """FFT sizes 18, 30, 36, which no bricks of 16, 12, 10 or 8 points tile: the mixed form's grid values are rounded
    once, from FP64 sums.  30,000 points on 19,440 cells: sums in FP32 leave 2.4e-7 (m = 4) to 5e-7 (m = 6); the
    transforms and the interpolation by themselves, 0.9e-7."""
    rng = np.random.default_rng(2)
    fs = [vp.curves.ring(200, 0.6 + 0.6 * rng.random(), L * rng.random(3), vp.curves.random_rotation(rng)) for _ in range(50)]
    got = {}
    for precision in ("fp64", "mixed"):
        sp = vp.GaussianSplitting(Ls=(L, L, L), alpha=1.7, rcut=L / 5, Ns=(12, 20, 24))
        p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, m), precision=precision)
        got[precision], _ = fields(vp, p, fs, LIA=False, shortrange=False, spread_mode=1)
    for name in ("velocity", "streamfunction"):
        assert rel(got["mixed"][name], got["fp64"][name]) <= 1.5e-7, name


@pytest.mark.gpu
@pytest.mark.parametrize("Ns,m,nodes", [(12, 3, 4000), (36, 1, 20000), (36, 4, 1000)])
def test_spreading_of_few_bricks_or_points_takes_atomics(vp, Ns, m, nodes):
    """Grids of few bricks (18^3) or points (54^3), where a CTA per brick is slower by 1.4 to 20 times: the stage's
    time by the default mode is well below that of the bricks."""
    rng = np.random.default_rng(2)
    fs = [vp.curves.ring(200, 0.6 + 0.6 * rng.random(), L * rng.random(3), vp.curves.random_rotation(rng)) for _ in range(nodes // 200)]
    sp = vp.GaussianSplitting(Ls=L, alpha=2.0, rcut=L / 5, Ns=Ns)
    cache = vp.init_cache(vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, m)))
    best = []
    try:
        cache.set_filaments(fs)
        cache.stage_timing(True)
        for mode in (0, 1):
            assert cache._lib.vpbs_spread_mode(cache.handle, mode) == 0
            times = []
            for _ in range(8):
                cache.compute(1, shortrange=False)
                times.append(cache.stage_times()["spread"])
            best.append(min(times[2:]))
    finally:
        cache.close()
    assert best[0] < 0.85 * best[1]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nsubdiv,rcut,explicit", [(1, L / 3, True), (1, L / 7, False), (2, 0.4 * L, True), (2, L / 6, False),
                                                   (3, L / 4, True)])
def test_pair_kernels(vp, oracle, nsubdiv, rcut, explicit, precision):
    """Neighbourhoods that span the whole period, cells of few and many nodes, rows of more than 32; nodes at the
    corners of the box, so every periodic image occurs; one and both fields; equal pair counts."""
    fs = [wobbly(vp, n, n, 1.0) + np.array(o) for n, o in ((64, (-3, -2, -1)), (37, (3.2, 4.2, 5.2)), (150, (0, 0, 0)), (21, (-3, 1, 5)))]
    p = params(vp, precision, rcut, nsubdiv=nsubdiv, avoid_explicit_erf=not explicit)
    v, s, st = oracle.compute_on_nodes(p, fs, velocity=True, streamfunction=True, LIA=False, longrange=False)
    for names in (("velocity", "streamfunction"), ("velocity",), ("streamfunction",)):
        got, counts = fields(vp, p, fs, names, LIA=False, longrange=False)
        for n, want in (("velocity", v), ("streamfunction", s)):
            if n in names:
                assert rel(got[n], want) <= TOL[precision], (n, names)
        if precision == "fp64":
            assert counts[0] == st["pairs_in_range"]


def pairs_in_range(oracle, p, fs):
    """The pair count of the CPU restatement; the mixed form always leaves a node's own two segments out."""
    from copy import copy
    q = copy(p)
    if p.precision == "mixed":
        q.avoid_explicit_erf = False
    return oracle.compute_on_nodes(q, fs, velocity=True, streamfunction=True, LIA=False, longrange=False)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("Ls,rcut", [((L, L, L), L / 3), ((L, 0.7 * L, 1.6 * L), 0.2 * L), ((L, L, 2.5 * L), L / 12),
                                     ((L, L, L), L / 60), ((0.3 * L, L, L), L / 40)])
@pytest.mark.parametrize("entry_bits", [0, 64])
def test_pair_counts(vp, oracle, Ls, rcut, precision, entry_bits):
    """The same pairs as the CPU restatement, also in the mixed form, whose screen and decision are in 32 bits: periods of
    different lengths, and cut-offs so short that the 32-bit places are coarse beside them (L / 60: margin 8e-5 of
    r_cut^2).  The queue entries of systems above 2^26 sources too."""
    rng = np.random.default_rng(5)
    fs = [vp.curves.ring(n, 0.2 + 0.7 * rng.random(), np.array(Ls) * rng.random(3), vp.curves.random_rotation(rng))
          for n in (64, 150, 33, 400, 7, 250, 250)]
    sp = vp.GaussianSplitting(Ls=Ls, alpha=3.4 / rcut, rcut=rcut, Ns=(16, 16, 16))
    p = vp.ParamsBiotSavart(Gamma=1.1, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, 4), precision=precision)
    v, s, st = pairs_in_range(oracle, p, fs)
    for names in (("velocity", "streamfunction"), ("velocity",), ("streamfunction",)):
        got, counts = fields(vp, p, fs, names, entry_bits=entry_bits, LIA=False, longrange=False)
        assert counts[0] == st["pairs_in_range"]
        for n, want in (("velocity", v), ("streamfunction", s)):
            if n in names:
                assert rel(got[n], want) <= TOL[precision], (n, names)


@pytest.mark.gpu
@pytest.mark.parametrize("beta,names", [(12.0, ("velocity", "streamfunction")), (18.0, ("velocity", "streamfunction")),
                                        (18.0, ("streamfunction",)), (35.0, ("velocity",))])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pairs_with_long_weight_tables(vp, oracle, beta, names, precision):
    """alpha r_cut beyond what the kernels keep in shared memory: 5.9 for the FP32 one (the mixed form takes the FP64
    one), 16.6 for both fields and 33.3 for one in the FP64 one (a warp per node with tables in global memory)."""
    fs = [wobbly(vp, n, n, 1.0) + np.array(o) for n, o in ((64, (-3, -2, -1)), (37, (3.2, 4.2, 5.2)), (150, (0, 0, 0)))]
    sp = vp.GaussianSplitting(Ls=L, alpha=beta / (L / 4), rcut=L / 4, Ns=16)
    p = vp.ParamsBiotSavart(Gamma=1.1, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, 4), precision=precision)
    v, s, st = pairs_in_range(oracle, p, fs)
    got, counts = fields(vp, p, fs, names, LIA=False, longrange=False)
    assert counts[0] == st["pairs_in_range"]
    for n, want in (("velocity", v), ("streamfunction", s)):
        if n in names:
            assert rel(got[n], want) <= TOL[precision], n


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("names", [("velocity",), ("velocity", "streamfunction")])
def test_candidates_are_pairs(vp, precision, names):
    """Node counts that do not fill the groups of 4 or 2 nodes a warp takes, and nodes apart from one another in a group:
    only pairs of nodes that are there are counted as candidates, so never more than there are."""
    for fs in ([wobbly(vp, 5, 1)], [wobbly(vp, 5, k) + np.array([0.0, 0.3 * k, 2.0 * k]) for k in range(3)]):
        _, (pairs, candidates) = fields(vp, params(vp, precision, 0.39 * L), fs, names, LIA=False, longrange=False)
        n = sum(map(len, fs))
        assert pairs <= candidates <= n * 3 * n


@pytest.mark.gpu
def test_mixed_pair_sums_of_many_pairs(vp):
    """20,000 pairs a node, 600 a lane: the rounding of the 32-bit sums does not grow with them.  One sum per lane leaves
    1.3e-7 (streamfunction) and 2.4e-7 (velocity); the weights and separations by themselves, 0.4e-7 and 1.0e-7."""
    rng = np.random.default_rng(4)
    fs = [vp.curves.ring(200, 0.8 + 0.7 * rng.random(), L * rng.random(3), vp.curves.random_rotation(rng)) for _ in range(500)]
    got = {}
    for precision in ("fp64", "mixed"):
        p = params(vp, precision, L / 4, Ns=32)
        got[precision], _ = fields(vp, p, fs, LIA=False, longrange=False)
    assert rel(got["mixed"]["streamfunction"], got["fp64"]["streamfunction"]) <= 8e-8
    assert rel(got["mixed"]["velocity"], got["fp64"]["velocity"]) <= 1.9e-7


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 42, 43, 127, 128, 129, 700])
def test_open_domain_sizes(vp, oracle, n):
    """One node block and its neighbours in size; 15 .. 2100 sources (tiles of 128, shared out over blocks)."""
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=vp.NoSplitting())
    fs = [wobbly(vp, n, n, 0.5)]
    v, s, _ = oracle.compute_on_nodes(p, fs, velocity=True, streamfunction=True)
    got, _ = fields(vp, p, fs)
    assert rel(got["velocity"], v) <= 1e-10 and rel(got["streamfunction"], s) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("n,names", [(90, ("velocity",)), (700, ("velocity", "streamfunction")), (4014, ("velocity",)),
                                     (4014, ("streamfunction",))])
def test_open_domain_repeats_itself(vp, n, names):
    """The same call gives the same bits, although the sources are shared out over groups of threads and over CTAs."""
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=vp.NoSplitting())
    fs = [wobbly(vp, n, n, 0.5)]
    first, _ = fields(vp, p, fs, names)
    for _ in range(20):
        again, _ = fields(vp, p, fs, names)
        for name in names:
            assert np.array_equal(again[name], first[name])


@pytest.mark.gpu
def test_open_domain_skips_nan_sources(vp):
    """A filament with a NaN node does not reach the nodes of the others, and its pairs are not counted."""
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=vp.NoSplitting())
    good, bad = wobbly(vp, 40, 1), wobbly(vp, 30, 2)
    alone, _ = fields(vp, p, [good], ("velocity",))
    bad[7] = np.nan
    both, counts = fields(vp, p, [good, bad], ("velocity",))
    assert rel(both["velocity"][:40], alone["velocity"]) <= 1e-13
    assert counts == (69 * 3 * 40, 70 * 3 * 70)  # every source of the bad filament is NaN, one of its nodes


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("nodes", [31, 33])
def test_interleaved_interpolation(vp, oracle, m, nodes):
    """Footprints that outnumber the grid points four times: the grid of interleaved components; node counts that do
    not fill the last block."""
    rng = np.random.default_rng(1)
    fs = [vp.curves.ring(nodes, 0.8, L * rng.random(3), vp.curves.random_rotation(rng)) for _ in range(3 + 1200 // m ** 3)]
    p = params(vp, "mixed", L / 6, Ns=10, m=m)
    v, s, _ = oracle.compute_on_nodes(p, fs, velocity=True, streamfunction=True, LIA=False, shortrange=False)
    got, _ = fields(vp, p, fs, LIA=False, shortrange=False)
    assert sum(map(len, fs)) * 8 * m ** 3 >= 4 * 16 ** 3
    assert rel(got["velocity"], v) <= 2e-6 and rel(got["streamfunction"], s) <= 2e-6
