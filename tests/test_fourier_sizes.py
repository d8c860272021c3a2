"""The pruned transforms of the long range (csrc/fourier.cu) over grid sizes: every radix and number of
passes, rows that are odd or even in number, lines shorter and longer than one tile, periods of
different lengths, and both fields from one transform.  The long-range fields at the nodes (with a weak
filter, so that every kept mode counts) against the CPU restatement; FP64 to 1e-10 as everywhere, mixed to
2e-6 (sixteen times the 1.2e-7 of the 32-bit grid sums and transforms; a wrong twiddle or row is above 1e-3)."""

import math

import numpy as np
import pytest

L = 2 * math.pi

# (Ns, sigma): FFT sizes 8 .. 2250 per dimension, with 2, 3 and 4 passes, radices 2 .. 32
SIZES = [((6, 6, 6), 1.3), ((12, 17, 31), 1.5), ((32, 20, 18), 1.5), ((50, 30, 36), 1.5), ((33, 48, 40), 2.0),
         ((54, 100, 25), 1.25), ((120, 16, 12), 2.0), ((16, 160, 14), 1.5), ((14, 12, 192), 1.5), ((256, 12, 10), 1.5),
         ((12, 256, 12), 1.5), ((10, 14, 256), 1.5), ((20, 12, 512), 1.5), ((400, 10, 12), 1.25), ((12, 10, 500), 1.25),
         # tiles of one line; lines too long for a block and a packed length of one factor (cuFFT)
         ((12, 10, 1360), 1.5), ((12, 10, 1500), 1.5), ((6, 12, 10), 1.5),
         # z lines of 1024 (two passes in FP32) and 1620 (too many threads for three components: cuFFT)
         ((12, 10, 682), 1.5), ((12, 10, 1080), 1.5)]


def system(vp):
    rng = np.random.default_rng(8)
    return [vp.curves.ring(n, 0.7 + 0.5 * rng.random(), L * rng.random(3), vp.curves.random_rotation(rng)) for n in (9, 24, 31)]


def params(vp, Ns, sigma, Ls=(L, 1.25 * L, 0.8 * L), **kw):
    m = 3 if min(Ns) < 10 else 4
    return vp.ParamsBiotSavart(Gamma=1.3, a=1e-8, splitting=vp.GaussianSplitting(Ls=Ls, alpha=12.0, rcut=L / 4, Ns=Ns),
                               backend_long=vp.NonuniformFFTsBackend(sigma, m), **kw)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("Ns,sigma", SIZES)
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 2e-6)])
def test_long_range_over_grid_sizes(vp, oracle, Ns, sigma, precision, tol):
    fs = system(vp)
    p = params(vp, Ns, sigma, precision=precision)
    v, s, _ = oracle.compute_on_nodes(p, fs, velocity=True, streamfunction=True, LIA=False, shortrange=False)
    cache = vp.init_cache(p)
    try:
        for names in (("velocity", "streamfunction"), ("velocity",), ("streamfunction",)):
            out = {n: [np.zeros((len(f), 3)) for f in fs] for n in names}
            vp.compute_on_nodes_(out, cache, fs, LIA=False, shortrange=False)
            for n, want in (("velocity", v), ("streamfunction", s)):
                if n in out:
                    assert rel(np.concatenate(out[n]), want) <= tol, (n, names)
    finally:
        cache.close()


@pytest.mark.gpu
@pytest.mark.parametrize("Ns", [72, 170, 288])
def test_mixed_transforms_do_not_shrink(vp, Ns):
    """FFT sizes 108, 256, 432 = 2^a 3^b.  With the transforms' constants rounded to FP32 every pass takes 1e-8 to 2e-8 of
    the amplitude, and the smooth streamfunction is off by 1.5e-7 to 1.8e-7; rounding that averages out leaves 0.5e-7
    to 0.9e-7."""
    rng = np.random.default_rng(6)
    fs = [vp.curves.ring(200, 0.8 + 0.7 * rng.random(), L * rng.random(3), vp.curves.random_rotation(rng)) for _ in range(100)]
    got = {}
    for precision in ("fp64", "mixed"):
        sp = vp.GaussianSplitting(Ls=L, alpha=Ns / 7.0, rcut=L / 5, Ns=Ns)
        p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=sp, backend_long=vp.NonuniformFFTsBackend(1.5, 5), precision=precision)
        cache = vp.init_cache(p)
        out = [np.zeros((200, 3)) for _ in fs]
        vp.compute_on_nodes_({"streamfunction": out}, cache, fs, LIA=False, shortrange=False)
        cache.close()
        got[precision] = np.concatenate(out)
    assert rel(got["mixed"], got["fp64"]) <= 1.2e-7


@pytest.mark.gpu
def test_memory_of_grids_without_a_plan(vp):
    """Grids that take cuFFT hold three real values a point, not the four of the interleaved layout, which they never
    use: 36 bytes a point with the two complex grids, and cuFFT's work space of 24."""
    import torch
    p = params(vp, (256, 256, 1080), 1.5, precision="mixed")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    cache = vp.init_cache(p)
    used = before - torch.cuda.mem_get_info()[0]
    cache.close()
    points = 384 * 384 * 1620
    modes = 3 * 16 * 129 * 256 * 1080
    assert used - modes < 62 * points
