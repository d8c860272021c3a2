"""Distinct handles used at the same time by different threads, which the C ABI allows: calls whose kernels need
different amounts of shared memory do not disturb one another."""

import math
import re
import threading
from pathlib import Path

import numpy as np
import pytest

L = 2 * math.pi


def run_together(*jobs):
    """Every job in a thread of its own; the first error any of them raised."""
    errors = []
    start = threading.Barrier(len(jobs))

    def body(job):
        try:
            start.wait()
            job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_shared_memory_limits_are_fixed():
    """cudaFuncSetAttribute changes the function, for every handle of the process: its sizes are constants (or sizes of
    types), never what one call needs, or a call with less could fail a concurrent launch that needs more."""
    csrc = Path(__file__).resolve().parents[1] / "vortexpasta.jl_b200" / "csrc"
    sizes = [m for f in csrc.glob("*.cu*") for m in
             re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*\(int\)\s*\(?(\w+)", f.read_text())]
    assert len(sizes) >= 6
    # k...: constants; tsmem, psmem: the size of a type and of the plane kernel's tile, one per template instance
    assert all(s.startswith("k") or s in ("tsmem", "psmem") for s in sizes), sizes


def test_no_lazily_filled_statics():
    """A static container of a function that is filled on first use would be filled by several threads at once: statics
    are const (initialised under the compiler's guard), or guarded by a mutex as the copy pool."""
    csrc = Path(__file__).resolve().parents[1] / "vortexpasta.jl_b200" / "csrc"
    found = [(f.name, line.strip()) for f in csrc.glob("*.cu*") for line in f.read_text().splitlines()
             if re.match(r"\s+static (?!const|assert)[\w:<>,\s*&]+;", line)]
    assert found == [("api.cu", "static std::mutex mu;")], found


@pytest.mark.gpu
def test_filaments_of_different_lengths_in_two_threads(vp):
    """Spline solves of 1000- and 30-node filaments (188 KB and 6 KB of shared memory a block) from two threads."""
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=vp.NoSplitting())

    def job(n):
        t = 2 * math.pi * (np.arange(n) + 0.5) / n
        x = np.stack([np.cos(t), np.sin(t), 0.1 * np.cos(2 * t)], axis=1)
        offsets = np.array([0, n])

        def run():
            cache = vp.init_cache(p)
            try:
                for _ in range(3000):
                    cache.set_filaments_flat(x, offsets)
                d1 = cache.pointdata()["d1"]
                assert np.allclose(np.linalg.norm(d1, axis=1), 1.0, atol=1e-2)
            finally:
                cache.close()
        return run

    run_together(job(1000), job(30), job(1000), job(30))


@pytest.mark.gpu
def test_spectra_of_different_sizes_in_two_threads(vp):
    """Spectra of 16,384 and of 6,200 bins (128 KB and 48.4 KB of shared memory) from two threads."""
    from vortexpasta_b200 import _lib
    lib = _lib.load()
    p = vp.ParamsBiotSavart(Gamma=1.0, a=1e-8, splitting=vp.GaussianSplitting(Ls=L, beta=3.5, rcut=L / 4))
    fs = [vp.curves.ring(40, 1.0, np.zeros(3), np.eye(3))]

    def job(nk):
        def run():
            cache = vp.init_cache(p)
            try:
                out = {"velocity": [np.zeros((40, 3))]}
                vp.compute_on_nodes_(out, cache, fs)
                e = np.zeros(nk)
                for _ in range(500):
                    _lib.check(lib.vpbs_spectrum(cache.handle, 0, 1.0, _lib.dptr(e), nk), cache.handle, "spectrum")
                assert e.sum() > 0
            finally:
                cache.close()
        return run

    run_together(job(16384), job(6200))
