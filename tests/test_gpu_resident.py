"""The resident launch (resident.cuh): whole calls as one persistent launch.

* the parallel time-step modes on small meshes: state, conservative state, time
  step, gradients and L-inf columns equal those of the pass kernels bit for bit
  in FP64 (the RMS column to the order of its sum), on meshes of one item, of a
  partly filled last item, with more than four faces a cell, with a cell face
  order other than the face-loop order, over all fluxes, reconstructions and
  time steps;
* FP32: both forms round each operation to FP32 in their own order. One stage
  forms a cell's update from some 200 roundings of 2^-24 each, most of them
  averaging out; 6 iterations of 4 stages stay below 24 * 200 * 2^-24 = 2.9e-4
  of each variable's largest value even if all of them added up;
* a call whose norm rows exceed the bound of one launch equals the same
  iterations in several calls;
* exact.cuh's straight-line division and square root equal the IEEE results on
  random and hard operands.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import make_case
from supersonicflowsolver_b200 import meshgen
from supersonicflowsolver_b200.psst import Grid, Solver

pytestmark = pytest.mark.gpu

MESHES = {
    "two_cells": lambda: meshgen.wedge2d(2, 1, 15.0),
    "item_33": lambda: meshgen.wedge2d(11, 3, 15.0),  # 33 cells: an item and one cell
    "quads": lambda: meshgen.wedge2d(61, 23, 15.0),
    "shuffled": lambda: meshgen.wedge2d(30, 10, 15.0, jitter=0.15, seed=3, shuffle_seed=1, interior_first=True),
    "adapted": lambda: meshgen.wedge2d_adapted(24, 9, 15.0, refine_frac=0.2, seed=5),
    "tets": lambda: meshgen.wedge3d(9, 5, 3, 12.0, tets=True),
    "hexes": lambda: meshgen.wedge3d(9, 5, 3, 12.0, tets=False, interior_first=True),
}
CASES = [
    ("two_cells", dict(flux=3, order=2, limiter=5, lc=1)),
    ("item_33", dict(flux=2, order=2, limiter=4, lc=1)),
    ("quads", dict(flux=3, order=2, limiter=4, lc=1)),
    ("quads", dict(flux=1, order=1, lc=2, rk_level=1, cfl=0.4)),
    ("quads", dict(flux=2, order=2, limiter=1, lc=0, rk_level=2)),
    ("shuffled", dict(flux=1, order=2, limiter=3, lc=1, grad=2)),
    ("shuffled", dict(flux=3, order=2, limiter=2, lc=2)),
    ("adapted", dict(flux=3, order=2, limiter=5, lc=1)),
    ("tets", dict(flux=3, order=2, limiter=3, lc=1)),
    ("tets", dict(flux=2, order=2, limiter=5, lc=2, grad=2)),
    ("hexes", dict(flux=1, order=2, limiter=4, lc=1)),
]


def pair(tmp_path, mesh, bits, **ckw):
    m = MESHES[mesh]()
    path, d, name = make_case(tmp_path, m, max_iter=6, mach=3.0 if m.dim == 3 else 2.5, **ckw)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = bits, 1
    a, b = Solver(g, sc), Solver(g, sc)
    b.use_wavefront(False)
    return g, a, b, prim


@pytest.mark.parametrize("mesh,ckw", CASES, ids=["%s-%d" % (c[0], i) for i, c in enumerate(CASES)])
@pytest.mark.parametrize("bits", [64, 32])
def test_resident_equals_passes(tmp_path, mesh, ckw, bits):
    g, a, b, prim = pair(tmp_path, mesh, bits, **ckw)
    assert a.schedule_info()["wavefront"] == (not (bits == 64 and mesh == "hexes"))
    assert not b.schedule_info()["wavefront"]
    a.set_state(prim)
    b.set_state(prim)
    for n in (1, 3, 2):
        la, ra = a.explicit_solve(n)
        lb, rb = b.explicit_solve(n)
        pa, wa = a.get_state(with_w=True)
        pb, wb = b.get_state(with_w=True)
        if bits == 64:
            assert np.array_equal(la, lb)
            np.testing.assert_allclose(ra, rb, rtol=1e-12, atol=0)
            assert np.array_equal(pa, pb) and np.array_equal(wa, wb)
            assert np.array_equal(a.get("dt"), b.get("dt")) and np.array_equal(a.get("rho"), b.get("rho"))
            if ckw.get("order") == 2:
                for k in ("grad_p", "grad_T", "grad_u"):
                    assert np.array_equal(a.get(k), b.get(k)), k
        else:
            nv = g.nvol
            speed = np.abs(prim[2 * nv:]).max()
            for q in range(2 + g.dim):
                x, y = pa[q * nv:(q + 1) * nv], pb[q * nv:(q + 1) * nv]
                assert np.max(np.abs(x - y)) <= 2.9e-4 * (np.abs(prim[q * nv:(q + 1) * nv]).max() if q < 2 else speed)
    assert a.iter == b.iter


def test_long_call_in_several_launches(tmp_path):
    """120 x 80 quads: an iteration's norm rows are 77 kB, so 3600 iterations take two launches."""
    m = meshgen.wedge2d(120, 80, 12.0)
    path, d, name = make_case(tmp_path, m, max_iter=1, flux=2, order=1, lc=1, rk_level=4, mach=2.5)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = 64, 1
    a, b = Solver(g, sc), Solver(g, sc)
    a.set_state(prim)
    b.set_state(prim)
    la, ra = a.explicit_solve(3600)
    assert a.last_stats()[0] == 2
    parts = [b.explicit_solve(1200) for _ in range(3)]
    assert np.array_equal(la, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(ra, np.concatenate([p[1] for p in parts]))
    assert np.array_equal(a.get_state(), b.get_state())


HARNESS = r"""
#include "exact.cuh"
template <typename R> __global__ void k(const R *a, const R *b, R *q, R *r, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = psst::lin_quot(a[i], b[i], psst::lin_recip(b[i]));
    r[i] = psst::lin_sqrt(b[i]);
}
template <typename R> int run(const R *a, const R *b, R *q, R *r, int n) {
    R *d;
    if (cudaMalloc(&d, 4 * sizeof(R) * n)) return 1;
    cudaMemcpy(d, a, n * sizeof(R), cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, n * sizeof(R), cudaMemcpyHostToDevice);
    k<R><<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, d + 3 * n, n);
    cudaMemcpy(q, d + 2 * n, n * sizeof(R), cudaMemcpyDeviceToHost);
    cudaMemcpy(r, d + 3 * n, n * sizeof(R), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)cudaGetLastError();
}
extern "C" int run64(const double *a, const double *b, double *q, double *r, int n) { return run(a, b, q, r, n); }
extern "C" int run32(const float *a, const float *b, float *q, float *r, int n) { return run(a, b, q, r, n); }
"""


def test_straight_line_division_and_root(tmp_path):
    """FP64: bit-equal to IEEE division and square root on random operands over
    the range, on quotients next to rounding boundaries (a = the product of b and
    a boundary, rounded) and roots next to them (x = a boundary squared,
    rounded), powers of two and their neighbours. FP32: the corrected quotient
    (root) is within half an ulp plus the reciprocal's own error of the
    correction, 2^-22 of half an ulp: at most one ulp from the IEEE result."""
    src, lib = tmp_path / "h.cu", tmp_path / "h.so"
    src.write_text(HARNESS)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "supersonicflowsolver_b200", "csrc")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-I", csrc,
                    "-shared", "-Xcompiler", "-fPIC", "-o", str(lib), str(src)], check=True)
    L = ctypes.CDLL(str(lib))
    rng = np.random.default_rng(0)
    n = 1 << 20

    def call(fn, a, b):
        q, r = np.empty_like(a), np.empty_like(b)
        assert fn(*(v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, q, r)), len(a)) == 0
        return q, r

    def mant(k):
        return 1.0 + rng.integers(0, 1 << 52, k).astype(np.float64) * 2.0 ** -52

    for trial in range(4):
        b = mant(n) * 2.0 ** rng.integers(-350, 350, n)
        a = rng.choice([-1.0, 1.0], n) * mant(n) * 2.0 ** rng.integers(-350, 350, n)
        # quotients next to a boundary between two doubles
        half = n // 4
        m = rng.integers(1 << 52, 1 << 53, half)
        a[:half] = [float(int(2 * int(x) + 1) * int(y)) for x, y in zip(m, (mant(half) * 2.0 ** 52).astype(np.int64))] \
            if trial == 0 else a[:half]
        if trial == 0:
            b[:half] = np.round(a[:half] / (2.0 * m + 1.0))
        # radicands next to a boundary squared
        b[half:2 * half] = [float((2 * int(x) + 1) ** 2) for x in rng.integers(1 << 52, 1 << 53, half)]
        b[2 * half:2 * half + 600] = np.repeat(2.0 ** np.arange(-100, 100), 3) * np.tile(
            [1.0, 1.0 + 2.0 ** -52, 1.0 + 2.0 ** -51], 200)
        # an ulp below round numbers: low words of ones only
        b[3 * half:3 * half + 2000] = np.nextafter(rng.integers(1, 1 << 20, 2000).astype(np.float64), 0.0)
        low = np.uint64((1 << 52) - 1)
        ones = (b.view(np.uint64) & low) == low  # den_ok sends these elsewhere
        q, r = call(L.run64, a, b)
        assert np.array_equal(q[~ones], (a / b)[~ones])
        assert np.array_equal(r, np.sqrt(b))
    a32, b32 = (mant(n) * 2.0 ** rng.integers(-50, 50, n)).astype(np.float32), (mant(n) * 2.0 ** rng.integers(-50, 50, n)).astype(np.float32)
    q, r = call(L.run32, a32, b32)
    for x, y in ((q, a32 / b32), (r, np.sqrt(b32))):
        assert np.max(np.abs(x.view(np.int32).astype(np.int64) - y.view(np.int32).astype(np.int64))) <= 1
