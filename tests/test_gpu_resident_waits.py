"""Waits of the resident launch that run out, and small solvers beside one another."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import make_case
from supersonicflowsolver_b200 import meshgen
from supersonicflowsolver_b200.psst import Grid, PsstError, Solver

pytestmark = pytest.mark.gpu


def test_run_out_wait_behind_another_error_leaves_nothing_behind(tmp_path):
    """Temperatures below zero everywhere: every CTA reports its cells' state in the first stage,
    which waits for nothing (first order, local time steps from stage-start values), so that is
    the error of the call although every wait of the second stage then runs out. The calls after
    it, with a good state and the usual bound, equal those of a new solver, residual columns included."""
    m = meshgen.wedge2d(61, 23, 15.0)
    path, d, name = make_case(tmp_path, m, max_iter=1, flux=2, order=1, lc=1, rk_level=2, mach=2.5)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = 64, 1
    a, b = Solver(g, sc), Solver(g, sc)
    assert a.schedule_info()["wavefront"] and a.schedule_info()["blocks"] > 1
    bad = prim.copy()
    bad[g.nvol:2 * g.nvol] *= -1.0
    a.set_state(prim)
    a.explicit_solve(3)
    a.set_state(bad)
    a.set_wait_limit(0)
    with pytest.raises(PsstError) as e:
        a.explicit_solve(2)
    assert e.value.status in (5, 6)  # not PSST_ERR_TIMEOUT
    a.set_wait_limit(-1)
    for s in (a, b):
        s.set_state(prim)
    for n in (3, 2):
        la, ra = a.explicit_solve(n)
        lb, rb = b.explicit_solve(n)
        assert np.array_equal(la, lb) and np.array_equal(ra, rb)
        for x, y in zip(a.get_state(with_w=True), b.get_state(with_w=True)):
            assert np.array_equal(x, y)


HARNESS = r"""
#include "resident.cuh"
using namespace psst;
// One warp: a wait that runs out (its limit is 1 ns, 4096 attempts at most), then a wait that ends after one
// attempt. out[0], out[1]: whether the operation may go on after each.
__global__ void k(unsigned *sync, int32_t *err, int *out) {
    bool ok = true;
    Waiter first{sync, err, 1, 0, 0u};
    for (int i = 0; i < 4096 && still_waiting(true, ok, first, 0); ++i) {}
    if (threadIdx.x == 0) out[0] = ok;
    Waiter second{sync, err, 1000000000, 0, 0u};
    for (int i = 0; i < 2 && still_waiting(i == 0, ok, second, 0); ++i) {}
    if (threadIdx.x == 0) out[1] = ok;
}
extern "C" int run(int *out) {
    unsigned *sync;
    int32_t *err;
    int *o;
    if (cudaMalloc(&sync, kWfSyncWords * 4) || cudaMalloc(&err, 16) || cudaMalloc(&o, 8)) return 1;
    cudaMemset(sync, 0, kWfSyncWords * 4);
    cudaMemset(err, 0, 16);
    k<<<1, 32>>>(sync, err, o);
    const int e = cudaMemcpy(out, o, 8, cudaMemcpyDeviceToHost);
    cudaFree(sync), cudaFree(err), cudaFree(o);
    return e;
}
"""


def test_a_wait_given_up_stays_given_up(tmp_path):
    """Cells of more than four faces wait once per four: a later wait that is met does not take back
    that an earlier one ran out."""
    src, lib = tmp_path / "h.cu", str(tmp_path / "h.so")
    src.write_text(HARNESS)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["nvcc", "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(root, "supersonicflowsolver_b200", "csrc"), "-I", os.path.join(root, "include"),
                    "-shared", "-Xcompiler", "-fPIC", str(src), "-o", lib], check=True)
    out = (ctypes.c_int * 2)()
    assert ctypes.CDLL(lib).run(out) == 0
    assert list(out) == [0, 0]


def test_solvers_on_threads_of_their_own(tmp_path):
    """Four solvers, two of them with launches of more than half of the device's CTAs and one
    sequential, step at the same time: nothing waits for another's launch beyond its end, and
    every result is that of the solver alone."""
    import threading

    cases = []
    for i, (nx, ny, bits, mode) in enumerate([(120, 40, 64, 1), (180, 60, 32, 1), (60, 20, 64, 1), (60, 20, 64, 0)]):
        p = tmp_path / str(i)
        p.mkdir()
        path, d, name = make_case(p, meshgen.wedge2d(nx, ny, 12.0), max_iter=1, flux=3, order=2, limiter=4, lc=1)
        g = Grid.read_fluent(path)
        sc, prim = g.read_case(d, name)
        sc.precision, sc.lc1_mode = bits, mode
        s = Solver(g, sc)
        assert s.schedule_info()["wavefront"]
        s.set_wait_limit(2_000_000_000)
        cases.append((s, prim))

    def steps(s, prim, out):
        s.set_state(prim)
        out += [s.explicit_solve(20) for _ in range(10)]
        out.append((s.get_state(),))

    alone, beside = [[] for _ in cases], [[] for _ in cases]
    for (s, prim), out in zip(cases, alone):
        steps(s, prim, out)
    threads = [threading.Thread(target=steps, args=c + (out,)) for c, out in zip(cases, beside)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, beside):
        assert len(a) == len(b) == 11
        for x, y in zip(a, b):
            for v, w in zip(x, y):
                assert np.array_equal(v, w)
