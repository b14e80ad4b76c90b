"""FP32 arithmetic of the production passes: roundings that the compiler could choose are pinned."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import make_case
from supersonicflowsolver_b200 import meshgen
from supersonicflowsolver_b200.psst import Grid, Solver

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "kernels.cuh"
using namespace psst;
// face i between the cells 2 i and 2 i + 1, of area 1; s: p, T, u.. of both and the normal, [13][n]
__global__ void k_setup(const float *s, int n, float rm, FaceRec<float, 3> *fr, CellRec<float> *c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int j = 0; j < 2; ++j) {
        const float *q = s + (int64_t)j * 5 * n + i;
        const float u[3] = {q[2 * (int64_t)n], q[3 * (int64_t)n], q[4 * (int64_t)n]};
        c[2 * i + j] = pack<float, 3>(q[0], q[n], q[0] / (rm * q[n]), u);
    }
    FaceRec<float, 3> f{};
    f.c0 = 2 * i;
    f.c1 = 2 * i + 1;
    f.S = 1.0;
    for (int d = 0; d < 3; ++d) f.n[d] = s[(10 + d) * (int64_t)n + i];
    fr[i] = f;
}
template <int FLUX, int REC>
int faces(const float *s, int n, float *out) {
    using FO = FaceOut<float, 3>;
    const Gas gas{287.0, 1004.5, 717.5, 1.4};
    const int nb = (n + 255) / 256;
    float *ds;
    FaceRec<float, 3> *fr;
    CellRec<float> *c;
    char *cols;
    DevGrid g{};
    DevState<float> st{};
    DevWork<float> wk{};
    if (cudaMalloc(&ds, (size_t)13 * n * 4) || cudaMalloc(&fr, n * sizeof *fr) || cudaMalloc(&c, 2 * n * sizeof *c) ||
        cudaMalloc(&cols, FaceCols<float, 3, REC>::bytes(n)) || cudaMalloc(&wk.grec, 2 * n * sizeof(GradRec<float, 3>)) ||
        cudaMalloc(&wk.fout, n * sizeof(FO)) || cudaMalloc(&wk.err, 16))
        return 1;
    cudaMemcpy(ds, s, (size_t)13 * n * 4, cudaMemcpyHostToDevice);
    cudaMemset(wk.grec, 0, 2 * n * sizeof(GradRec<float, 3>));
    cudaMemset(wk.err, 0, 16);
    k_setup<<<nb, 256>>>(ds, n, (float)gas.rm, fr, c);
    g.nint = g.nall = 2 * n;
    g.nface = g.nfi = n;
    g.frec = fr;
    g.fcols = cols;
    st.rec = c;
    k_face_columns<float, 3, REC><<<nb, 256>>>(g, cols);
    k_face<float, 3, FLUX, REC, 1, 1><<<nb, 256>>>(g, st, wk, gas);
    int32_t err = 0;
    cudaMemcpy(&err, wk.err, 4, cudaMemcpyDeviceToHost);
    const int e = cudaMemcpy(out, wk.fout, n * sizeof(FO), cudaMemcpyDeviceToHost);
    cudaFree(ds), cudaFree(fr), cudaFree(c), cudaFree(cols), cudaFree(wk.grec), cudaFree(wk.fout), cudaFree(wk.err);
    return e ? e : err;
}
extern "C" int run(int flux, int rec, const float *s, int n, float *out) {
    if (flux == 2) return rec ? faces<2, 2>(s, n, out) : faces<2, 0>(s, n, out);
    return rec ? faces<3, 2>(s, n, out) : faces<3, 0>(s, n, out);
}
"""


@pytest.fixture(scope="module")
def face_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("face")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-prec-sqrt=false", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "supersonicflowsolver_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-shared", "-Xcompiler", "-fPIC", str(d / "h.cu"), "-o",
                    str(d / "h.so")], check=True)
    return ctypes.CDLL(str(d / "h.so"))


@pytest.mark.parametrize("rec", [0, 2], ids=["first_order", "muscl"])
@pytest.mark.parametrize("flux", [2, 3], ids=["hll", "hllc"])
def test_energy_flux_rounds_the_enthalpy_once(face_lib, flux, rec):
    """Supersonic faces (the normal within 30 degrees of a Mach 2.5 to 4 flow) take the flux of the
    side upwind: mass flux rho v, energy flux (rho v) H, where cp T + (v.v) / 2 is rounded once (a
    rounding of cp T before the sum is 20% more error in H). v.v is a chain of fused products; in
    64 bits its sums may round at the 53rd bit first, which changes a 24-bit result one time in 2^28."""
    n = 1 << 16
    rng = np.random.default_rng(10 * flux + rec)
    f32 = np.float32
    base = np.concatenate([1e5 * rng.uniform(0.3, 3.0, (1, n)), rng.uniform(200.0, 400.0, (1, n)),
                           rng.uniform(1000.0, 1300.0, (1, n)), rng.uniform(-100.0, 100.0, (2, n))])
    sides = [base * (1.0 + 0.01 * rng.normal(size=base.shape)) for _ in range(2)]
    nn = np.concatenate([np.ones((1, n)), rng.uniform(-0.4, 0.4, (2, n))])
    s = np.ascontiguousarray(np.concatenate(sides + [nn / np.linalg.norm(nn, axis=0)]), dtype=f32)
    out = np.empty((n, 8), f32)
    assert face_lib.run(flux, rec, s.ctypes.data_as(ctypes.c_void_p), n, out.ctypes.data_as(ctypes.c_void_p)) == 0
    T, u = s[6].astype(np.float64), s[7:10].astype(np.float64)  # the upwind side is the face's second cell
    vs = (u[0] * u[0]).astype(f32).astype(np.float64)
    for d in (1, 2):
        vs = (u[d] * u[d] + vs).astype(f32).astype(np.float64)
    H = (np.float64(f32(1004.5)) * T + 0.5 * vs).astype(f32)
    assert np.array_equal(out[:, 4], out[:, 3] * H)


@pytest.mark.parametrize("mesh", ["quads", "shuffled", "tets"])
def test_resident_gradient_has_the_bits_of_the_pass(tmp_path, mesh):
    """Four faces a cell, FP32: the gradients that the resident launch forms from a state are those of the
    gradient pass (one fused product a face, coefficients rounded once)."""
    m = {"quads": lambda: meshgen.wedge2d(61, 23, 15.0), "tets": lambda: meshgen.wedge3d(9, 5, 3, 12.0, tets=True),
         "shuffled": lambda: meshgen.wedge2d(30, 10, 15.0, jitter=0.15, seed=3, shuffle_seed=1, interior_first=True)}[mesh]()
    path, d, name = make_case(tmp_path, m, max_iter=4, flux=3, order=2, limiter=3, lc=1, mach=3.0 if m.dim == 3 else 2.5)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = 32, 1
    a, b = Solver(g, sc), Solver(g, sc)
    b.use_wavefront(False)
    assert a.schedule_info()["wavefront"]
    b.set_state(prim)
    b.explicit_solve(3)
    start = b.get_state()  # FP32 values: both solvers start from the same bits
    got = []
    for s in (a, b):
        s.set_state(start)
        s.explicit_solve(1)
        got.append([s.get(k) for k in ("grad_p", "grad_T", "grad_u")])
    for x, y in zip(*got):
        assert np.abs(y).max() > 0 and np.array_equal(x, y)
