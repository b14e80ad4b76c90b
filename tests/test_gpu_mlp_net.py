"""The network's fused kernels at the edges of their tiles (128 points a CTA, 64-row
boxes, 256-row partial sums, 64 partial sums a pass)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    t = np.stack([np.sin(2 * x[:, 2]) * x[:, 0], x[:, 3] ** 2, 0.3 * x[:, 1] * x[:, 2], np.cos(x[:, 2] + x[:, 3])],
                 axis=1).astype(np.float32)
    return x, t


@pytest.mark.parametrize("n", [1, 63, 127, 128, 129, 300, 19201])
def test_forward_of_a_point_does_not_depend_on_its_batch(n):
    from supersonicflowsolver_b200.mlp import MLP

    net = MLP(seed=3)
    x = torch.from_numpy(data(n, n)[0]).cuda()
    y = net.forward(x)
    for i in sorted({0, n // 2, max(n - 65, 0), n - 1}):
        assert torch.equal(y[i:i + 1], net.forward(x[i:i + 1].contiguous())), i
    # BF16 operands against FP64 arithmetic on the same rounded operands: the 2e-3 of the batch of 300
    oy = mo.loss_and_grads(net.params(), x[:300].cpu().numpy(), data(n, n)[1][:300], bf16_points=True)[2]
    assert np.linalg.norm(y[:300].cpu().numpy() - oy) <= 2e-3 * np.linalg.norm(oy)


@pytest.mark.parametrize("n", [1, 64, 65, 127, 129, 255, 257, 500, 64 * 256 + 1, 3 * 64 * 256 - 70])
def test_gradients(n):
    from supersonicflowsolver_b200.mlp import MLP

    net = MLP(seed=12)
    big = data(700, 1)
    net.gradients(*(torch.from_numpy(v).cuda() for v in big))  # a workspace with older, longer contents
    x, t = data(n, 2)
    g, loss = net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    p = net.params()
    oloss, og, _ = mo.loss_and_grads(p, x, t, bf16_points=True)
    # five layers of BF16 deltas, each within half an ulp (2^-9) or a flipped rounding (2^-8) of the
    # oracle's: 5 * 2^-8 = 2e-2 of the norm
    assert abs(loss - oloss) <= 2e-3 * oloss
    off = 0
    for l in range(6):
        for k in (mo.DOUT[l] * mo.DIN[l], mo.DOUT[l]):
            a, b = g[off:off + k], og[off:off + k]
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), (l, k)
            off += k


def test_train_step_is_adam_on_the_gradients():
    """Two steps, FP32 Adam restated in FP64: the update is at most 1.1 lr, formed and
    added in FP32 (a few 2^-24 of the update and half an ulp of the parameter, below 1)."""
    from supersonicflowsolver_b200.mlp import MLP

    net, ref = MLP(seed=4), MLP(seed=4)
    n, lr = 64 * 256 + 300, 1e-3
    m = v = np.zeros(net.n)
    for k in range(2):
        x, t = (torch.from_numpy(q).cuda() for q in data(n, 7 + k))
        p = net.params().astype(np.float64)
        assert np.array_equal(p, ref.params())
        g, loss = ref.gradients(x, t)
        assert net.train_step(x, t, lr) == loss
        ref.train_step(x, t, lr)
        m = 0.9 * m + 0.1 * g.astype(np.float64)
        v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
        want = p - lr * (m / (1 - 0.9 ** (k + 1))) / (np.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
        # float32 0.9 and 0.999 differ from the decimal ones by 2^-24 and 2^-24 / 0.001 relative to 1 - b:
        # 2.4e-7 and 2e-5 in the two corrections, which cancel against those of m and v only in part
        assert np.abs(net.params() - want).max() <= 2e-5 * 1.1 * lr + 2.0 ** -24


HARNESS = r"""
#include <cuda_runtime.h>
#include "exact.cuh"
__global__ void k(const float *a, const float *b, float *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = psst::rn_div(a[i], b[i]);
}
extern "C" int run(const float *a, const float *b, float *q, int n) {
    float *d[3];
    for (int i = 0; i < 3; ++i)
        if (cudaMalloc(&d[i], n * 4)) return 1;
    cudaMemcpy(d[0], a, n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], b, n * 4, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d[0], d[1], d[2], n);
    const int e = cudaMemcpy(q, d[2], n * 4, cudaMemcpyDeviceToHost);
    for (int i = 0; i < 3; ++i) cudaFree(d[i]);
    return e;
}
"""


def test_silu_quotients_have_the_bits_of_the_division(tmp_path):
    """z / (1 + e^-z) and 1 / (1 + e^-z) over the range that takes the straight-line quotient."""
    import ctypes
    import os
    import subprocess

    src, lib = tmp_path / "h.cu", str(tmp_path / "h.so")
    src.write_text(HARNESS)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "supersonicflowsolver_b200", "csrc")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", csrc, "-shared",
                    "-Xcompiler", "-fPIC", str(src), "-o", lib], check=True)
    L = ctypes.CDLL(lib)
    rng = np.random.default_rng(0)
    n = 1 << 22
    z = np.concatenate([rng.uniform(-87, 87, n), rng.normal(0, 2, n)]).astype(np.float32)
    b = (np.float32(1) + np.exp(-z)).astype(np.float32)
    for a in (z, np.ones_like(z)):
        q = np.empty_like(z)
        assert L.run(*(v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, q)), len(z)) == 0
        assert np.array_equal(q, a / b)
