"""Waits of the network's kernels that run out, and waits that a call does not have."""
import numpy as np
import pytest

from test_gpu_mlp_net import data

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 200, 500, 19201])
def test_waits_that_run_out_are_reported_and_change_nothing(n):
    """No polls at all: every wait gives up at once. One poll and a few: some waits are met and others
    run out, at any point of the kernels; a call then fails with PSST_ERR_TIMEOUT or is right."""
    from supersonicflowsolver_b200.mlp import MLP
    from supersonicflowsolver_b200.psst import PsstError

    net, ref = MLP(seed=6), MLP(seed=6)
    x, t = (torch.from_numpy(q).cuda() for q in data(n, 3))
    y = ref.forward(x)
    assert net.train_step(x, t, 1e-3) == ref.train_step(x, t, 1e-3)
    ref_y = ref.forward(x)
    assert not torch.equal(y, ref_y)
    for polls in (0, 0, 1, 2, 4, 16, 0):
        net.set_wait_polls(polls)
        try:
            assert torch.equal(net.forward(x), ref_y) and polls > 0
        except PsstError as e:
            assert e.status == 7
        before = net.params()
        try:
            loss = net.train_step(x, t, 1e-3)
            assert polls > 0 and loss == ref.train_step(x, t, 1e-3)
            ref_y = ref.forward(x)
        except PsstError as e:
            assert e.status == 7
            assert np.array_equal(net.params(), before)
    net.set_wait_polls(-1)
    for _ in range(2):  # Adam's moments and step as well
        assert net.train_step(x, t, 1e-3) == ref.train_step(x, t, 1e-3)
    assert np.array_equal(net.params(), ref.params())
    assert torch.equal(net.forward(x), ref.forward(x))


def test_gradients_wait_for_nothing_on_the_default_stream():
    """On a stream of its own a call does not wait for what the legacy default stream has to do (a spin
    of some 200 ms, against a call of a millisecond)."""
    from supersonicflowsolver_b200.mlp import MLP

    if not hasattr(torch.cuda, "_sleep"):
        pytest.skip("torch.cuda._sleep not available")
    net = MLP(seed=2)
    x, t = (torch.from_numpy(q).cuda() for q in data(300, 4))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        g0, l0 = net.gradients(x, t)
    torch.cuda._sleep(400_000_000)
    done = torch.cuda.Event()
    done.record()
    with torch.cuda.stream(side):
        g1, l1 = net.gradients(x, t)
    assert not done.query()
    assert np.array_equal(g0, g1) and l0 == l1
    torch.cuda.synchronize()
