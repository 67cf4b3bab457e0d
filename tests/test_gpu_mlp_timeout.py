"""A tensor-core wait of the prefetch network that gave up (the state is set
from the host, nothing waits): no step is made from incomplete products, and
every synchronising call of that network, and of no other, says so once."""
import numpy as np
import pytest

import visualtur_b200 as vt

pytestmark = pytest.mark.gpu

DIMS, B = (12, 64, 96, 128), 32


def net(torch, seed):
    m = vt.MLP(DIMS, seed=seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.randn(B, DIMS[0], generator=g, device="cuda")
    y = (torch.rand(B, DIMS[3], generator=g, device="cuda") < 0.3).float()
    return m, x, y


def same(a, b):
    return all(np.array_equal(p, q) for l, k in zip(a, b) for p, q in zip(l, k))


@pytest.mark.parametrize("call", ["weights", "set_weights", "train_step", "gradients"])
def test_timeout_is_reported_and_no_step_is_made(call, cuda):
    m, x, y = net(cuda, 1)
    other, _, _ = net(cuda, 2)
    m.train_step(x, y, B, 1e-2)
    before = m.weights()
    m.debug_timeout()
    for _ in range(2):
        m.train_step(x, y, B, 1e-2, want_loss=False)
    other.train_step(x, y, B, 1e-2)          # another network's calls neither report nor clear it
    other.weights()
    with pytest.raises(vt.VtError) as e:
        {"weights": m.weights, "set_weights": lambda: m.set_weights(before),
         "train_step": lambda: m.train_step(x, y, B, 1e-2), "gradients": lambda: m.gradients(x, y, B)}[call]()
    assert e.value.status == vt.VT_ERR_TIMEOUT and "wait bound" in str(e.value)
    assert same(m.weights(), before)
    first = m.train_step(x, y, B, 1e-2)      # and on it goes
    assert not same(m.weights(), before)
    for _ in range(20):
        last = m.train_step(x, y, B, 1e-2)
    assert last < first
