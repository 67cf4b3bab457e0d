"""Training batches of more rows than one grid dimension of 16-row blocks
holds (65535 * 16)."""
import numpy as np
import pytest

import visualtur_b200 as vt
from test_gpu_mlp import cpu_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [65535 * 16, 65535 * 16 + 1, 2000003])
def test_large_training_batch(batch, cuda):
    """Gradients against the CPU implementation.  A gradient is summed over
    the batch in FP32, sixteen rows a step: at most an ulp (2^-23) of the sum
    a step on top of the 2e-3 of the other shapes."""
    torch = cuda
    dims = (4, 8, 8, 8)
    m = vt.MLP(dims, seed=4)
    rng = np.random.default_rng(8)
    x = rng.standard_normal((batch, dims[0])).astype(np.float32)
    y = (rng.random((batch, dims[3])) < 0.3).astype(np.float32)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    layers = m.weights()
    g, loss = m.gradients(dx, dy, batch)
    gc, lc, _ = cpu_grads(layers, x, y)
    tol = 2e-3 + (batch / 16) * 2.0 ** -23
    assert abs(loss - lc) <= tol * max(1, abs(lc))
    for (gw, gb), (cw, cb) in zip(g, gc):
        assert np.abs(gw - cw).max() <= tol * np.abs(cw).max()
        assert np.abs(gb - cb).max() <= tol * np.abs(cb).max()
    m.train_step(dx, dy, batch, 1e-2, want_loss=False)
    for (w0, b0), (w1, b1), (gw, gb) in zip(layers, m.weights(), g):
        for a0, a1, gg in ((w0, w1, gw), (b0, b1, gb)):
            want = a0 - 1e-2 * gg / (np.abs(gg) + 1e-8)
            assert np.abs(a1 - want).max() <= 1e-5 * (1 + np.abs(a0).max())


def test_narrow_network_over_many_rows(cuda):
    """A forward pass of 4-8-8-8 over 2^20 rows: 830 us with the kernel that
    staged one K step at a time, 1025 where every CTA takes the shared memory
    of eight whatever K is, and so an SM to itself."""
    torch, batch = cuda, 1 << 20
    m = vt.MLP((4, 8, 8, 8), seed=4)
    x, p = torch.randn(batch, 4, device="cuda"), torch.empty(batch, 8, device="cuda")
    us = []
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        m.forward(x, batch, p)
        b.record()
        torch.cuda.synchronize()
        us.append(a.elapsed_time(b) * 1e3)
    assert min(us) < 830
    # and the last rows are those of the same rows alone
    q = torch.empty(100, 8, device="cuda")
    m.forward(x[-100:].contiguous(), 100, q)
    assert torch.equal(p[-100:], q)
