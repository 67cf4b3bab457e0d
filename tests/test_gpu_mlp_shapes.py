"""The tensor-core kernels of the prefetch network at shapes where their
tiling can go wrong: one of everything, exact tiles, one past a tile, rows
that are no whole 16-byte chunks, K split over CTAs (wide outputs, few rows)
and not.  Gradients against the CPU implementation of test_gpu_mlp.py, which
rounds the same operands to BF16: agreement up to FP32 summation order, the
same bound of 2e-3 of a layer's largest gradient."""
import numpy as np
import pytest

import visualtur_b200 as vt
from test_gpu_mlp import cpu_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,batch", [((1, 1, 1, 1), 1), ((3, 8, 16, 64), 128), ((12, 129, 65, 513), 129),
                                        ((30, 7, 9, 200), 300), ((70, 64, 128, 1000), 65),
                                        ((12, 512, 512, 4096), 1), ((12, 96, 511, 4096), 257)])
def test_gradients_and_update_at_ragged_shapes(dims, batch, cuda):
    torch = cuda
    m = vt.MLP(dims, seed=4)
    rng = np.random.default_rng(8)
    x = rng.standard_normal((batch, dims[0])).astype(np.float32)
    y = (rng.random((batch, dims[3])) < 0.3).astype(np.float32)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    layers = m.weights()
    g, loss = m.gradients(dx, dy, batch)
    gc, lc, p = cpu_grads(layers, x, y)
    assert abs(loss - lc) <= 1e-4 * max(1, abs(lc))
    for (gw, gb), (cw, cb) in zip(g, gc):
        assert np.abs(gw - cw).max() <= 2e-3 * (np.abs(cw).max() + 1e-12)
        assert np.abs(gb - cb).max() <= 2e-3 * (np.abs(cb).max() + 1e-12)
    # the update: the first Adam step from the gradients the kernels report
    # (m / c1 = g and v / c2 = g^2 up to rounding), every weight and bias
    m.train_step(dx, dy, batch, 1e-2, want_loss=False)
    for (w0, b0), (w1, b1), (gw, gb) in zip(layers, m.weights(), g):
        for a0, a1, gg in ((w0, w1, gw), (b0, b1, gb)):
            want = a0 - 1e-2 * gg / (np.abs(gg) + 1e-8)
            assert np.abs(a1 - want).max() <= 1e-5 * (1 + np.abs(a0).max())
    # the updated BF16 weights are the ones a forward pass reads
    out, ref = torch.empty(batch * dims[3], device="cuda"), torch.empty(batch * dims[3], device="cuda")
    m2 = vt.MLP(dims, seed=5)
    m2.set_weights(m.weights())
    m.forward(dx, batch, out)
    m2.forward(dx, batch, ref)
    assert torch.equal(out, ref)


def test_noalloc_forward_in_row_blocks(cuda):
    """Layers narrower than a 16-byte chunk take more scratch than the
    accepted bound counts: the call goes by row blocks, with the same result."""
    torch = cuda
    m = vt.MLP((5, 1, 1, 3), seed=2)
    batch = 262144 // 2
    x = torch.randn(batch, 5, device="cuda")
    a, b = torch.empty(batch * 3, device="cuda"), torch.empty(batch * 3, device="cuda")
    m.forward(x, batch, a)
    m.forward_noalloc(x, batch, b)
    assert torch.equal(a, b)
