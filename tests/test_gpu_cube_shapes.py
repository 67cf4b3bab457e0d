"""renderCube where its tiles and its short tap addressing end: screens that
are no multiple of the 8 x 4 pixel tiles, bricks that are no cube, aprons of
0 and 1 (taps outside the brick), against the oracle bit for bit.  Outside
the brick's allocation both give 0."""
import numpy as np
import pytest

import visualtur_b200 as vt
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (8, 4), (37, 21), (65, 3)])
@pytest.mark.parametrize("dim,inc", [((16, 16, 16), 3), ((16, 16, 16), 0), ((12, 16, 9), 1), ((16, 10, 14), 2)])
def test_render_cube_at_odd_sizes(W, H, dim, inc, cuda):
    torch = cuda
    lo = (5, 7, 9)
    full = tuple(d + 2 * inc for d in dim)
    g = [np.arange(n, dtype=np.float32) - n / 2 for n in full]
    brick = np.sqrt(g[0][:, None, None] ** 2 + g[1][None, :, None] ** 2 + g[2][None, None, :] ** 2).astype(np.float32)
    mv = (lo[0] + dim[0] / 2, lo[1] + dim[1] / 2, lo[2] + 60.0)
    cam, ocam = vt.Camera(H, W, 50.0, 15.0, 18.0), orc.Camera(H, W, 50.0, 15.0, 18.0)
    cam.Move(mv)
    ocam.Move(mv)
    out = torch.zeros(W * H * 4, dtype=torch.float32, device="cuda")
    vt.rayCaster(4.5).renderCube(cam, torch.from_numpy(brick.ravel()).cuda(), lo, dim, (inc,) * 3, out)
    torch.cuda.synchronize()
    exp, _ = orc.render_cube(ocam, brick, lo, dim, (inc,) * 3, 4.5)
    assert np.array_equal(out.cpu().numpy().reshape(-1, 4).view(np.uint32), exp.view(np.uint32))
