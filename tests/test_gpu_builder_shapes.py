"""The GPU octree builder at extents around its 8 x 8 x 64 boxes, 2 x 4 x 4
words and 2048-word count blocks, float32 and uint8, against the oracle's
builder: the same bytes.  The isovalues include 0 and a negative one (the
zero padding then lies inside), the values infinities and NaN."""
import os

import numpy as np
import pytest

import visualtur_b200 as vt
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 4, 5), (1, 9, 2), (8, 8, 64), (9, 7, 65), (16, 130, 63), (64, 64, 64),
                                   (65, 33, 129)])
@pytest.mark.parametrize("u8,iso", [(False, 0.25), (False, -0.5), (True, 128.0), (True, 0.0)])
def test_gpu_builder_equals_oracle_at_odd_extents(shape, u8, iso, workdir, cuda):
    rng = np.random.default_rng(sum(shape))
    x = [np.linspace(0, 3, n) for n in shape]
    v = np.sin(x[0])[:, None, None] * np.cos(2 * x[1])[None, :, None] + 0.4 * np.sin(3 * x[2])[None, None, :]
    v = (v + 0.05 * rng.standard_normal(shape)).astype(np.float32)
    if u8:
        v = np.clip(v * 100 + 128, 0, 255).astype(np.uint8)
    else:
        flat = v.reshape(-1)
        for k, val in enumerate((np.nan, np.inf, -np.inf)):
            flat[(k * 37 + 5) % flat.size] = val
    name = "%dx%dx%d_%d_%g" % (shape + (u8, iso))
    a, b = os.path.join(workdir, "g%s.oct" % name), os.path.join(workdir, "o%s.oct" % name)
    vt.build_octree(vt.FileManager.wrap(v), iso, a)
    orc.build_octree(v, iso, b)
    assert open(a, "rb").read() == open(b, "rb").read()
