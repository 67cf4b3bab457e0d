"""Rays that wait in a queue more than once for the same brick.

With candidates set aside behind absent bricks (skip > 0) a ray resumes with
them first.  Where one of those bricks is absent again -- the request list,
the demand batch or the device cache had no room for it -- the ray waits
once more and must still go on from the candidate its walk had stopped at:
every candidate is marched once, and none is passed over unmarched."""
import numpy as np
import pytest

import vt_fixtures as F
import visualtur_b200 as vt
from visualtur_b200.prefetch import look_at
from test_gpu_faults import frame, make
from test_gpu_parity import assert_parity, oracle_render

pytestmark = pytest.mark.gpu

LIMITS = {"requests": dict(max_requests=3), "batch": dict(demand_batch=2), "cache": dict(dev=24, host=16)}


@pytest.mark.parametrize("limit", sorted(LIMITS))
@pytest.mark.parametrize("skip", [1, 2, 4])
@pytest.mark.parametrize("case", ["c1", "c1plane"])
def test_every_candidate_is_marched_once(case, skip, limit, workdir, cuda):
    """The octree's volume replaced by zeros: nothing crosses the isovalue,
    so a ray takes all its candidates whatever is set aside, and candidates
    and samples are those of the in-order search exactly."""
    zeros = np.zeros_like(F.case_volume(case))
    r = make(case, workdir, fm=vt.FileManager.wrap(zeros), skip=skip, lookahead=0, max_passes=100000, **LIMITS[limit])
    st = frame(r)["stats"]
    agg = oracle_render(case, workdir, vol=zeros)["agg"]
    assert agg["hits"] == 0 and st["hits"] == 0 and st["passes"] > 2
    assert st["candidates"] == agg["candidates"]
    assert st["samples"] == agg["samples"]
    r.close()


@pytest.mark.parametrize("limit", sorted(LIMITS))
@pytest.mark.parametrize("skip", [1, 2, 4])
@pytest.mark.parametrize("case", ["c1", "c1plane", "c1in"])
def test_image_with_bricks_absent_again(case, skip, limit, workdir, cuda):
    """c1plane: a camera on node planes, whose rays meet coinciding planes
    late and then pass over the candidates taken before."""
    r = make(case, workdir, skip=skip, lookahead=0, max_passes=100000, **LIMITS[limit])
    got = frame(r)
    want = oracle_render(case, workdir)
    assert_parity(got, want)
    assert got["stats"]["hits"] == want["agg"]["hits"]
    r.close()


@pytest.fixture(scope="module")
def blobs(cuda, workdir):
    torch, n = cuda, 512
    vol = torch.empty((n, n, n), dtype=torch.float32, device="cuda")
    vt.generate_volume(vt.VT_GEN_BLOBS, 1001, (n, n, n), (256, n / 102.4, n / 17.0667, 0.5, 1.5, 0.05),
                       device_ptr=vol.data_ptr())
    path = workdir + "/resume_blobs.oct"
    vt.build_octree_device(vol.data_ptr(), vt.VT_F32, vol.shape, 0.6, path)
    return vt.FileManager.wrap(vol.cpu().numpy()), vt.Octree(path)


def blobs_frame(torch, blobs, bricks=4096, **opt):
    fm, oc = blobs
    p = vt.make_params(W=960, H=540, octreeFile=None, hdf5File=None, octreeLevel=oc.nLevels - 2,
                       levelCubes=oc.nLevels - 4, dimCube=16, maxElementsCache=bricks, maxElementsCache_CPU=32768)
    r = vt.visualTur(p, vt.default_options(lookahead=0, max_passes=100000, **opt), volume=fm, octree=oc)
    c = (fm.dims[0] - 1) / 2
    r.set_camera(look_at(960, 540, 50.0, 30.0, c + 768 * np.array([0.6, 0.3, 0.74]), np.full(3, c)))
    rgba, _ = r.render_host()
    st = r.stats()
    r.close()
    return rgba, st


@pytest.mark.parametrize("opt", [dict(skip=2, max_requests=500), dict(skip=4, demand_batch=256),
                                 dict(skip=4, bricks=3000)])
def test_large_frame_with_bricks_absent_again(opt, blobs, cuda):
    """512^3 blobs, rays enough that some meet coinciding planes: the frame
    paged in with set-aside candidates is the in-order one."""
    want, ref = blobs_frame(cuda, blobs, bricks=32768, preload=1, skip=0)
    got, st = blobs_frame(cuda, blobs, preload=0, **opt)
    assert ref["passes"] == 1 and st["passes"] > 2
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert st["hits"] == ref["hits"] > 100000
