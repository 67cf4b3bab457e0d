"""Rays that take the literal depth-first search instead of the 64-ary walk:
a camera inside the volume on node planes of several axes (every ray meets
coinciding planes at t = 0), and the rays left over after wavefront rounds."""
import numpy as np
import pytest

import vt_fixtures as F
import visualtur_b200 as vt
from oracle import oracle as orc
from test_gpu_parity import assert_parity
from visualtur_b200.prefetch import look_at

pytestmark = pytest.mark.gpu

W, H = 1920, 1080
GENS = {  # generator, dims, its parameters, isovalue, brick edge
    "blobs": (vt.VT_GEN_BLOBS, (512, 512, 512), (256, 5.0, 30.0, 0.5, 1.5, 0.05), 0.6, 16),
    "fractal": (vt.VT_GEN_FRACTAL_U8, (401, 290, 333), (32, 4.95, 39.2, 200.0), 128.0, 32),
}


@pytest.fixture(scope="module")
def scenes(cuda, workdir):
    torch, out = cuda, {}
    for name, (kind, dims, prm, iso, brick) in GENS.items():
        vol = torch.empty(dims, dtype=torch.uint8 if name == "fractal" else torch.float32, device="cuda")
        vt.generate_volume(kind, 1001, dims, prm, device_ptr=vol.data_ptr())
        path = "%s/literal_%s.oct" % (workdir, name)
        vt.build_octree_device(vol.data_ptr(), vt.VT_U8 if name == "fractal" else vt.VT_F32, dims, iso, path)
        out[name] = (vt.FileManager.wrap(vol.cpu().numpy()), vt.Octree(path), brick)
    return out


INSIDE, LATTICE = (128.5, 128.25, 129.5), (128, 128, 128)


def trace_ms(scene, pos, wavefront=0):
    """the trace kernels' time of one frame, every brick resident: the
    shortest of several; pos None: from outside"""
    fm, oc, brick = scene
    c = (np.array(fm.dims, float) - 1) / 2
    lc = oc.nLevels - int(np.log2(brick))
    p = vt.make_params(W=W, H=H, octreeFile=None, hdf5File=None, octreeLevel=oc.nLevels - 2, levelCubes=lc,
                       dimCube=brick, maxElementsCache=8 ** lc, maxElementsCache_CPU=8 ** lc)
    r = vt.visualTur(p, vt.default_options(preload=1, skip=0, lookahead=0, wavefront=wavefront), volume=fm, octree=oc)
    to = c if pos is None else (168, 188, 218)
    if pos is None:
        pos = c + 1.5 * max(fm.dims) * np.array([0.6, 0.3, 0.74])
    r.set_camera(look_at(W, H, 50.0, 30.0, np.array(pos, float), np.array(to, float)))
    ms = []
    for _ in range(6):
        r.updateVisibleCubes(None)
        s = r.stats()
        assert s["passes"] == 1
        ms.append(s["ms_trace_last_frame"])
    r.close()
    return min(ms[1:])


@pytest.mark.parametrize("name", sorted(GENS))
@pytest.mark.parametrize("rays", ["lattice", "waiting"])
def test_literal_rays_cost_a_search_not_more(name, rays, scenes, cuda):
    """The binary search over all rays of these frames takes 2.0 to 3.7 times
    what the walk takes on a general frame; 5 leaves room for both clocks.
    (A search that adds each ray's counters to global memory: 4.8 to 22.)"""
    if rays == "lattice":
        got, general = trace_ms(scenes[name], LATTICE), trace_ms(scenes[name], INSIDE)
    else:
        got, general = trace_ms(scenes[name], None, wavefront=1), trace_ms(scenes[name], None)
    assert got < 5 * general


@pytest.mark.parametrize("name, most", [("blobs", 2.1), ("fractal", 3.1)])
def test_camera_on_a_lattice_point_costs_no_more_than_the_binary_search(name, most, scenes, cuda):
    """Before the walk the frame from the lattice point took 1437 and 1103 us,
    2.02 and 2.95 times what the walk takes next to it."""
    assert trace_ms(scenes[name], LATTICE) < most * trace_ms(scenes[name], INSIDE)


@pytest.mark.parametrize("mode", ["resident", "slab", "cold", "cold_skip"])
@pytest.mark.parametrize("pos, fov, edge", [((64, 64, 200), 45.0, 200), ((64, 64, 200), 45.0, 201), ((63, 61, 160), 45.0, 128),
                                            ((128, 128, 192), 45.0, 160)])
def test_late_coincidences_parity(pos, fov, edge, mode, workdir, cuda):
    """Cameras on lattice points outside with a pixel grid of round numbers,
    against the oracle: the image, and (in order) every candidate once."""
    c = F.CASES["c1"]
    vol, path = F.case_volume("c1"), F.case_octree("c1", workdir)
    nb = 8 ** c["levelC"] if not mode.startswith("cold") else 40
    p = vt.make_params(W=edge, H=edge, octreeFile=None, hdf5File=None, octreeLevel=c["levelO"], levelCubes=c["levelC"],
                       dimCube=8, cubeInc=c["inc"], distance=c["dist"], fov_H=fov, fov_W=fov,
                       maxElementsCache=nb, maxElementsCache_CPU=nb)
    opt = vt.default_options(resident=mode == "resident", preload=0, record_hits=1, lookahead=0, max_passes=100000,
                             skip=2 if mode == "cold_skip" else 0)
    r = vt.visualTur(p, opt, volume=vt.FileManager.wrap(vol), octree=vt.Octree(path))
    r.camera_Move(pos)
    rgba, rgb8 = r.render_host()
    node, brick, t, nrm = r.debug_hits()
    st = r.stats()
    r.close()
    cam = orc.Camera(edge, edge, c["dist"], fov, fov)
    orc.apply_ops(cam, [("mv", pos)])
    want = orc.render(orc.Octree(path), vol, cam, c["levelO"], c["levelC"], c["inc"])
    assert_parity(dict(rgba=rgba, rgb8=rgb8, node=node, brick=brick, t=t, normal=nrm), want)
    assert st["hits"] == want["agg"]["hits"] > 0
    if mode != "cold_skip":
        assert st["samples"] == want["agg"]["samples"] and st["candidates"] == want["agg"]["candidates"]


@pytest.mark.parametrize("edge", [64, 384])     # few rays a warp, full warps (the search's own kernel)
@pytest.mark.parametrize("mode", ["resident", "slab", "cold", "cold_skip", "wave"])
@pytest.mark.parametrize("pos", [(64, 64, 64), (32, 60.5, 64), (64, 44, 128)])
def test_lattice_camera_parity(pos, mode, edge, workdir, cuda):
    """Cameras inside the volume on node planes of three and two axes, and on
    a face of it, against the oracle."""
    c = F.CASES["c1"]
    vol = F.case_volume("c1")
    path = F.case_octree("c1", workdir)
    nb = 8 ** c["levelC"] if not mode.startswith("cold") else 40
    p = vt.make_params(W=edge, H=edge, octreeFile=None, hdf5File=None, octreeLevel=c["levelO"], levelCubes=c["levelC"],
                       dimCube=8, cubeInc=c["inc"], distance=c["dist"], fov_H=c["fov"], fov_W=c["fov"],
                       maxElementsCache=nb, maxElementsCache_CPU=nb)
    opt = vt.default_options(resident=mode == "resident", preload=0, record_hits=1, lookahead=0, max_passes=100000,
                             skip=2 if mode == "cold_skip" else 0, wavefront=2 if mode == "wave" else 0)
    r = vt.visualTur(p, opt, volume=vt.FileManager.wrap(vol), octree=vt.Octree(path))
    r.camera_Move(pos)
    rgba, rgb8 = r.render_host()
    node, brick, t, nrm = r.debug_hits()
    st = r.stats()
    r.close()
    cam = orc.Camera(edge, edge, c["dist"], c["fov"], c["fov"])
    orc.apply_ops(cam, [("mv", pos)])
    want = orc.render(orc.Octree(path), vol, cam, c["levelO"], c["levelC"], c["inc"])
    assert_parity(dict(rgba=rgba, rgb8=rgb8, node=node, brick=brick, t=t, normal=nrm), want)
    assert st["rays"] == edge * edge and st["hits"] == want["agg"]["hits"] > 0
    if mode != "cold_skip":
        assert st["samples"] == want["agg"]["samples"] and st["candidates"] == want["agg"]["candidates"]


def test_cameras_on_and_off_the_lattice_through_one_graph(scenes, cuda):
    """Pass 0 is a captured graph whose kernel changes with the camera."""
    torch = cuda
    fm, oc, brick = scenes["blobs"]
    lc = oc.nLevels - 4
    p = vt.make_params(W=640, H=480, octreeFile=None, hdf5File=None, octreeLevel=oc.nLevels - 2, levelCubes=lc,
                       dimCube=brick, maxElementsCache=8 ** lc, maxElementsCache_CPU=8 ** lc)
    cams = [look_at(640, 480, 50.0, 30.0, np.array(pos, float), np.array((168.0, 188.0, 218.0)))
            for pos in (INSIDE, LATTICE, LATTICE, INSIDE, (256, 256, 256), INSIDE)]
    images = []
    for graph in (0, 1):
        r = vt.visualTur(p, vt.default_options(preload=1, skip=0, lookahead=0, use_graph=graph), volume=fm, octree=oc)
        s, out = torch.cuda.Stream(), []
        for c in cams:
            r.set_camera(c)
            rgba = torch.empty(640 * 480, 4, device="cuda")
            torch.cuda.synchronize()
            r.updateVisibleCubes(rgba, stream=s.cuda_stream)
            s.synchronize()
            out.append(rgba)
        images.append(out)
        r.close()
    for a, b in zip(*images):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert not torch.equal(images[0][0], images[0][1])
