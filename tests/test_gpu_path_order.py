"""Path numbering and queue layout: results do not depend on how a frame is cut into chunks,
on which views of a batch have lights, or on lights that appear between batches.

The reference is the same frame in one chunk (itself equal to the oracle in test_gpu_parity.py);
every comparison is bit for bit. Small frames without lights are rendered path by path in one
kernel: cut into chunks they take the wavefront, so the two are compared here as well.
"""
import numpy as np
import pytest

from kuafu_gb300 import _native as N
from kuafu_gb300 import api, scenes

pytestmark = pytest.mark.gpu

AOVS = (N.KF_AOV_RADIANCE_F32, N.KF_AOV_ALBEDO_F32, N.KF_AOV_NORMAL_F32, N.KF_AOV_DEPTH_F32, N.KF_AOV_SEGMENTATION,
        N.KF_AOV_PATH_RADIANCE, N.KF_AOV_PRIMARY_HITS)


def _aov(r, cam, kind):
    a = r.downloadAov(cam, kind)
    if kind == N.KF_AOV_SEGMENTATION:
        a = a[..., [0, 1, 3]]  # not the material: its number counts every material of the process
    return a


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def _frame(lit, w, h, spp, chunk):
    cfg = scenes.icosphere_config(spp=spp, depth=5, count=6) if lit else scenes.cornell_config(spp=spp, depth=4)
    cfg.setDebugOutputs(True)
    if chunk:
        cfg.setMaxPathsInFlight(chunk)
    with api.Kuafu(cfg) as r:
        cam = scenes.icospheres(r, w, h, count=6, level=2) if lit else scenes.cornell(r, w, h)
        r.run()
        return [_aov(r, cam, k) for k in AOVS] + [r.downloadLatestFrame(cam)]


# odd sizes; chunks that end inside a pixel, inside a band of rows and at band ends (8 rows)
@pytest.mark.parametrize("lit", [False, True])
@pytest.mark.parametrize("w,h,spp,chunk", [(37, 19, 7, 1000), (33, 24, 9, 33 * 8 * 9), (41, 9, 3, 1), (64, 17, 12, 777)])
def test_chunks_do_not_change_the_frame(lit, w, h, spp, chunk):
    if chunk == 1:
        w, h, spp, chunk = 5, 3, 2, 4
    for kind, a, b in zip(AOVS + ("frame",), _frame(lit, w, h, spp, 0), _frame(lit, w, h, spp, chunk)):
        assert _same(a, b), kind


@pytest.mark.parametrize("w,h", [(512, 320), (641, 256), (163841, 1)])
def test_whole_paths_and_wavefront_agree(w, h):
    """Both sides of the limit between whole paths and the wavefront, with spheres (metal, glass and
    mirror paths), Russian roulette, an environment map and textures: one launch against the
    thread-per-ray wavefront."""
    spp = 1  # 163840 paths, 164096, and 163841 of a one-row frame (nearly all of them miss)
    rng = np.random.default_rng(3)
    env = rng.random((6, 8, 8, 4), dtype=np.float32)
    tex = api.createTexture(rng.integers(0, 256, (16, 16, 4), dtype=np.uint8))
    out = []
    for traversal in (1, 0):
        cfg = scenes.icosphere_config(spp=spp, depth=6, count=64)
        cfg.setTraversal(traversal)
        cfg.setDebugOutputs(True)
        with api.Kuafu(cfg) as r:
            cam = scenes.icospheres(r, w, h, count=40, level=2, seed=1)
            s = r.getScene()
            s.removeLights()
            s.setEnvironmentMap(env)
            ground = api.createYZPlane(False, api.NiceMaterial(diffuseTex=tex, roughness=0.8))
            s.submitGeometry(ground)
            s.submitGeometryInstance(api.instance(ground, scenes.translate(0, 0, -22) @ scenes.rot_axis("y", -90) @
                                                  scenes.scale(30.0, 30.0, 30.0)))
            r.run()
            st = r.stats()
            out.append([_aov(r, cam, k) for k in AOVS] + [r.downloadLatestFrame(cam),
                                                           np.array([st.rays_primary, st.rays_extension])])
    for k, (a, b) in enumerate(zip(*out)):
        assert _same(a, b), k
    assert h == 1 or out[0][-1][1] > 1000


# lights of every kind, more slots than lanes of a path, and none that emit; a small frame (whole
# paths), one just past that limit and larger ones whose tail is finished path by path, in one and
# several chunks
@pytest.mark.parametrize("w,h,spp,chunk,points", [(64, 64, 4, 0, 4), (31, 17, 3, 0, 11), (16385, 1, 1, 0, 1),
                                                  (200, 150, 2, 0, 4), (200, 150, 2, 17000, 11), (8, 8, 1, 0, 0)])
def test_whole_paths_with_lights(w, h, spp, chunk, points):
    out = []
    for traversal in (1, 0):
        cfg = scenes.icosphere_config(spp=spp, depth=7, count=64)
        cfg.setTraversal(traversal)
        cfg.setDebugOutputs(True)
        if chunk:
            cfg.setMaxPathsInFlight(chunk)
        with api.Kuafu(cfg) as r:
            cam = scenes.icospheres(r, w, h, count=48, level=2, seed=2)
            s = r.getScene()
            s.removeLights()
            for k in range(points):
                s.addPointLight(api.PointLight(position=(-10.0 + 3 * k, 5.0 - k, 4.0 + k), color=(1.0, 0.5 + 0.04 * k, 0.3),
                                               radius=0.4 * (k % 2), strength=200.0))
            s.setDirectionalLight(api.DirectionalLight(direction=(-1.0, 0.2, -1.0), strength=1.0, softness=0.05))
            s.addActiveLight(api.ActiveLight(viewMat=scenes.look_at_view((0.0, 3.0, 25.0), (0, 0, 0), (0, 1, 0)),
                                             fov=1.0, strength=500.0, softness=0.1))
            r.run()
            st = r.stats()
            out.append([_aov(r, cam, k) for k in AOVS] + [np.array([st.rays_primary, st.rays_extension, st.rays_shadow])])
            if not chunk:
                r.runBatch([(s, cam, spp)])
                out[-1].append(_aov(r, cam, N.KF_AOV_PATH_RADIANCE))
    for k, (a, b) in enumerate(zip(*out)):
        assert _same(a, b), k


def test_resolve_sample_counts():
    """Sample counts around the resolve's groups of 8: the mean of the downloaded paths, in order."""
    for spp in (1, 3, 4, 8, 9, 17):
        cfg = scenes.cornell_config(spp=spp, depth=2)
        with api.Kuafu(cfg) as r:
            cam = scenes.cornell(r, 45, 13)
            r.run()
            paths = r.downloadAov(cam, N.KF_AOV_PATH_RADIANCE, spp)[..., :3]
            total = np.zeros_like(paths[0])
            for k in range(spp):
                total = total + paths[k]
            assert _same(r.downloadAov(cam, N.KF_AOV_RADIANCE_F32)[..., :3], total / np.float32(spp)), spp


def _mixed(r):
    """A room without lights to sample, spheres with seven, and a second camera of the room."""
    room, spheres = r.getScene(), r.createScene()
    c0 = scenes.cornell(r, 40, 31, scene=room)
    c1 = scenes.icospheres(r, 53, 27, count=5, level=2, scene=spheres)
    c2 = room.createCamera(24, 24)
    c2.setPosition((-3.0, 0.1, 0.2))
    c2.setFront((1.0, 0.0, 0.0))
    c2.setUp((0.0, 0.0, 1.0))
    scenes.pinhole(c2, 24, 24, 50.0)
    return room, [(room, c0, 5), (spheres, c1, 3), (room, c2, 9)]


@pytest.mark.parametrize("chunk", [0, 1234])
def test_batch_of_lit_and_unlit_views(chunk):
    def render(pick):
        cfg = scenes.icosphere_config(spp=1, depth=4, count=64)
        if chunk:
            cfg.setMaxPathsInFlight(chunk)
        with api.Kuafu(cfg) as r:
            _, items = _mixed(r)
            part = [items[k] for k in pick]
            r.runBatch(part)
            return [_aov(r, c, k) for _, c, _ in part for k in AOVS[:5]]

    alone = [x for k in range(3) for x in render([k])]  # one view each: a new renderer's first frame word
    for a, b in zip(render([0, 1, 2]), alone):
        assert _same(a, b)


def test_lights_added_between_batches():
    """The captured launch sequence is renewed when a batch gains lights (its buffers move)."""
    light = lambda: api.PointLight(position=(0.0, 0.0, 0.5), color=(1.0, 0.9, 0.8), radius=0.1, strength=2.0)

    def render(when):
        with api.Kuafu(scenes.icosphere_config(spp=1, depth=4, count=64)) as r:
            room, items = _mixed(r)
            items = [items[0], items[2]]
            for batch in range(2):
                if batch == when:
                    for _ in range(3):
                        room.addPointLight(light())
                r.runBatch(items)
            return [r.downloadAov(c, N.KF_AOV_RADIANCE_F32) for _, c, _ in items]

    for a, b, dark in zip(render(1), render(0), render(2)):
        assert _same(a, b)
        assert not _same(a, dark)


def test_changed_lights_reach_the_next_frame():
    """Lights are uploaded when they change: a point light recoloured and a directional light added
    between frames give the frame of a renderer that had them from the start."""
    import ctypes as C

    def render(when):
        with api.Kuafu(scenes.icosphere_config(spp=2, depth=3, count=64)) as r:
            s = r.getScene()
            cam = scenes.cornell(r, 31, 22, scene=s)
            light = api.PointLight(position=(0.0, 0.0, 0.5), color=(1.0, 0.2, 0.1), radius=0.1, strength=2.0)
            s.addPointLight(light)
            for frame in range(2):
                if frame == when:
                    c = N.kf_point_light((C.c_float * 3)(0.1, 0.0, 0.5), (C.c_float * 3)(0.2, 1.0, 0.4), 0.1, 3.0)
                    N.check(N.load().kf_light_update_point(s._lights[id(light)][1], C.byref(c)))
                    s.setDirectionalLight(api.DirectionalLight(direction=(1.0, 0.1, -0.4), strength=1.5))
                r.resetFrame()
                r.run()
            return r.downloadAov(cam, N.KF_AOV_RADIANCE_F32)

    assert _same(render(1), render(0))
    assert not _same(render(1), render(2))


def test_replayed_frames_follow_buffers_that_moved():
    """Frames between which other launches grow the wavefront's buffers (more light slots, more
    paths, deeper paths) and a camera is resized to and fro: captured launches against direct ones."""
    light = lambda k: api.PointLight(position=(-10.0 + 3 * k, 5.0 - k, 4.0 + k), radius=0.2, strength=200.0)

    def render(use_graph):
        cfg = scenes.icosphere_config(spp=2, depth=4, count=64)
        cfg.setUseGraph(use_graph)
        out = []
        with api.Kuafu(cfg) as r:
            s, many = r.getScene(), r.createScene()
            cam = scenes.icospheres(r, 150, 130, count=8, level=2, seed=3, scene=s)
            wide = scenes.icospheres(r, 211, 190, count=8, level=2, seed=4, scene=many)
            s.removeLights()
            s.addPointLight(light(0))
            for k in range(9):
                many.addPointLight(light(k))

            def frame():
                r.resetFrame()
                r.run()
                out.append([_aov(r, cam, k) for k in AOVS[:6]])

            frame()
            r.runBatch([(many, wide, 3)])
            out.append([_aov(r, wide, AOVS[0])])
            frame()
            cam.setSize(170, 140)
            r.runBatch([(s, cam, 1), (many, wide, 2)])
            cam.setSize(150, 130)
            frame()
            r.config.setPathDepth(7)
            r.applyConfig()
            r.runBatch([(many, wide, 3)])
            r.config.setPathDepth(4)
            r.applyConfig()
            frame()
        return out

    for n, (a, b) in enumerate(zip(render(True), render(False))):
        for k, (x, y) in enumerate(zip(a, b)):
            assert _same(x, y), (n, k)


@pytest.mark.parametrize("kind,words", [(N.KF_AOV_PATH_RADIANCE, 1), (N.KF_AOV_PRIMARY_HITS, 2)])
def test_path_data_comes_in_one_copy(kind, words):
    """A download of per-path data costs about what its bytes cost: at 64 x 64 pixels and 1024
    samples at most three times a plain copy of as many bytes to ordinary memory (a copy per sample
    takes 37 times as long). Best of several, both sides."""
    import time

    import torch

    w, h, spp = 64, 64, 1024
    cfg = scenes.cornell_config(spp=spp, depth=2)
    cfg.setDebugOutputs(True)
    out = np.zeros(w * h * spp * 4 * words, np.float32)
    plain, host = torch.zeros(out.size, device="cuda"), torch.from_numpy(out)
    with api.Kuafu(cfg) as r:
        cam = scenes.cornell(r, w, h)
        r.run()

        def best(f):
            times = []
            for _ in range(9):
                torch.cuda.synchronize()
                t = time.perf_counter()
                f()
                torch.cuda.synchronize()
                times.append(time.perf_counter() - t)
            return min(times)

        copy = best(lambda: host.copy_(plain))
        got = best(lambda: N.check(N.load().kf_renderer_download_aov(r._h, cam._h, kind, out.ctypes.data, out.nbytes)))
    assert got <= 3.0 * copy, (got, copy)
