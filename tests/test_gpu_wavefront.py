"""The persistent wavefront past the first bounce, against the oracle and on both streams.

Small frames run whole paths in one kernel, and the last paths of larger lit ones as well, so these
frames are made to stay on the wavefront: the profiling schedule runs its kernels alone, and the
two-stream frames keep more rays in every bounce than the kernel of the last paths takes."""
import numpy as np
import pytest

from kuafu_gb300 import _native as N
from kuafu_gb300 import api, scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TAIL = 12288  # rays of a bounce that are finished path by path (kTailMax of kf_wavefront.cu)


def _ground(s, rng):
    tex = api.createTexture(rng.integers(0, 256, (16, 16, 4), dtype=np.uint8))
    plane = api.createYZPlane(False, api.NiceMaterial(diffuseTex=tex, roughness=0.8))
    s.submitGeometry(plane)
    s.submitGeometryInstance(api.instance(plane, scenes.translate(0, 0, -22) @ scenes.rot_axis("y", -90) @
                                          scenes.scale(30.0, 30.0, 30.0)))


def _environment(rng, n=16):
    y, x = np.mgrid[0:n, 0:n] / (n - 1)
    faces = np.ones((6, n, n, 4), np.float32)
    for f in range(6):
        for c in range(3):
            a, b, ph = rng.uniform(0.5, 3.0, 3)
            faces[f, :, :, c] = 0.3 + 0.25 * np.sin(a * x * 6.28 + ph) * np.cos(b * y * 6.28) + 0.1 * f
    return faces


def _same_paths(r, scene, cam, spp, depth, rr, env, clear=(0.1, 0.1, 0.1, 1.0)):
    """Primary hits equal to the oracle's and path radiance within 1e-4 (all but 1 path in 1000)."""
    w, h = cam._size()
    ref = O.render(scene.export(), cam.ubo(), w, h, O.push_constants(spp, depth, clear=clear, rr=rr, rr_min=1, env=env),
                   seed=r.config._c.seed, frame=0, camera_index=1, use_bvh=True)
    hits = r.downloadAov(cam, N.KF_AOV_PRIMARY_HITS, spp)
    assert np.array_equal(hits["instance"], ref["hits"]["instance"])
    got = r.downloadAov(cam, N.KF_AOV_PATH_RADIANCE, spp)[..., :3].astype(np.float64)
    want = ref["paths"].astype(np.float64)
    err = (np.abs(got - want) / np.maximum(np.abs(want), 1e-6)).max(axis=-1)
    assert (err <= 1e-4).mean() >= 0.999
    return ref


@pytest.mark.parametrize("lights", ["all", "none", "black"])
def test_wavefront_kernels_against_the_oracle(lights):
    """Spheres (diffuse, metal, glass) over a textured ground under an environment map, with Russian
    roulette: lights of every kind, none, and light slots that never emit."""
    spp, depth = 3, 6
    cfg = scenes.icosphere_config(spp=spp, depth=depth, count=64)
    cfg.setDebugOutputs(True)
    cfg.setRussianRouletteMinBounces(1)
    cfg.setTraversal(1)
    cfg.setProfile(True)
    with api.Kuafu(cfg) as r:
        s = r.getScene()
        cam = scenes.icospheres(r, 97, 61, count=40, level=2, seed=6)
        rng = np.random.default_rng(8)
        _ground(s, rng)
        s.setEnvironmentMap(_environment(rng))
        if lights != "all":
            s.removeLights()
        if lights == "black":
            for k in range(3):
                s.addPointLight(api.PointLight(position=(k, 2.0, 5.0), color=(0.0, 0.0, 0.0), radius=0.2, strength=9.0))
        r.run()
        _same_paths(r, s, cam, spp, depth, True, True)
        st = r.stats()
        assert st.rays_extension > 3000 and (st.rays_shadow > 3000 if lights == "all" else st.rays_shadow == 0)


def test_light_slots_that_never_emit_on_whole_paths():
    """The same on the kernel that runs whole paths, several lanes to a path: no shadow ray, and the
    frame of a scene without lights."""
    out = []
    for points in (0, 3):
        cfg = scenes.icosphere_config(spp=3, depth=6, count=64)
        cfg.setDebugOutputs(True)
        cfg.setRussianRouletteMinBounces(1)
        with api.Kuafu(cfg) as r:
            s = r.getScene()
            cam = scenes.icospheres(r, 45, 33, count=40, level=2, seed=6)
            s.removeLights()
            for k in range(points):
                s.addPointLight(api.PointLight(position=(k, 2.0, 5.0), color=(0.0, 0.0, 0.0), radius=0.2, strength=9.0))
            r.run()
            _same_paths(r, s, cam, 3, 6, True, False)
            assert r.stats().rays_shadow == 0
            out.append([r.downloadAov(cam, k) for k in (N.KF_AOV_PATH_RADIANCE, N.KF_AOV_ALBEDO_F32,
                                                        N.KF_AOV_NORMAL_F32, N.KF_AOV_DEPTH_F32)])
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def _room(depth, profile, chunk):
    """A lit room of 512 x 512 pixels at 2 samples: frames, path radiance and extension rays."""
    cfg = scenes.cornell_config(spp=2, depth=depth)
    cfg.setProfile(profile)
    cfg.setMaxPathsInFlight(chunk)
    with api.Kuafu(cfg) as r:
        cam = scenes.cornell(r, 512, 512)
        s = r.getScene()
        for k in range(3):
            s.addPointLight(api.PointLight(position=(0.3 * k - 0.3, 0.2, 0.5), color=(1.0, 0.9 - 0.2 * k, 0.5),
                                           radius=0.1 * k, strength=1.0))
        r.run()
        r.run()
        return (r.downloadAov(cam, N.KF_AOV_RADIANCE_F32), r.downloadLatestFrame(cam),
                r.downloadAov(cam, N.KF_AOV_PATH_RADIANCE), r.stats().rays_extension)


@pytest.mark.parametrize("chunk", [1 << 24, 180000])
def test_streams_overlap_at_every_bounce(chunk):
    """Shadow rays and their sums run beside the next bounce's rays: the same bytes as kernel after
    kernel on one stream, with more rays in each bounce of each chunk than are finished path by path."""
    depth = 4
    two, one = _room(depth, False, chunk), _room(depth, True, chunk)
    assert all(np.array_equal(a, b) for a, b in zip(two[:3], one[:3])) and two[3] == one[3]
    last = one[3] - _room(depth - 1, True, chunk)[3]  # rays of the last bounce, two frames
    chunks = -(-512 * 512 * 2 // chunk)
    assert last / 2 > 2 * TAIL * chunks
