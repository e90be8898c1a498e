"""The wavefront integrator (vt_render_wavefront) against the megakernel (vt_render) on the B200.

Both draw the same numbers from the same samplers; the wavefront's traversals are the persistent
quantised-node kernels of traverse.cu (the megakernel walks the 128-byte nodes), whose closest hit can
differ only between triangles hit at exactly the same distance, and its stages prepare an OPENPBR vertex
once for all its uses where the megakernel prepares it at each (other contractions of the same
formulas). So the images agree pixel for pixel to float rounding, 1e-6, except on a handful of pixels (with
layered OPENPBR slots 1e-4 on 98 %, since narrow lobes amplify a rounding), and their means to well within
the estimator's noise:
* Cornell box, spectral and RGB, sampling modes 1-3;
* the OpenPBR Cornell box (spectral), an imported scene under its light tree and an open scene with
  the procedural sky (shadow rays with the endpoint slack, MIS-weighted escapes);
* a pass of 8M paths, more samples than one pass's 16M paths hold, and a strided frame.
"""
import numpy as np
import pytest
import torch

import metal_vibe_tracer_b200 as vt
from metal_vibe_tracer_b200 import scenes, spectral_tables

pytestmark = pytest.mark.gpu


def both(ctx, mesh, mats, light, params, spp, spectral, env=None):
    out = []
    for wavefront in (False, True):
        scene = vt.Scene(ctx, mesh, mats, light, spectral_tables.load() if spectral else None)
        if env:
            scene.set_environment(**env)
        (scene.render_wavefront if wavefront else scene.render)(params, spp)
        img, n = scene.readback()
        scene.close()
        assert n == spp and np.isfinite(img).all()
        out.append(img)
    return out


def assert_same(mega, wave, frac=0.995):
    same = np.all(np.abs(wave - mega) <= 1e-6 * np.maximum(np.abs(mega), 1e-3), axis=-1)
    assert same.mean() >= frac, same.mean()
    gm, wm = mega.reshape(-1, 3).mean(0), wave.reshape(-1, 3).mean(0)
    assert np.all(np.abs(wm / gm - 1) < 2e-3), (wm, gm)


@pytest.fixture(scope="module")
def cornell(ctx):
    faces, verts, mats, light, cam = scenes.cornell_box()
    mesh = vt.Mesh(ctx, faces, verts)
    yield mats, light, cam, mesh
    mesh.close()


@pytest.mark.parametrize("spectral,mode", [(True, 1), (False, 1), (True, 2), (True, 3)])
def test_cornell_equals_megakernel(ctx, cornell, spectral, mode):
    mats, light, cam, mesh = cornell
    mega, wave = both(ctx, mesh, mats, light, vt.make_params(cam, 96, 64, 8, 1, spectral, mode), 16, spectral)
    assert_same(mega, wave)


def test_openpbr_and_imported_scenes_equal_megakernel(ctx):
    faces, verts, mats, light, cam = scenes.cornell_openpbr()
    mesh = vt.Mesh(ctx, faces, verts)
    assert_same(*both(ctx, mesh, mats, light, vt.make_params(cam, 64, 64, 8, 1, True, 1), 16, True))
    mesh.close()
    faces, verts, mats, cam = scenes.cornell_emitters()
    mesh = vt.Mesh(ctx, faces, verts)
    assert_same(*both(ctx, mesh, mats, None, vt.make_params(cam, 64, 48, 8, 1, True, 1), 16, True))
    mesh.close()
    faces, verts, mats, cam = scenes.sky_scene(emitter=True)
    mesh = vt.Mesh(ctx, faces, verts)
    env = {"intensity": 1.0, "sun_dir": (0.4, 0.6, -0.5), "sun_intensity": 30.0, "sky_mode": 0}
    assert_same(*both(ctx, mesh, mats, None, vt.make_params(cam, 64, 64, 8, 1, True, 1), 16, True, env))
    mesh.close()


@pytest.mark.parametrize("spectral", [False, True])
def test_layered_openpbr_equals_megakernel(ctx, spectral):
    """Every layer the shared preparation carries (film, coat, fuzz, anisotropy, part metal, pure metal,
    diffuse roughness) on its own slot: the stage kernels' one preparation per vertex against the
    megakernel's one per use. (1e-4 on 98 % of pixels: the two compile a vertex's f and pdf with other
    contractions, which narrow lobes amplify.)"""
    faces, verts, mats, light, cam = scenes.cornell_openpbr()
    layers = [dict(thin_film_weight=1.0, thin_film_thickness=0.4, thin_film_ior=1.4), dict(coat=0.8), dict(fuzz=0.7),
              dict(anisotropy=0.6, metalness=1.0), dict(metalness=0.4), dict(diffuse_roughness=0.8, coat=0.3, fuzz=0.2),
              dict(metalness=1.0, thin_film_weight=0.5, thin_film_thickness=0.25, thin_film_ior=1.6)]
    mats = [dict(m, **layers[i % len(layers)]) if m["type"] == 4 else m for i, m in enumerate(mats)]
    mesh = vt.Mesh(ctx, faces, verts)
    mega, wave = both(ctx, mesh, mats, light, vt.make_params(cam, 96, 64, 6, 1, spectral, 1), 8, spectral)
    mesh.close()
    same = np.all(np.abs(wave - mega) <= 1e-4 * np.maximum(np.abs(mega), 1e-3), axis=-1)
    assert same.mean() >= 0.98, same.mean()
    assert np.all(np.abs(wave.mean((0, 1)) / mega.mean((0, 1)) - 1) < 2e-3)


def test_long_paths_equal_megakernel(ctx):
    """Paths far longer than the stages' 64 slots of counters: a closed box of albedo 0.98 walls."""
    faces, verts, mats, cam = scenes.cornell_emitters()
    pts = verts["p"][np.stack([faces["a"], faces["b"], faces["c"]], 1)]
    front = [((-1, -1, -1), (1, -1, -1), (1, 1, -1)), ((-1, -1, -1), (1, 1, -1), (-1, 1, -1))]
    faces, verts = scenes._mesh_from_triangles(list(pts) + front, list(faces["tag"]) + [0, 0])
    mats = [dict(m, albedo=(0.98,) * 3) if m["type"] == 0 else m for m in mats]
    cam = dict(cam, pos=(0.3, 0.2, -0.9), target=(0.0, -0.1, 0.3))
    mesh = vt.Mesh(ctx, faces, verts)
    mega, wave = both(ctx, mesh, mats, None, vt.make_params(cam, 40, 24, 150, 1, False, 1), 4, False)
    mesh.close()
    assert_same(mega, wave)


@pytest.mark.parametrize("spectral", [False, True])
def test_open_scene_of_every_class_equals_megakernel(ctx, spectral):
    """An open scene without an environment (escaped paths are dropped, their last light sample still
    counts) whose slots cover every class the stages regroup by: Lambert, dielectric, metal, film,
    emitter. (Tolerance as for the layered slots.)"""
    faces, verts, mats, cam = scenes.sky_scene(emitter=True, subdivisions=3)
    pbr = dict(type=4, albedo=(0.7, 0.4, 0.3), emission=(0.0, 0.0, 0.0))
    first = len(mats)
    mats = mats + [dict(pbr, roughness=0.3), dict(pbr, roughness=0.4, metalness=1.0),
                   dict(pbr, roughness=0.35, thin_film_weight=1.0, thin_film_thickness=0.4, thin_film_ior=1.4)]
    sphere = np.flatnonzero(faces["tag"] == 1)
    faces["tag"][sphere[sphere % 4 > 0]] = first - 1 + (sphere % 4)[sphere % 4 > 0]
    mesh = vt.Mesh(ctx, faces, verts)
    mega, wave = both(ctx, mesh, mats, None, vt.make_params(cam, 96, 64, 6, 1, spectral, 1), 8, spectral)
    mesh.close()
    same = np.all(np.abs(wave - mega) <= 1e-4 * np.maximum(np.abs(mega), 1e-3), axis=-1)
    assert same.mean() >= 0.98, same.mean()
    assert np.all(np.abs(wave.mean((0, 1)) / mega.mean((0, 1)) - 1) < 2e-3)


@pytest.mark.parametrize("mode,sampler", [(1, 0), (2, 0), (1, 1)])
def test_openpbr_under_a_light_tree_equals_megakernel(ctx, mode, sampler):
    """Spectral OpenPBR slots (a film among them) under a light tree, where the light samples have a launch of
    their own, beside Lambert and mirror slots. (Tolerance as for the layered slots.)"""
    faces, verts, mats, cam = scenes.cornell_emitters()
    pbr = dict(type=4, emission=(0.0, 0.0, 0.0), roughness=0.35, ior=1.5)
    mats[2] = dict(pbr, albedo=(0.7, 0.6, 0.5))
    mats[3] = dict(pbr, albedo=(0.6, 0.1, 0.1), thin_film_weight=1.0, thin_film_thickness=0.4, thin_film_ior=1.4)
    mats[4] = dict(pbr, albedo=(0.9, 0.7, 0.3), metalness=1.0)
    mats[5] = scenes.cornell_delta()[2][5]
    mesh = vt.Mesh(ctx, faces, verts)
    params = vt.make_params(cam, 96, 64, 6, 1, True, mode, sampler=sampler)
    mega, wave = both(ctx, mesh, mats, None, params, 8, True)
    mesh.close()
    same = np.all(np.abs(wave - mega) <= 1e-4 * np.maximum(np.abs(mega), 1e-3), axis=-1)
    assert same.mean() >= 0.98, same.mean()
    assert np.all(np.abs(wave.mean((0, 1)) / mega.mean((0, 1)) - 1) < 2e-3)


def test_passes_and_stride(ctx, cornell):
    mats, light, cam, mesh = cornell
    # 1024 x 1024 x 8 spp = 8M paths in one pass (test_largest_passes takes two).
    mega, wave = both(ctx, mesh, mats, light, vt.make_params(cam, 1024, 1024, 4, 1, False, 1), 8, False)
    assert_same(mega, wave)
    mega, wave = both(ctx, mesh, mats, light, vt.make_params(cam, 96, 64, 8, 1, True, 1, pixel_stride=3), 8, True)
    assert_same(mega, wave)


def test_largest_passes(ctx, cornell):
    """More samples than one pass of 16M paths holds: 4 + 1 samples of 4M pixels."""
    mats, light, cam, mesh = cornell
    mega, wave = both(ctx, mesh, mats, light, vt.make_params(cam, 2000, 2000, 2, 1, False, 1), 5, False)
    assert_same(mega, wave)


def test_state_holds_only_what_the_render_uses(ctx, cornell):
    """The path state of a first wavefront render: 229 bytes a path, and 20 more for the queues by kind of vertex
    where slots are OPENPBR (no light samples of their own in RGB, no spread without a cache)."""
    spp, paths = 4, 4 * 1024 * 1024
    faces, verts, mats, light, cam = scenes.cornell_openpbr()
    mesh = vt.Mesh(ctx, faces, verts)
    for m, materials, per_path in ((cornell[3], cornell[0], 229), (mesh, mats, 249)):
        scene = vt.Scene(ctx, m, materials, cornell[1], None)
        params = vt.make_params(cam, 1024, 1024, 2, 1, False, 1)
        scene.render(params, spp)  # the accumulation and the jitter
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        scene.render_wavefront(params, spp)
        taken = before - torch.cuda.mem_get_info()[0]
        assert per_path * paths - (8 << 20) <= taken <= per_path * paths + (8 << 20), taken / paths
        scene.close()
    mesh.close()


def test_rejects_restir(ctx, cornell):
    mats, light, cam, mesh = cornell
    scene = vt.Scene(ctx, mesh, mats, light, None)
    with pytest.raises(vt.MaterialLibraryError, match="sampling modes 1-3"):
        scene.render_wavefront(vt.make_params(cam, 16, 16, 8, 1, False, 0), 1)
    scene.close()
