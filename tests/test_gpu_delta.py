"""Ideal glass and mirrors on the B200: the reference's DIELECTRIC and GLOSSY material types
(sample_bsdf's delta branches, main.swift:3318-3352; is_delta, :3285-3287) and the bounce loop's rules
for them (no scattering event spent, no NEE, emission weight 1 after an ideal bounce, roulette ceiling
0.99; main.swift:7716-7823), against the FP64 oracle drawing the same numbers:

* a Cornell box with a mirror tall box, a glass short box and a rough GLOSSY (OpenPBR metal) wall, in
  RGB, in spectral transport with a thin film on the mirror, and with the Z++ sampler;
* the wavefront integrator's images equal the megakernel's;
* ReSTIR DI (sampling mode 0) renders the scene as the oracle does, by threads and by stages, and does
  not block the host;
* the radiance cache renders it in sampling mode 1 and refuses it in mode 0.

The GPU draws the oracle's numbers, so nearly every pixel agrees to 1e-3. Refraction in float and in
double can still part at a total-internal-reflection or Fresnel threshold, and a path that then reaches
the light through the glass carries a caustic firefly worth a few percent of the image mean. So means
and relMSE are compared over the pixels outside the 0.5 % that differ most.
"""
import time

import numpy as np
import pytest
import torch

import metal_vibe_tracer_b200 as vt
from metal_vibe_tracer_b200 import scenes, spectral_tables
from metal_vibe_tracer_b200.nrc import RadianceCache

pytestmark = pytest.mark.gpu


def relmse(a, b):
    return float(np.mean((a - b) ** 2 / (b ** 2 + 1e-2)))


def assert_agrees(gpu, ref, other, frac=0.97, mean_tol=5e-3):
    """gpu and ref drew the same numbers, other independent ones."""
    d = np.abs(gpu - ref).sum(-1)
    rel = d / (ref.sum(-1) + 1e-3)
    assert (rel < 1e-3).mean() >= frac, (rel < 1e-3).mean()
    keep = d <= np.quantile(d, 0.995)
    gm, rm = gpu[keep].mean(0), ref[keep].mean(0)
    assert np.all(np.abs(gm / rm - 1) < mean_tol), (gm, rm)
    assert relmse(gpu[keep], ref[keep]) < 0.25 * relmse(other[keep], ref[keep])


def gpu_render(ctx, mesh, mats, light, params, spp, spectral, wavefront=False):
    scene = vt.Scene(ctx, mesh, mats, light, spectral_tables.load() if spectral else None)
    (scene.render_wavefront if wavefront else scene.render)(params, spp)
    img, n = scene.readback()
    scene.close()
    assert n == spp and np.isfinite(img).all()
    return img


@pytest.mark.parametrize("spectral,sampler", [(False, 0), (True, 0), (False, 1)])
def test_delta_cornell_matches_oracle(ctx, oracle, spectral, sampler):
    faces, verts, mats, light, cam = scenes.cornell_delta(film=spectral)
    tables = spectral_tables.load() if spectral else None
    mesh = vt.Mesh(ctx, faces, verts)
    gpu = gpu_render(ctx, mesh, mats, light, vt.make_params(cam, 96, 96, 8, 1, spectral, 1, sampler=sampler), 32, spectral)
    mesh.close()
    kw = dict(max_depth=8, spectral=tables, sampler=sampler)
    ref = oracle.render(faces, verts, mats, light, cam, 96, 96, 32, **kw)
    other = oracle.render(faces, verts, mats, light, cam, 96, 96, 32, first_sample=1001, **kw)
    assert_agrees(gpu, ref, other)
    # Glass and mirrors change the picture: with those slots Lambert the box's mean radiance moves by
    # 3-11 % per channel, beyond the 1-1.5 % between independent sample sets.
    lam = oracle.render(faces, verts, [dict(m, type=0) if m["type"] in (1, 2) else m for m in mats], light, cam,
                        96, 96, 32, **kw)
    rm = ref.reshape(-1, 3).mean(0)
    assert np.abs(lam.reshape(-1, 3).mean(0) / rm - 1).max() > 0.06


@pytest.mark.parametrize("spectral", [False, True])
def test_delta_wavefront_equals_megakernel(ctx, spectral):
    faces, verts, mats, light, cam = scenes.cornell_delta(film=spectral)
    mesh = vt.Mesh(ctx, faces, verts)
    params = vt.make_params(cam, 96, 64, 8, 1, spectral, 1)
    mega = gpu_render(ctx, mesh, mats, light, params, 16, spectral)
    wave = gpu_render(ctx, mesh, mats, light, params, 16, spectral, wavefront=True)
    mesh.close()
    # Both run the same float arithmetic on the same numbers: the same paths, summed in another order.
    same = np.all(np.abs(wave - mega) <= 1e-6 * np.maximum(np.abs(mega), 1e-3), axis=-1)
    assert same.mean() >= 0.99, same.mean()
    gm, wm = mega.reshape(-1, 3).mean(0), wave.reshape(-1, 3).mean(0)
    assert np.all(np.abs(wm / gm - 1) < 2e-3), (wm, gm)


def test_delta_restir_matches_oracle(ctx, oracle):
    faces, verts, mats, light, cam = scenes.cornell_delta()
    mesh = vt.Mesh(ctx, faces, verts)
    gpu = gpu_render(ctx, mesh, mats, light, vt.make_params(cam, 64, 64, 8, 1, False, 0), 32, False)
    mesh.close()
    ref = oracle.render(faces, verts, mats, light, cam, 64, 64, 32, max_depth=8, mode=0)
    other = oracle.render(faces, verts, mats, light, cam, 64, 64, 32, max_depth=8, mode=0, first_sample=5001)
    # Reservoirs pass samples between pixels, so a parted path moves its neighbours too.
    assert_agrees(gpu, ref, other, frac=0.9)


def test_staged_delta_restir_matches_oracle(ctx, oracle):
    """As above, of a frame large enough for the stages: paths that outlive the depth end in k_wf_rest."""
    faces, verts, mats, light, cam = scenes.cornell_delta()
    mesh = vt.Mesh(ctx, faces, verts)
    gpu = gpu_render(ctx, mesh, mats, light, vt.make_params(cam, 200, 160, 3, 1, False, 0), 8, False)
    mesh.close()
    ref = oracle.render(faces, verts, mats, light, cam, 200, 160, 8, max_depth=3, mode=0)
    other = oracle.render(faces, verts, mats, light, cam, 200, 160, 8, max_depth=3, mode=0, first_sample=5001)
    assert_agrees(gpu, ref, other, frac=0.9)


@pytest.mark.parametrize("size", [(96, 72), (200, 160)])
def test_delta_restir_keeps_the_mis_energy(ctx, size):
    """By threads and by stages, at a depth that most paths through the glass outlive: the reference's 6 %."""
    faces, verts, mats, light, cam = scenes.cornell_delta()
    mesh = vt.Mesh(ctx, faces, verts)
    restir, mis = (gpu_render(ctx, mesh, mats, light, vt.make_params(cam, *size, 3, 1, False, mode), 96, False).mean() for mode in (0, 1))
    mesh.close()
    assert abs(restir / mis - 1) < 0.06, (restir, mis)


@pytest.mark.parametrize("size", [(64, 48), (200, 160)])
def test_restir_of_delta_scenes_is_stream_ordered(ctx, size):
    """vt_render queues a mode-0 frame of glass and mirrors behind half a second of other work on its stream and
    returns: nothing is read back in between."""
    faces, verts, mats, light, cam = scenes.cornell_delta()
    mesh = vt.Mesh(ctx, faces, verts)
    scene = vt.Scene(ctx, mesh, mats, light)
    params = vt.make_params(cam, *size, 8, 1, False, 0)
    scene.render(params, 2)  # allocates
    torch.cuda.synchronize()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    torch.cuda._sleep(1_000_000_000)
    end.record()
    started = time.perf_counter()
    scene.render(params, 2)
    took = time.perf_counter() - started
    torch.cuda.synchronize()
    assert took < 0.25e-3 * begin.elapsed_time(end), (took, begin.elapsed_time(end))
    scene.close()
    mesh.close()


def test_cache_takes_delta_scenes_in_mode_1_only(ctx):
    faces, verts, mats, light, cam = scenes.cornell_delta(film=True)
    mesh = vt.Mesh(ctx, faces, verts)
    scene = vt.Scene(ctx, mesh, mats, light, spectral_tables.load())
    info = mesh.info()
    cache = RadianceCache(ctx, list(info.lo), list(info.hi), train_records=4096, seed=3, spectral=1)
    for f in range(4):
        cache.render(scene, vt.make_params(cam, 32, 32, 8, 1 + 4 * f, True, 1), 4)
    img, n = scene.readback()
    assert n == 16 and np.isfinite(img).all() and img.mean() > 0.0
    with pytest.raises(vt.MaterialLibraryError, match="glass or mirror"):
        cache.render(scene, vt.make_params(cam, 32, 32, 8, 101, True, 0), 1)
    cache.close()
    scene.close()
    mesh.close()


def test_unknown_material_type_is_rejected(ctx):
    faces, verts, mats, light, cam = scenes.cornell_delta()
    mesh = vt.Mesh(ctx, faces, verts)
    bad = [dict(m) for m in mats]
    bad[2]["type"] = 7
    with pytest.raises(vt.MaterialLibraryError, match="unknown type"):
        vt.Scene(ctx, mesh, bad, light)
    mesh.close()
