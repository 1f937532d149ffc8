"""Parity of the CUDA passes with the CPU oracle, through the C ABI.

Visibility outputs (LodRecords, StrandRefs, center / conservative / beta
G-buffers, deep opacity map) must be bit-exact.  Shaded colour is compared on
identical inputs (the GPU's own G-buffer and map fed to the oracle) within
SHADE_RTOL / SHADE_ATOL; the filter's coverage alpha is exact and its colour
within FILTER_RTOL.
"""
import math
import os
from pathlib import Path

import numpy as np
import pytest

import oracle
from bevy_hair_gb300 import abi, configs, groom, host
from bevy_hair_gb300.pipeline import HairRenderer, Light, pack_lights

pytestmark = pytest.mark.gpu

# Colour tolerances: the GPU evaluates exp/log/asin/cos/pow with CUDA's
# functions and FMA contraction, the oracle with libm and none.
SHADE_RTOL, SHADE_ATOL = 2e-3, 1e-5
FILTER_RTOL, FILTER_ATOL = 1e-4, 1e-6
EMPTY = np.uint64(0xFFFFFFFFFFFFFFFF)


@pytest.fixture(scope="module")
def renderer():
    r = HairRenderer(0)
    yield r
    r.close()


def _assert_equal(name, got, want):
    got, want = np.asarray(got), np.asarray(want)
    assert got.shape == want.shape, (name, got.shape, want.shape)
    bad = np.flatnonzero(got != want)
    if bad.size:
        i = bad[:5]
        pytest.fail(f"{name}: {bad.size} of {got.size} differ; first {i.tolist()}: got {got[i].tolist()} "
                    f"want {want[i].tolist()}")


def _scenes():
    return {
        "config1": lambda: configs.config1(scale=0.05),
        "config2": lambda: configs.config2(scale=0.02),
        "config3": lambda: configs.config3(scale=0.01),
    }


def _visibility(r: HairRenderer, sc: configs.Scene, cam, dom, scene_depth=None):
    w, h = int(cam["screen"][0]), int(cam["screen"][1])
    r.ensure_targets(w, h, *sc.dom_size)
    g = r.upload(sc.mesh)
    depth_ptr = None
    if scene_depth is not None:
        r.write(abi.BUF_DEPTH, scene_depth)
        depth_ptr, _ = r.buffer(abi.BUF_DEPTH)
    r.clear()
    r.lod(g, cam, abi.SLOT_CAMERA)
    r.scan(g, cam, abi.SLOT_CAMERA)
    r.raster(g, cam, abi.SLOT_CAMERA, depth_ptr)
    out = {"lod": g.read(abi.SLOT_CAMERA, abi.GBUF_LOD), "refs": g.read(abi.SLOT_CAMERA, abi.GBUF_REFS),
           "indirect": g.read(abi.SLOT_CAMERA, abi.GBUF_INDIRECT)}
    out["center"] = r.read(abi.BUF_CENTER)
    out["cons"] = r.read(abi.BUF_CONSERVATIVE)
    out["beta"] = r.read(abi.BUF_BETA)
    if dom is not None:
        r.clear_dom()
        r.lod(g, dom, abi.SLOT_DOM)
        r.scan(g, dom, abi.SLOT_DOM)
        r.raster(g, dom, abi.SLOT_DOM)
        out["dom_depth"] = r.read(abi.BUF_DOM)
        r.raster(g, host.dom_layers_params(dom), abi.SLOT_DOM)
        out["dom"] = r.read(abi.BUF_DOM)
        out["dom_lod"] = g.read(abi.SLOT_DOM, abi.GBUF_LOD)
        out["dom_refs"] = g.read(abi.SLOT_DOM, abi.GBUF_REFS)
        out["dom_indirect"] = g.read(abi.SLOT_DOM, abi.GBUF_INDIRECT)
    assert r.synchronize() == 0
    g.close()
    return out


def _oracle_visibility(sc, cam, dom, scene_depth=None):
    w, h = int(cam["screen"][0]), int(cam["screen"][1])
    cap = max(sc.mesh.strand_count(), 1)
    center, cons, beta = oracle.clear_targets(w, h)
    lod = oracle.lod(cam, sc.mesh)
    refs, total = oracle.scan(cam, lod, cap)
    counts = oracle.raster(cam, sc.mesh, refs, total, center, cons, beta, None, scene_depth)
    out = dict(lod=lod, refs=refs, total=total, center=center, cons=cons, beta=beta, counts=counts)
    if dom is not None:
        d = oracle.clear_dom(*sc.dom_size)
        dl = oracle.lod(dom, sc.mesh)
        drefs, dtotal = oracle.scan(dom, dl, cap)
        oracle.raster(dom, sc.mesh, drefs, dtotal, center, cons, beta, d)
        out["dom_depth"] = d.copy()
        oracle.raster(host.dom_layers_params(dom), sc.mesh, drefs, dtotal, center, cons, beta, d)
        out.update(dom=d, dom_lod=dl, dom_refs=drefs, dom_total=dtotal)
    return out


def _check_visibility(got, want, with_dom=True):
    n = len(want["lod"])
    _assert_equal("lod", got["lod"][:n].view(np.uint32), want["lod"].view(np.uint32))
    total = int(got["indirect"][0])
    assert total == want["total"]
    assert got["indirect"][1] == 1 and got["indirect"][2] == 1
    _assert_equal("refs", got["refs"][:total].view(np.uint32), want["refs"][:total].view(np.uint32))
    _assert_equal("center", got["center"], want["center"])
    _assert_equal("conservative", got["cons"], want["cons"])
    _assert_equal("beta", got["beta"], want["beta"])
    if with_dom:
        _assert_equal("dom_lod", got["dom_lod"][: len(want["dom_lod"])].view(np.uint32),
                      want["dom_lod"].view(np.uint32))
        assert int(got["dom_indirect"][0]) == want["dom_total"]
        _assert_equal("dom depth pass", got["dom_depth"], want["dom_depth"])
        _assert_equal("dom layers pass", got["dom"], want["dom"])


@pytest.mark.parametrize("name", list(_scenes()))
def test_visibility_and_dom_bit_exact(renderer, name):
    sc = _scenes()[name]()
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    assert (want["center"] != EMPTY).sum() > 100, "scene draws too little to be a test"
    _check_visibility(got, want)


@pytest.mark.parametrize("name", ["config2", "config3_far"])
def test_strand_cache_gives_the_same_visibility(renderer, name):
    """hg_generate then the rasters: refs at 65 control points read the strand
    cache, the others generate in the raster; the buffers must not change."""
    if name == "config2":
        sc = configs.config2(scale=0.02)
    else:  # LOD levels: only part of the camera refs are at 65 control points
        sc = configs.config3(scale=0.01)
        sc.view = configs._camera(sc.view.width, sc.view.height, 1200.0)
        sc.groom.lam = 1.0
    cam, dom = sc.params()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.generate(g, cam)
    renderer.clear()
    renderer.lod(g, cam, abi.SLOT_CAMERA)
    renderer.scan(g, cam, abi.SLOT_CAMERA)
    renderer.raster(g, cam, abi.SLOT_CAMERA)
    renderer.clear_dom()
    renderer.lod(g, dom, abi.SLOT_DOM)
    renderer.scan(g, dom, abi.SLOT_DOM)
    renderer.raster(g, dom, abi.SLOT_DOM)
    renderer.raster(g, host.dom_layers_params(dom), abi.SLOT_DOM)
    assert renderer.synchronize() == 0
    want = _oracle_visibility(sc, cam, dom)
    _assert_equal("center", renderer.read(abi.BUF_CENTER), want["center"])
    _assert_equal("conservative", renderer.read(abi.BUF_CONSERVATIVE), want["cons"])
    _assert_equal("beta", renderer.read(abi.BUF_BETA), want["beta"])
    _assert_equal("dom", renderer.read(abi.BUF_DOM), want["dom"])
    cps = want["lod"]["control_points"][want["lod"]["n_lod"] > 0]
    if name != "config2":
        assert (cps == 65).any() and (cps != 65).any()
    g.close()


@pytest.mark.parametrize("n", [1, 2, 33, 160_001])
def test_strand_cache_equals_strands_generated_in_the_raster(renderer, n):
    """The cache's generation takes strands in pairs and their last points 32 at
    a time (160,001: more than 16 pairs a warp, and an odd one); the rasters
    without a cache generate a strand per warp."""
    sc = configs.config1(scale=0.01)
    sc.mesh = configs._mesh(n, 8, "curly", 77)
    cam, dom = sc.params()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    got = []
    for cached in (False, True):
        if cached:
            renderer.generate(g, cam)
        renderer.clear()
        renderer.clear_dom()
        for p, slot in ((cam, abi.SLOT_CAMERA), (dom, abi.SLOT_DOM)):
            renderer.lod(g, p, slot)
            renderer.scan(g, p, slot)
            renderer.raster(g, p, slot)
        renderer.raster(g, host.dom_layers_params(dom), abi.SLOT_DOM)
        assert renderer.synchronize() == 0
        got.append([renderer.read(b) for b in (abi.BUF_CENTER, abi.BUF_CONSERVATIVE, abi.BUF_BETA, abi.BUF_DOM)])
    g.close()
    for name, want, have in zip(("center", "conservative", "beta", "dom"), *got):
        _assert_equal(name, have, want)
    assert (got[0][1] != EMPTY).any()


@pytest.mark.parametrize("n", [1216, 1217, 1219])
def test_strand_cache_at_the_line_of_single_strands(renderer, n):
    """Up to sm_count x 8 strands (1,216 on 152 SMs) a warp takes one strand,
    above a pair, the last one cut short at an odd count."""
    test_strand_cache_equals_strands_generated_in_the_raster(renderer, n)


@pytest.mark.parametrize("n", [1, 3, 32, 9728, 9729, 9731, 20_000])
def test_lod_of_many_bundles_matches_the_oracle(renderer, n):
    """Four bundles share a warp from sm_count x 64 bundles up (9,728 on 152
    SMs), a bundle has its own below; last warps in part."""
    sc = configs.config2(scale=0.001)
    mesh = sc.mesh
    sc.mesh = groom.HairMesh(np.resize(mesh.bundles, n), mesh.layers, mesh.style, mesh.bounds_min, mesh.bounds_max)
    cam, dom = sc.params()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    for p, slot in ((cam, abi.SLOT_CAMERA), (dom, abi.SLOT_DOM)):
        renderer.lod(g, p, slot)
        assert renderer.synchronize() == 0
        want = oracle.lod(p, sc.mesh)
        _assert_equal("lod", g.read(slot, abi.GBUF_LOD)[:n].view(np.uint32), want[:n].view(np.uint32))
    g.close()


@pytest.mark.parametrize("n", [1, 3648, 3649, 7296, 7297])
def test_one_camera_stage_equals_two(renderer, n):
    """A frame draws the camera's refs in one stage while its warps take at most
    two each (2 x 3,648 on 152 SMs); the pass by itself always takes two."""
    sc = configs.config1(scale=n / 10_000) if n > 16 else configs.config1(scale=0.0016)
    if n == 1:
        sc.mesh = configs._mesh(1, 32, "straight", 3)
    assert sc.mesh.strand_count() == n
    cam, dom = sc.params()
    want = _visibility(renderer, sc, cam, dom)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, sc.light_array())
    assert renderer.synchronize() == 0
    for name, which in (("center", abi.BUF_CENTER), ("cons", abi.BUF_CONSERVATIVE), ("beta", abi.BUF_BETA),
                        ("dom", abi.BUF_DOM)):
        _assert_equal(name, renderer.read(which), want[name])
    # the frame's refs drawn once more by the pass: no draw order of an earlier scan is taken for theirs
    renderer.lod(g, dom, abi.SLOT_CAMERA)
    renderer.scan(g, cam, abi.SLOT_CAMERA)
    renderer.render_groom(g, cam, dom, sc.light_array())
    renderer.clear()
    renderer.raster(g, cam, abi.SLOT_CAMERA)
    assert renderer.synchronize() == 0
    _assert_equal("center", renderer.read(abi.BUF_CENTER), want["center"])
    g.close()


def test_dense_groom_with_tile_depth_rejection(renderer):
    """A dense groom at low resolution (deep overdraw) with a small deep
    opacity map: the later stages of the camera and DOM depth passes skip most
    segments behind the tile depths, and no buffer may change."""
    sc = configs.config2(scale=0.25)
    sc.view = configs._camera(384, 216, 900.0)
    sc.dom_size = (192, 192)
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    _check_visibility(got, want)
    covered = int((want["center"] != EMPTY).sum())
    assert covered > 5000 and want["counts"]["samples"] > 50 * covered


def test_two_grooms_into_one_g_buffer(renderer):
    """A second groom rastered over the first without a clear: the tile depths
    of its later stages start from the first groom's words."""
    a = configs.config2(scale=0.05)
    b = configs.config3(scale=0.02)
    a.view = configs._camera(480, 270, 900.0)
    cam_a, _ = a.params()
    b.view = a.view
    cam_b, _ = b.params()
    renderer.ensure_targets(480, 270, *a.dom_size)
    ga, gb = renderer.upload(a.mesh), renderer.upload(b.mesh)
    renderer.clear()
    for g, cam in ((ga, cam_a), (gb, cam_b)):
        renderer.lod(g, cam, abi.SLOT_CAMERA)
        renderer.scan(g, cam, abi.SLOT_CAMERA)
        renderer.raster(g, cam, abi.SLOT_CAMERA)
    assert renderer.synchronize() == 0
    center, cons, beta = oracle.clear_targets(480, 270)
    for sc, cam in ((a, cam_a), (b, cam_b)):
        lod = oracle.lod(cam, sc.mesh)
        refs, total = oracle.scan(cam, lod, max(sc.mesh.strand_count(), 1))
        oracle.raster(cam, sc.mesh, refs, total, center, cons, beta, None)
    _assert_equal("center", renderer.read(abi.BUF_CENTER), center)
    _assert_equal("conservative", renderer.read(abi.BUF_CONSERVATIVE), cons)
    _assert_equal("beta", renderer.read(abi.BUF_BETA), beta)
    assert (center != EMPTY).sum() > 1000
    ga.close()
    gb.close()


@pytest.mark.parametrize("diameter", [0.01, 0.3, 0.7, 1.0, 1.41421356, 2.5])
def test_center_disk_diameters(renderer, diameter):
    """The centre-sample acceptance disk (raster.wgsl:201,212) at several
    diameters, including the 0.05 floor and one whose radius squares inexactly."""
    sc = configs.config1(scale=0.03)
    sc.groom.center_diameter = diameter
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, None)
    want = _oracle_visibility(sc, cam, None)
    _check_visibility(got, want, with_dom=False)


def test_clear_sentinels(renderer):
    renderer.ensure_targets(37, 19, 7, 5)
    renderer.clear()
    renderer.clear_dom()
    assert (renderer.read(abi.BUF_CENTER) == EMPTY).all()
    assert (renderer.read(abi.BUF_CONSERVATIVE) == EMPTY).all()
    assert (renderer.read(abi.BUF_BETA) == 0xFFFFFFFF).all()
    dom = renderer.read(abi.BUF_DOM)
    assert (dom[:35] == 0xFFFFFFFF).all() and (dom[35:] == 0).all() and dom.size == 35 * 17


def test_forward_z_scene_depth_and_ao_off(renderer):
    """Forward-Z projection, a scene depth buffer that hides part of the groom,
    ambient occlusion off (raster.wgsl:93-107)."""
    sc = configs.config1(scale=0.05)
    sc.groom.ambient_occlusion = False
    v = sc.view
    sc.view = host.View(v.world_from_view, host.perspective_rh(math.pi / 4, v.width / v.height, 0.1, 5000.0),
                        v.width, v.height)
    cam, dom = sc.params()
    assert cam["pass_mode"][2] == 0
    w, h = v.width, v.height
    rng = np.random.default_rng(5)
    scene_depth = np.where(rng.random(w * h) < 0.5, np.float32(1.0), np.float32(0.9990)).astype(np.float32)
    got = _visibility(renderer, sc, cam, None, scene_depth)
    want = _oracle_visibility(sc, cam, None, scene_depth)
    _check_visibility(got, want, with_dom=False)
    assert (want["center"] != EMPTY).sum() > 50
    assert ((want["center"][want["center"] != EMPTY] & np.uint64(0x3F)) == 63).all()


def test_camera_inside_the_groom_clips_at_the_near_plane(renderer):
    """Segments behind the camera or straddling it (project_world's in_front,
    the near-plane rejection in write_pixel)."""
    sc = configs.config2(scale=0.01)
    c = (sc.mesh.bounds_min + sc.mesh.bounds_max) * 0.5
    wfv = host.looking_at(c + np.array([0, 0, 20.0], np.float32), c + np.array([0, 0, -100.0], np.float32))
    sc.view = host.View(wfv, sc.view.clip_from_view, sc.view.width, sc.view.height)
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    _check_visibility(got, want)


def test_groom_outside_the_view_is_culled(renderer):
    sc = configs.config1(scale=0.02)
    wfv = host.looking_to(np.array([0, 0, 1000.0], np.float32), np.array([0, 0, 1.0], np.float32), (0, 1, 0))
    sc.view = host.View(wfv, sc.view.clip_from_view, sc.view.width, sc.view.height)
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, None)
    want = _oracle_visibility(sc, cam, None)
    _check_visibility(got, want, with_dom=False)
    assert int(got["indirect"][0]) == 0 and (got["center"] == EMPTY).all()


def test_lod_levels_and_strand_thinning(renderer):
    """A far camera: bundles take several control-point levels and n_lod < strand_count."""
    sc = configs.config3(scale=0.01)
    sc.view = configs._camera(sc.view.width, sc.view.height, 6000.0)
    sc.groom.lam = 0.6
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    _check_visibility(got, want)
    lod = want["lod"]
    assert len(set(lod["control_points"][lod["n_lod"] > 0].tolist())) >= 2
    assert (lod["n_lod"] < lod["strand_count"]).any()


def test_empty_groom(renderer):
    from bevy_hair_gb300.groom import HairMesh

    sc = configs.config1(scale=0.02)
    sc.mesh = HairMesh(np.zeros(0, abi.GPU_BUNDLE), np.zeros(0, abi.GPU_LAYER), np.zeros((0, 4), np.float32),
                       np.zeros(3, np.float32), np.zeros(3, np.float32))
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    assert int(got["indirect"][0]) == 0 and int(got["dom_indirect"][0]) == 0
    assert (got["center"] == EMPTY).all() and (got["cons"] == EMPTY).all()
    n = sc.dom_size[0] * sc.dom_size[1]
    assert (got["dom"][:n] == 0xFFFFFFFF).all() and (got["dom"][n:] == 0).all()


@pytest.mark.parametrize("name", list(_scenes()))
def test_shade_filter_composite_within_tolerance(renderer, name):
    """Shade, filter and composite on identical inputs: the GPU's G-buffer and
    map go to the oracle's passes and both outputs are compared."""
    sc = _scenes()[name]()
    cam, dom = sc.params()
    lights = sc.light_array()
    w, h = sc.view.width, sc.view.height
    renderer.ensure_targets(w, h, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights)
    assert renderer.synchronize() == 0
    center, cons, beta = renderer.read(abi.BUF_CENTER), renderer.read(abi.BUF_CONSERVATIVE), renderer.read(abi.BUF_BETA)
    dmap = renderer.read(abi.BUF_DOM)
    shaded, sdepth = renderer.read(abi.BUF_SHADED), renderer.read(abi.BUF_SHADED_DEPTH)
    filt, fdepth = renderer.read(abi.BUF_FILTERED), renderer.read(abi.BUF_FILTERED_DEPTH)
    color, depth = renderer.read(abi.BUF_COLOR), renderer.read(abi.BUF_DEPTH)
    g.close()

    o_shaded, o_sdepth = oracle.shade(cam, center, beta, dmap, lights)
    hit = center != EMPTY
    assert hit.sum() > 50
    np.testing.assert_array_equal(sdepth, o_sdepth)
    np.testing.assert_allclose(shaded, o_shaded, rtol=SHADE_RTOL, atol=SHADE_ATOL)
    assert np.isfinite(shaded).all()

    o_filt, o_fdepth = oracle.filter_(cam, center, cons, shaded, sdepth)
    np.testing.assert_array_equal(fdepth, o_fdepth)
    np.testing.assert_array_equal(filt.reshape(-1, 4)[:, 3], o_filt.reshape(-1, 4)[:, 3])
    np.testing.assert_allclose(filt, o_filt, rtol=FILTER_RTOL, atol=FILTER_ATOL)

    o_color = np.zeros(w * h * 4, np.float32)
    o_depth = np.full(w * h, 0.0 if cam["pass_mode"][2] == 1 else 1.0, np.float32)
    oracle.composite(cam, filt, fdepth, o_color, o_depth)
    np.testing.assert_array_equal(depth, o_depth)
    np.testing.assert_allclose(color, o_color, rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("size", [(31, 9), (33, 17), (640, 384), (641, 384), (1024, 512), (1031, 517)])
def test_filter_at_the_edges_of_its_thread_split(renderer, size):
    """Four, two or one threads per pixel pair (up to 245,760 and 524,288 pixels),
    ragged tiles, every kind of texel and tangents that lie along the rows or
    toward the viewer: coverage and view distance exact, colour within the
    filter's tolerance."""
    w, h = size
    sc = configs.config1(scale=0.02)
    cam, _ = host.groom_params(configs._camera(w, h, 1000.0), sc.groom, sc.mesh.bounds_min, sc.mesh.bounds_max,
                               sc.mesh.bundle_count, sc.directionals, sc.dom_size)
    rng = np.random.default_rng(w * 4096 + h)
    n = w * h
    x, y = np.meshgrid(np.arange(w), np.arange(h))
    base = 0.4 + 0.1 * np.sin(0.05 * x) * np.cos(0.07 * y)
    depth = ((base.ravel() + rng.normal(0.0, 1e-3, n)) * 16777214.0).astype(np.uint64)
    oct_x, oct_y = rng.integers(0, 256, n, dtype=np.uint64), rng.integers(0, 256, n, dtype=np.uint64)
    axis = rng.random(n)
    oct_x[axis < 0.1], oct_y[axis < 0.1] = 255, 128     # nearly along +X
    oct_x[axis > 0.9], oct_y[axis > 0.9] = 128, 128     # nearly along +Z
    words = (depth << np.uint64(40)) | (oct_x << np.uint64(32)) | (oct_y << np.uint64(24)) | np.uint64(0xFFF)
    kind = rng.random(n)
    center = np.where(kind < 0.6, words, EMPTY)
    near = words - (rng.integers(0, 20_000, n, dtype=np.uint64) << np.uint64(40))
    cons = np.where(kind < 0.8, np.where(kind < 0.3, near, words), EMPTY)
    shaded = rng.random((n, 4)).astype(np.float32)
    shaded[:, 3] = (rng.random(n) < 0.9).astype(np.float32)
    renderer.ensure_targets(w, h, 0, 0)
    renderer.write(abi.BUF_CENTER, center)
    renderer.write(abi.BUF_CONSERVATIVE, cons)
    renderer.write(abi.BUF_SHADED, shaded)
    renderer.filter(cam)
    assert renderer.synchronize() == 0
    filt = renderer.read(abi.BUF_FILTERED).reshape(-1, 4)
    fdepth = renderer.read(abi.BUF_FILTERED_DEPTH)
    want, want_depth = oracle.filter_(cam, center, cons, shaded, np.zeros(n, dtype=np.float32))
    want = np.asarray(want).reshape(-1, 4)
    _assert_equal("filter alpha", filt[:, 3], want[:, 3])
    _assert_equal("filter depth", fdepth, np.asarray(want_depth))
    np.testing.assert_allclose(filt[:, :3], want[:, :3], rtol=FILTER_RTOL, atol=FILTER_ATOL)


@pytest.mark.parametrize("s_par, s_perp", [(1.0, 0.2), (1.0, 0.02), (100.0, 0.02), (0.05, 0.02), (0.05, 1.0), (0.3, 0.3)])
@pytest.mark.parametrize("size", [(97, 61), (800, 500), (1021, 531)])
def test_filter_widths_at_the_ends_of_their_ranges(renderer, size, s_par, s_perp):
    """Narrow and wide filters (the widths are clamped to 0.05 along the strand
    and 0.02 across it) in every direction, four, two and one threads a pair.

    A weight's relative error is at most 1.3e-5 here and 2.3e-5 in the oracle,
    whose float distance across the strand it comes from, both at width 0.02;
    a colour, the weighted mean of values in [0, 1], moves by no more than their
    sum, and by 3e-6 for the 121 terms of its sums."""
    w, h = size
    sc = configs.config1(scale=0.02)
    cam, _ = host.groom_params(configs._camera(w, h, 1000.0), sc.groom, sc.mesh.bounds_min, sc.mesh.bounds_max,
                               sc.mesh.bundle_count, sc.directionals, sc.dom_size)
    cam = cam.copy()
    cam["filter_params"][:2] = s_par, s_perp
    rng = np.random.default_rng(w + h)
    n = w * h
    depth = ((0.4 + rng.normal(0.0, 2e-4, n)) * 16777214.0).astype(np.uint64)
    oct_x, oct_y = rng.integers(0, 256, n, dtype=np.uint64), rng.integers(0, 256, n, dtype=np.uint64)
    words = (depth << np.uint64(40)) | (oct_x << np.uint64(32)) | (oct_y << np.uint64(24)) | np.uint64(0xFFF)
    center = np.where(rng.random(n) < 0.9, words, EMPTY)
    shaded = rng.random((n, 4)).astype(np.float32)
    shaded[:, 3] = (rng.random(n) < 0.5).astype(np.float32)
    renderer.ensure_targets(w, h, 0, 0)
    renderer.write(abi.BUF_CENTER, center)
    renderer.write(abi.BUF_CONSERVATIVE, words)
    renderer.write(abi.BUF_SHADED, shaded)
    renderer.filter(cam)
    assert renderer.synchronize() == 0
    filt = renderer.read(abi.BUF_FILTERED).reshape(-1, 4)
    want, want_depth = oracle.filter_(cam, center, words, shaded, np.zeros(n, dtype=np.float32))
    want = np.asarray(want).reshape(-1, 4)
    _assert_equal("filter depth", renderer.read(abi.BUF_FILTERED_DEPTH), np.asarray(want_depth))
    # without a centre hit a pixel counts only from a total weight of 1e-5 up,
    # which the two sides may see on either side of it
    sure = (center != EMPTY) | ((filt[:, 3] > 0) == (want[:, 3] > 0))
    assert sure.mean() > 0.999
    _assert_equal("filter alpha", filt[sure, 3], want[sure, 3])
    np.testing.assert_allclose(filt[sure, :3], want[sure, :3], rtol=0.0, atol=1.3e-5 + 2.3e-5 + 3e-6)


@pytest.mark.parametrize("scale", [0.02, 1.0])
def test_full_frame_against_the_oracle_frame(renderer, scale):
    """hg_groom_frame against the oracle's whole hair_pass sequence; at scale 1
    the benchmark frame itself, light probe included."""
    sc = configs.config2(scale=scale)
    cam, dom = sc.params()
    lights = sc.light_array()
    env = None
    if scale == 1.0:
        from bevy_hair_gb300 import envmap

        env = envmap.procedural()
    renderer.set_environment(env)
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights)
    assert renderer.synchronize() == 0
    renderer.set_environment(None)
    want = oracle.frame(sc.mesh, cam, dom, lights, env=env)
    _assert_equal("center", renderer.read(abi.BUF_CENTER), want["center"])
    _assert_equal("conservative", renderer.read(abi.BUF_CONSERVATIVE), want["cons"])
    _assert_equal("beta", renderer.read(abi.BUF_BETA), want["beta"])
    _assert_equal("dom", renderer.read(abi.BUF_DOM), want["dom"])
    np.testing.assert_allclose(renderer.read(abi.BUF_SHADED), want["shaded"], rtol=SHADE_RTOL, atol=SHADE_ATOL)
    color = renderer.read(abi.BUF_COLOR)
    # colour differences from shading propagate through the filter and blend
    np.testing.assert_allclose(color, want["color"], rtol=5 * SHADE_RTOL, atol=10 * SHADE_ATOL)
    g.close()


@pytest.mark.parametrize("composite,clear_color", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("use_filter", [True, False])
@pytest.mark.parametrize("deep_opacity", [True, False])
def test_frame_equals_its_passes(renderer, deep_opacity, use_filter, composite, clear_color):
    """hg_groom_frame's merged launches (setup of both views, both clears, filter
    with colour clear and composite) against the single passes, every target
    bit for bit, on a screen and map whose sizes leave vector tails."""
    sc = configs.config1(scale=0.02)
    sc.groom.deep_opacity, sc.groom.filter = deep_opacity, use_filter
    w, h = 197, 131
    sc.view = configs._camera(w, h, 1000.0)
    sc.dom_size = (37, 37)
    cam, dom = sc.params()
    lights = sc.light_array()
    r = renderer
    r.ensure_targets(w, h, *sc.dom_size)
    g = r.upload(sc.mesh)
    rng = np.random.default_rng(5)
    old_color = rng.random(w * h * 4).astype(np.float32)
    old_depth = (rng.random(w * h) * 2e-4).astype(np.float32)
    names = ["CENTER", "CONSERVATIVE", "BETA", "SHADED", "SHADED_DEPTH", "COLOR", "DEPTH"]
    names += ["DOM"] if deep_opacity else []
    names += ["FILTERED", "FILTERED_DEPTH"] if use_filter else []

    def outputs(draw):
        for n in names:  # nothing may be left over from the other way
            ptr_bytes = r.buffer(getattr(abi, "BUF_" + n))[1]
            r.write(getattr(abi, "BUF_" + n), np.full(ptr_bytes, 0x5A, dtype=np.uint8))
        r.write(abi.BUF_COLOR, old_color)
        r.write(abi.BUF_DEPTH, old_depth)
        draw()
        assert r.synchronize() == 0
        return {n: r.read(getattr(abi, "BUF_" + n)).copy() for n in names}

    def passes():
        r.clear()
        r.lod(g, cam, abi.SLOT_CAMERA)
        r.scan(g, cam, abi.SLOT_CAMERA)
        if deep_opacity:
            r.generate(g, cam)
            r.clear_dom()
            r.lod(g, dom, abi.SLOT_DOM)
            r.scan(g, dom, abi.SLOT_DOM)
            r.raster(g, dom, abi.SLOT_DOM)
            r.raster(g, host.dom_layers_params(dom), abi.SLOT_DOM)
        r.raster(g, cam, abi.SLOT_CAMERA)
        r.shade(cam, lights)
        if use_filter:
            r.filter(cam)
        if composite and clear_color:
            r.clear_color(0.0 if cam["pass_mode"][2] == 1 else 1.0)
        if composite:
            r.composite(cam, use_filter)

    want = outputs(passes)
    got = outputs(lambda: r.render_groom(g, cam, dom if deep_opacity else None, lights, composite=composite,
                                         clear_color=clear_color))
    for n in names:
        _assert_equal(n, got[n].view(np.uint32), want[n].view(np.uint32))
    g.close()


@pytest.mark.parametrize("deep_opacity", [True, False])
def test_frame_behind_scene_depth_equals_its_passes(renderer, deep_opacity):
    """hg_groom_frame with a scene depth that hides some of the hair, with and
    without a map, against the single passes."""
    import torch

    sc = configs.config1(scale=0.02)
    sc.groom.deep_opacity = deep_opacity
    w, h = 197, 131
    sc.view = configs._camera(w, h, 1000.0)
    cam, dom = sc.params()
    lights = sc.light_array()
    r = renderer
    r.ensure_targets(w, h, *sc.dom_size)
    g = r.upload(sc.mesh)
    names = ["CENTER", "CONSERVATIVE", "BETA", "SHADED", "FILTERED", "COLOR", "DEPTH"]
    scene = torch.from_numpy(np.random.default_rng(8).random(w * h).astype(np.float32) * np.float32(2e-4)).cuda()
    torch.cuda.synchronize()

    def outputs():
        assert r.synchronize() == 0
        return {n: r.read(getattr(abi, "BUF_" + n)).copy() for n in names}

    r.clear()
    r.clear_color(0.0)
    for p, slot in ((cam, abi.SLOT_CAMERA), (dom, abi.SLOT_DOM))[:1 + deep_opacity]:
        r.lod(g, p, slot)
        r.scan(g, p, slot)
    if deep_opacity:
        r.generate(g, cam)
        r.clear_dom()
        r.raster(g, dom, abi.SLOT_DOM)
        r.raster(g, host.dom_layers_params(dom), abi.SLOT_DOM)
    r.raster(g, cam, abi.SLOT_CAMERA, scene.data_ptr())
    r.shade(cam, lights)
    r.filter(cam)
    r.composite(cam, True)
    want = outputs()
    r.render_groom(g, cam, dom if deep_opacity else None, lights)
    open_view = outputs()
    r.render_groom(g, cam, dom if deep_opacity else None, lights, scene_depth_ptr=scene.data_ptr())
    got = outputs()
    for n in names:
        _assert_equal(n, got[n].view(np.uint32), want[n].view(np.uint32))
    assert 0 < (got["CENTER"] != EMPTY).sum() < (open_view["CENTER"] != EMPTY).sum()
    g.close()


def test_light_kinds(renderer):
    """Point, spot, directional (DOM) and rect lights, given out of kind order."""
    sc = configs.config1(scale=0.05)
    cam, dom = sc.params()
    c = (sc.mesh.bounds_min + sc.mesh.bounds_max) * 0.5
    lights = pack_lights([
        Light(kind=abi.LIGHT_RECT, color=(2.0, 2.0, 2.0), position=tuple((c + [0, 400, 300]).tolist()),
              right=(1, 0, 0), up=(0, 0.6, -0.8), width=200.0, height=100.0, range=2000.0),
        Light(kind=abi.LIGHT_SPOT, color=(8e4, 6e4, 4e4), position=tuple((c + [300, 100, 300]).tolist()),
              direction=tuple((-np.array([300, 100, 300]) / np.linalg.norm([300, 100, 300])).tolist()),
              spot_scale=4.0, spot_offset=-2.5, range=1500.0),
        Light(kind=abi.LIGHT_DIRECTIONAL, color=(1.0, 1.0, 1.0), direction=(0.0, 1.0, 0.0), casts_shadows=False),
        Light(kind=abi.LIGHT_POINT, color=(5e4, 5e4, 5e4), position=tuple((c + [-300, 0, 200]).tolist()),
              range=1000.0),
        Light(kind=abi.LIGHT_DIRECTIONAL, color=(3.0, 3.0, 3.0), direction=configs.KEY_DIR, casts_shadows=True),
    ])
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights, exposure=0.7)
    assert renderer.synchronize() == 0
    center, beta, dmap = renderer.read(abi.BUF_CENTER), renderer.read(abi.BUF_BETA), renderer.read(abi.BUF_DOM)
    o_shaded, _ = oracle.shade(cam, center, beta, dmap, lights, exposure=0.7)
    np.testing.assert_allclose(renderer.read(abi.BUF_SHADED), o_shaded, rtol=SHADE_RTOL, atol=SHADE_ATOL)
    g.close()


@pytest.mark.parametrize("size, keep", [((1, 1), 1.0), ((33, 9), 1.0), ((97, 61), 0.02), ((64, 24), 0.5), ((31, 40), 0.0)])
def test_shade_lists_hair_pixels_of_partial_blocks(renderer, size, keep):
    """The shade pass lists a block's hair pixels: blocks cut by the image's
    edges, with all, some, one in fifty or none of their pixels covered, against
    the oracle's pixel by pixel shading."""
    sc = configs.config1(scale=0.02)
    sc.view = configs._camera(*size, 160.0)
    cam, dom = sc.params()
    lights = sc.light_array()
    renderer.ensure_targets(*size, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights)
    assert renderer.synchronize() == 0
    center, beta, dmap = renderer.read(abi.BUF_CENTER), renderer.read(abi.BUF_BETA), renderer.read(abi.BUF_DOM)
    center[np.random.default_rng(5).random(center.shape) >= keep] = EMPTY
    renderer.write(abi.BUF_CENTER, center)
    renderer.shade(cam, lights)
    assert renderer.synchronize() == 0
    o_shaded, o_sdepth = oracle.shade(cam, center, beta, dmap, lights)
    np.testing.assert_array_equal(renderer.read(abi.BUF_SHADED_DEPTH), o_sdepth)
    np.testing.assert_allclose(renderer.read(abi.BUF_SHADED), o_shaded, rtol=SHADE_RTOL, atol=SHADE_ATOL)
    g.close()


@pytest.mark.parametrize("tilt", [0.0, -0.3, 1e4, 1e20, -3e38])
def test_shade_at_any_tilt(renderer, tilt):
    """The cuticle tilt is any float: lobes tilted out of reach vanish."""
    sc = configs.config1(scale=0.02)
    cam, dom = sc.params()
    cam = cam.copy()
    cam["appearance"][1] = tilt
    lights = sc.light_array()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights)
    assert renderer.synchronize() == 0
    want, want_depth = oracle.shade(cam, renderer.read(abi.BUF_CENTER), renderer.read(abi.BUF_BETA),
                                    renderer.read(abi.BUF_DOM), lights)
    np.testing.assert_array_equal(renderer.read(abi.BUF_SHADED_DEPTH), want_depth)
    np.testing.assert_allclose(renderer.read(abi.BUF_SHADED), want, rtol=SHADE_RTOL, atol=SHADE_ATOL)
    assert np.isfinite(want).all()
    g.close()


def test_invalid_arguments_are_rejected(renderer):
    import ctypes as C

    lib = renderer.lib
    sc = configs.config1(scale=0.02)
    bad = sc.mesh.bundles.copy()
    bad[0]["layer_offset"] = len(sc.mesh.layers)  # past the end
    out = C.c_void_p()
    st = lib.hg_groom_upload(renderer.ctx, bad.ctypes.data, len(bad), sc.mesh.layers.ctypes.data,
                             len(sc.mesh.layers), sc.mesh.style.ctypes.data, len(sc.mesh.style), C.byref(out))
    assert st == abi.HG_INVALID_ARG and not out.value
    bad = sc.mesh.bundles.copy()
    bad[-1]["style_offset"] = len(sc.mesh.style) - 1
    st = lib.hg_groom_upload(renderer.ctx, bad.ctypes.data, len(bad), sc.mesh.layers.ctypes.data,
                             len(sc.mesh.layers), sc.mesh.style.ctypes.data, len(sc.mesh.style), C.byref(out))
    assert st == abi.HG_INVALID_ARG
    cam, dom = sc.params()
    renderer.ensure_targets(sc.view.width + 1, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    with pytest.raises(abi.HairGbError) as e:
        renderer.raster(g, cam, abi.SLOT_CAMERA)  # params screen differs from the targets
    assert e.value.status == abi.HG_INVALID_ARG
    renderer.ensure_targets(sc.view.width, sc.view.height, sc.dom_size[0] + 1, sc.dom_size[1])
    with pytest.raises(abi.HairGbError):
        renderer.raster(g, dom, abi.SLOT_DOM)  # DOM params vs map size
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    many = pack_lights([Light(kind=abi.LIGHT_POINT, color=(1, 1, 1))] * (abi.MAX_LIGHTS + 1))
    with pytest.raises(abi.HairGbError) as e:
        renderer.shade(cam, many)
    assert e.value.status == abi.HG_CAPACITY_EXCEEDED
    odd = pack_lights([Light(kind=7, color=(1, 1, 1))])
    with pytest.raises(abi.HairGbError):
        renderer.shade(cam, odd)
    with pytest.raises(abi.HairGbError):
        renderer.ensure_targets(0, 10, 0, 0)
    assert renderer.synchronize() == 0
    g.close()


def test_hair_visibility_for_receivers(renderer):
    """The deep-opacity lookup other surfaces use (hair_shadow.wesl:30-75) on
    the frame's map, against the oracle, for points through the groom."""
    import ctypes as C

    import torch

    sc = configs.config1(scale=0.05)
    cam, dom = sc.params()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, sc.light_array())
    light = np.zeros((), dtype=abi.SHADOW_LIGHT)
    assert renderer.lib.hg_shadow_light_from(dom.ctypes.data, light.ctypes.data) == abi.HG_OK
    rng = np.random.default_rng(3)
    lo, hi = sc.mesh.bounds_min - 20, sc.mesh.bounds_max + 20
    pts = np.concatenate([rng.uniform(lo, hi, size=(4000, 3)), np.ones((4000, 1))], axis=1).astype(np.float32)
    d_pts = torch.from_numpy(pts).cuda()
    d_out = torch.empty(len(pts), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    st = renderer.lib.hg_hair_visibility(renderer.ctx, light.ctypes.data, C.c_void_p(d_pts.data_ptr()), len(pts),
                                         C.c_void_p(d_out.data_ptr()))
    assert st == abi.HG_OK
    renderer.synchronize()
    got = d_out.cpu().numpy()
    dmap = renderer.read(abi.BUF_DOM)
    want = oracle.hair_visibility(np.atleast_1d(light).view(np.float32), dmap, *sc.dom_size, pts)
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-6)
    assert (want < 0.99).sum() > 100 and (want == 1.0).sum() > 100  # shadowed and unshadowed points
    g.close()


def test_async_readback_lands_before_the_next_frame_writes(renderer):
    """hg_copy_out_async: a frame's colour and depth copied on the copy stream
    while the next frame (another camera) is already enqueued; the next
    frame's writes wait for the copies on the device."""
    torch = pytest.importorskip("torch")
    sc = configs.config2(scale=0.02)
    cam_a, dom_a = sc.params()
    lights = sc.light_array()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam_a, dom_a, lights)
    want_color, want_depth = renderer.read(abi.BUF_COLOR).copy(), renderer.read(abi.BUF_DEPTH).copy()
    sc.view = configs._camera(sc.view.width, sc.view.height, 700.0, azimuth=1.1)
    cam_b, dom_b = sc.params()
    color = torch.empty(want_color.size, dtype=torch.float32, pin_memory=True)
    depth = torch.empty(want_depth.size, dtype=torch.float32, pin_memory=True)
    renderer.render_groom(g, cam_a, dom_a, lights)
    renderer.read_async(abi.BUF_COLOR, color.data_ptr(), color.numel() * 4)
    renderer.read_async(abi.BUF_DEPTH, depth.data_ptr(), depth.numel() * 4)
    renderer.render_groom(g, cam_b, dom_b, lights)
    renderer.copy_wait()
    assert renderer.synchronize() == 0
    np.testing.assert_array_equal(color.numpy(), want_color)
    np.testing.assert_array_equal(depth.numpy(), want_depth)
    other = renderer.read(abi.BUF_COLOR)
    assert np.abs(other - want_color).max() > 1e-3  # frame B did overwrite the target
    with pytest.raises(abi.HairGbError):
        renderer.read_async(abi.BUF_COLOR, color.data_ptr(), 16)
    g.close()


@pytest.mark.parametrize("model", [abi.SHADE_KARIS, abi.SHADE_SURROGATE_COMPACT])
def test_orthographic_camera(renderer, model):
    """An orthographic camera: visibility bit-exact, and the shade pass's view
    direction the camera axis (hg_shade_desc.ortho), against the oracle."""
    from bevy_hair_gb300 import surrogate as S

    sc = configs.config1(scale=0.05)
    w, h = sc.view.width, sc.view.height
    ext = float(np.max(np.asarray(sc.mesh.bounds_max) - np.asarray(sc.mesh.bounds_min)))
    half = 0.6 * ext
    proj = host.orthographic_rh(-half * w / h, half * w / h, -half, half, 1.0, 4000.0)
    view = host.View(sc.view.world_from_view, proj, w, h)
    cam, dom = host.groom_params(view, sc.groom, sc.mesh.bounds_min, sc.mesh.bounds_max, sc.mesh.bundle_count,
                                 sc.directionals, sc.dom_size)
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    assert (want["center"] != EMPTY).sum() > 100
    _check_visibility(got, want)
    lights = sc.light_array()
    s, mlp, arch = None, None, abi.MLP_ARCH_DEEP
    if model == abi.SHADE_SURROGATE_COMPACT:
        arch = abi.MLP_ARCH_COMPACT
        mlp = S.load_params(arch)
        s = S.Surrogate(renderer, mlp, arch)
        renderer.bind_surrogate(s)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights, ortho=True, model=model)
    assert renderer.synchronize() == 0
    center = renderer.read(abi.BUF_CENTER)
    _assert_equal("center", center, want["center"])
    shaded = renderer.read(abi.BUF_SHADED)
    o_shaded, _ = oracle.shade(cam, center, renderer.read(abi.BUF_BETA), renderer.read(abi.BUF_DOM), lights,
                               ortho=True, mlp=mlp, mlp_arch=arch)
    hit = center != EMPTY
    got4, want4 = shaded.reshape(-1, 4)[hit, :3], o_shaded.reshape(-1, 4)[hit, :3]
    if model == abi.SHADE_KARIS:
        np.testing.assert_allclose(shaded, o_shaded, rtol=SHADE_RTOL, atol=SHADE_ATOL)
    else:
        assert np.abs(got4 - want4).sum() / np.abs(want4).sum() < 2e-3
    # the perspective view direction gives a different picture
    o_persp, _ = oracle.shade(cam, center, renderer.read(abi.BUF_BETA), renderer.read(abi.BUF_DOM), lights,
                              ortho=False, mlp=mlp, mlp_arch=arch)
    assert np.abs(o_persp.reshape(-1, 4)[hit, :3] - want4).max() > 1e-3
    if s is not None:
        renderer.bind_surrogate(None)
        s.close()
    g.close()


@pytest.mark.parametrize("name", ["config1", "config2", "config3"])
def test_full_size_visibility_bit_exact(renderer, name):
    """The configurations at full size (config 2 is the benchmark workload:
    100k strands, 1920x1080, DOM 1024^2): LOD records, refs, G-buffer words
    and both DOM passes equal to the oracle's."""
    sc = getattr(configs, name)(scale=1.0)
    cam, dom = sc.params()
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    assert (want["center"] != EMPTY).sum() > 20_000
    _check_visibility(got, want)


def test_dom_pass_over_part_of_the_bundles(renderer):
    """A DOM view over the first half of the bundles (pass_mode.y): the depth
    pass cannot use the hashed order of a full draw and must fall back to the
    refs' own order; the map stays bit-exact."""
    sc = configs.config2(scale=0.02)
    cam, dom = sc.params()
    dom = dom.copy()
    dom["pass_mode"][1] = max(1, sc.mesh.bundle_count // 2)
    got = _visibility(renderer, sc, cam, dom)
    want = _oracle_visibility(sc, cam, dom)
    assert int(got["dom_indirect"][0]) < sc.mesh.strand_count()
    assert (want["dom_depth"][: sc.dom_size[0] * sc.dom_size[1]] != 0xFFFFFFFF).any()
    _check_visibility(got, want)


def _camera_scenes():
    """Scenes for the two camera raster kinds: a plain one, deep overdraw, the
    camera inside the groom (segments cut by the near plane span the screen
    and take the long-segment path), a close-up whose segments cross several
    32x32 tiles, and forward Z with a scene depth buffer."""
    def inside():
        sc = configs.config2(scale=0.01)
        c = (sc.mesh.bounds_min + sc.mesh.bounds_max) * 0.5
        wfv = host.looking_at(c + np.array([0, 0, 20.0], np.float32), c + np.array([0, 0, -100.0], np.float32))
        sc.view = host.View(wfv, sc.view.clip_from_view, sc.view.width, sc.view.height)
        return sc, None

    def close_up():
        sc = configs.config1(scale=0.05)
        sc.view = configs._camera(1024, 768, 160.0)
        return sc, None

    def dense():
        sc = configs.config2(scale=0.25)
        sc.view = configs._camera(384, 216, 900.0)
        sc.dom_size = (192, 192)
        return sc, None

    def scene_depth():
        sc = configs.config1(scale=0.05)
        v = sc.view
        sc.view = host.View(v.world_from_view, host.perspective_rh(math.pi / 4, v.width / v.height, 0.1, 5000.0),
                            v.width, v.height)
        rng = np.random.default_rng(6)
        depth = np.where(rng.random(v.width * v.height) < 0.5, np.float32(1.0), np.float32(0.9990))
        return sc, depth.astype(np.float32)

    return {"config3": lambda: (configs.config3(scale=0.01), None), "inside": inside, "close_up": close_up,
            "dense": dense, "scene_depth": scene_depth}


@pytest.mark.parametrize("mode", [abi.CAMERA_RASTER_BINNED, abi.CAMERA_RASTER_DIRECT])
@pytest.mark.parametrize("name", list(_camera_scenes()))
def test_camera_raster_kinds_bit_exact(renderer, name, mode):
    """hg_set_camera_raster: the binned pass (tiles resolved in shared memory)
    and the direct pass (global atomics) both give the oracle's G-buffer."""
    sc, scene_depth = _camera_scenes()[name]()
    cam, _ = sc.params()
    renderer.set_camera_raster(mode)
    try:
        got = _visibility(renderer, sc, cam, None, scene_depth)
    finally:
        renderer.set_camera_raster(abi.CAMERA_RASTER_DIRECT)
    want = _oracle_visibility(sc, cam, None, scene_depth)
    assert (want["center"] != EMPTY).sum() > 50
    _check_visibility(got, want, with_dom=False)


def test_set_camera_raster_rejects_unknown_modes(renderer):
    assert renderer.lib.hg_set_camera_raster(renderer.ctx, 7) == abi.HG_INVALID_ARG


_REF = os.environ.get("BEVY_HAIR_REFERENCE")


@pytest.mark.skipif(not _REF or not (Path(_REF) / "assets" / "hair" / "woman.obj").exists(),
                    reason="the reference's grooms are not present (set BEVY_HAIR_REFERENCE)")
@pytest.mark.parametrize("name", ["wStraight", "wCurly"])
def test_reference_groom_frame_against_the_oracle(renderer, name):
    """A real groom (the reference's Yuksel asset, 50,000 strands, baked
    against woman.obj) through hg_groom_frame at 960x540: LOD records, G-buffer
    words and the deep opacity map bit-exact with the oracle's frame, colour
    within the shading tolerance."""
    hair = Path(_REF) / "assets" / "hair"
    if not (hair / f"{name}.hair").exists():
        pytest.skip(f"{name}.hair is not present")
    sc = configs.real_groom(hair / f"{name}.hair", hair / "woman.obj", 960, 540, 512)
    cam, dom = sc.params()
    lights = sc.light_array()
    renderer.ensure_targets(sc.view.width, sc.view.height, *sc.dom_size)
    g = renderer.upload(sc.mesh)
    renderer.render_groom(g, cam, dom, lights)
    assert renderer.synchronize() == 0
    want = oracle.frame(sc.mesh, cam, dom, lights)
    _assert_equal("center", renderer.read(abi.BUF_CENTER), want["center"])
    _assert_equal("conservative", renderer.read(abi.BUF_CONSERVATIVE), want["cons"])
    _assert_equal("beta", renderer.read(abi.BUF_BETA), want["beta"])
    _assert_equal("dom", renderer.read(abi.BUF_DOM), want["dom"])
    assert (want["center"] != EMPTY).sum() > 20_000
    np.testing.assert_allclose(renderer.read(abi.BUF_SHADED), want["shaded"], rtol=2e-3, atol=1e-5)
    g.close()
