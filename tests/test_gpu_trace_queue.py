"""The wavefront's per-warp queue of triangle tests and its pool at the sizes
where they can go wrong: leaf groups that overfill the ring, warps with fewer
rays than lanes, pools smaller than the work, images with partial tiles.

The megakernel traces the same sample streams one ray per thread and tests
each ray's triangles in order, so images agree up to the order of the film's
float additions (a few hundred terms per pixel at 2^-24 each: 1e-5 relative,
and 1e-6 of the largest value where terms cancel) and ray counts exactly."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hikari_b200 as hk  # noqa: E402
from hikari_b200 import scenes  # noqa: E402
from hikari_b200.scenedesc import BSDF_DIFFUSE, BSDFDesc, CameraDesc, FilterDesc, MeshDesc, SceneDesc  # noqa: E402


def _sheets(n, width, height):
    """n large triangles facing the camera, one behind another and jittered, so that a ray meets most of their
    boxes in one node, lit by a quad beside the camera."""
    rng = np.random.default_rng(n)
    sd = SceneDesc()
    pos, idx = [], []
    for k in range(n):
        z = -0.05 * k + 0.01 * rng.random()
        c = rng.uniform(-0.3, 0.3, 2)
        for a in (0.5, 2.6, 4.7):   # counter-clockwise as seen from +z
            pos.append((c[0] + 1.2 * np.cos(a), c[1] + 1.2 * np.sin(a), z))
        idx.append((3 * k, 3 * k + 1, 3 * k + 2))
    sd.meshes.append(MeshDesc(np.float32(pos), np.uint32(idx), BSDFDesc(type=BSDF_DIFFUSE, kd=[0.7, 0.6, 0.5])))
    lp, li = scenes.quad((-1, 2, 1), (1, 2, 1), (1, 2, 3), (-1, 2, 3))
    n0 = np.cross(lp[1] - lp[0], lp[2] - lp[0])
    if n0[1] > 0:
        lp = lp[::-1].copy()
    sd.meshes.append(MeshDesc(lp, li, BSDFDesc(type=BSDF_DIFFUSE, kd=[0.0, 0.0, 0.0]), radiance=[4.0, 5.0, 6.0]))
    sd.camera = CameraDesc(width, height, scenes.look_at((0, 0.2, 3.0), (0, 0, 0), (0, 1, 0)), 50.0, 1e-4, 1e4)
    sd.filter = FilterDesc(2, 2.0, 0.5)
    sd.depth = 8
    return sd


def _agree(a, ca, b, cb):
    scale = float(np.abs(a).max())
    assert scale > 0
    assert tuple(ca[:3]) == tuple(cb[:3]), f"rays, shadow rays, dropped: {ca[:3]} vs {cb[:3]}"
    assert np.allclose(a, b, rtol=1e-5, atol=1e-6 * scale), f"max abs difference {np.abs(a - b).max():.3e} of {scale}"


# 1 and 3: one leaf; 24: a node full of three-triangle leaves (32 lanes x 24 tests overfill the ring); 25, 70: beyond
@pytest.mark.parametrize("n", [1, 3, 24, 25, 70])
@pytest.mark.parametrize("size", [(1, 1), (37, 29)])
def test_queued_triangle_tests_agree_with_the_serial_order(n, size):
    gs = hk.Scene.from_desc(_sheets(n, *size))
    gs.set_image_form(hk.FORM_MEGAKERNEL)
    a, ca = gs.render_image(16, 8, seed=5)
    gs.set_image_form(hk.FORM_WAVEFRONT)
    for idle in (0, 1, 32):
        gs.set_wavefront_config(dict(fetch_min_idle=idle, fetch_min_idle_shadow=idle))
        b, cb = gs.render_image(16, 8, seed=5)
        _agree(a, ca, b, cb)


# pools of 1024 slots (the least) against 33 x 17 and 80 x 56 x 8 paths; 0: fitted to the work, then reused for less and for more
@pytest.mark.parametrize("no_graph", [False, True])
def test_pool_sizes_render_the_same_images(no_graph):
    sd = scenes.cornell_box(width=80, height=56)
    gs = hk.Scene.from_desc(sd)
    sizes = [(33, 17), (80, 56), (16, 16)]
    ref = None
    for capacity, spp in ((1024, 8), (0, 1), (0, 8), (0, 2), (1 << 16, 8)):
        films = [torch.zeros(gs.film_shape(w, h), device="cuda") for w, h in sizes]
        ctr = torch.zeros(7, dtype=torch.int64, device="cuda")
        gs.render_batch(films, spp, sd.depth, seeds=[1, 2, 3], sizes=sizes, counters=ctr, capacity=capacity,
                        no_graph=no_graph)
        if spp != 8:
            continue
        got = np.concatenate([f.cpu().numpy().astype(np.float64).reshape(-1) for f in films])
        c = ctr.cpu().numpy()
        if ref is None:
            ref = (got, c)
        _agree(ref[0], ref[1], got, c)


# 512 x 512 x 1 and 256 x 256 x 4: 2^18 paths; 511 x 256 x 1: below the least that hk_render gives to the wavefront, 2^17; 1024 x 257: ragged
@pytest.mark.parametrize("size,spp", [((512, 512), 1), ((256, 256), 4), ((511, 512), 1), ((512, 256), 1), ((511, 256), 1), ((1024, 257), 1)])
def test_queued_film_renders_agree_with_the_megakernel(size, spp):
    sd = scenes.cornell_box(width=size[0], height=size[1])
    gs = hk.Scene.from_desc(sd)
    out = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_AUTO):
        gs.set_image_form(form)
        film = torch.zeros(gs.film_shape(), device="cuda")
        ctr = torch.zeros(5, dtype=torch.int64, device="cuda")
        for k in range(3):   # three calls on the stream, none waited for
            gs.render(film, spp, sd.depth, seed=7, sample_offset=k * spp, counters=ctr)
        out.append((film.cpu().numpy().astype(np.float64), ctr.cpu().numpy()))
    _agree(*out[0], *out[1])


def test_film_render_is_still_captured():
    """A capture of hk_render holds the megakernel whatever the size: a graph with a loop cannot be captured."""
    sd = scenes.cornell_box(width=512, height=512)
    gs = hk.Scene.from_desc(sd)
    film, ref = (torch.zeros(gs.film_shape(), device="cuda") for _ in range(2))
    gs.render(ref, 2, sd.depth, seed=3)   # the wavefront
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        gs.render(film, 2, sd.depth, seed=3)
    film.zero_()
    g.replay()
    torch.cuda.synchronize()
    a, b = ref.cpu().numpy(), film.cpu().numpy()
    assert np.allclose(a, b, rtol=1e-5, atol=1e-6 * float(np.abs(a).max()))


# first bounces of 151552 rays: 32 for each warp of 148 x 4 blocks, none left to claim; 151560: one claim of 8; 152144, 302253: the
# parts of the rest ragged, the last ones empty or cut; capacity 1 << 17: all dealt
@pytest.mark.parametrize("size", [(592, 256), (421, 360), (592, 257), (777, 389)])
@pytest.mark.parametrize("threads", [128, 256])
def test_each_ray_of_a_queue_is_claimed_once(size, threads):
    sd = scenes.cornell_box(width=size[0], height=size[1])
    gs = hk.Scene.from_desc(sd)
    gs.set_image_form(hk.FORM_MEGAKERNEL)
    a, ca = gs.render_image(1, 6, seed=2)
    gs.set_image_form(hk.FORM_WAVEFRONT)
    for capacity in (1 << 17, 1 << 19):
        gs.set_wavefront_config(dict(capacity=capacity, threads_extend=threads))
        b, cb = gs.render_image(1, 6, seed=2)
        _agree(a, ca, b, cb)


def test_pool_with_many_emitters():
    """1100 area lights: a pool of 2^18 slots would hold more than 2^28 shadow records, the fitted one holds fewer.
    A path's radiance is a sum of 1100 terms a vertex in any order: 2^-24 each. A capacity that needs 2^31 is refused."""
    sd = scenes.cornell_box(width=512, height=512)
    lp, li = scenes.quad((0, 0, 0), (0.01, 0, 0), (0.01, 0, 0.01), (0, 0, 0.01))
    for k in range(1099):
        off = np.float32([-0.9 + 0.05 * (k % 36), 1.97, -0.9 + 0.05 * (k // 36)])
        sd.meshes.append(MeshDesc(lp + off, li, BSDFDesc(type=BSDF_DIFFUSE, kd=[0.0, 0.0, 0.0]), radiance=[9.0, 8.0, 7.0]))
    gs = hk.Scene.from_desc(sd)
    out = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_AUTO):
        gs.set_image_form(form)
        film = torch.zeros(gs.film_shape(), device="cuda")
        ctr = torch.zeros(5, dtype=torch.int64, device="cuda")
        gs.render(film, 1, 2, seed=7, counters=ctr)
        out.append((film.cpu().numpy().astype(np.float64), ctr.cpu().numpy()))
    (a, ca), (b, cb) = out
    assert tuple(ca[:3]) == tuple(cb[:3])
    assert np.allclose(a, b, rtol=1100 * 2.0 ** -24, atol=1e-6 * float(np.abs(a).max()))
    with pytest.raises(hk.HikariError):
        gs.render_batch([film], 1, 2, seeds=[1], capacity=1 << 21)


# powers of two: every coordinate, and so every distance and box, scales exactly; the last camera stands 2^40.9 away
@pytest.mark.parametrize("exponent,away,fov", [(-6, 3.8, 40.0), (0, 3.8, 40.0), (30, 3.8, 40.0), (30, 1945.6, 0.08)])
def test_scaled_scenes(exponent, away, fov):
    f = np.float32(2.0 ** exponent)
    sd = scenes.cornell_box(width=32, height=32)
    for m in sd.meshes:
        m.positions = m.positions * f
    sd.camera = CameraDesc(32, 32, scenes.look_at((0, 1 * f, away * f), (0, 1 * f, 0), (0, 1, 0)), fov, float(1e-4 * f),
                           float(1e4 * f))
    gs = hk.Scene.from_desc(sd)
    gs.set_image_form(hk.FORM_MEGAKERNEL)
    a, ca = gs.render_image(16, 8, seed=5)
    gs.set_image_form(hk.FORM_WAVEFRONT)
    b, cb = gs.render_image(16, 8, seed=5)
    _agree(a, ca, b, cb)
