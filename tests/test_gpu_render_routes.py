"""Renders whose form, pool or launches the library chooses, at the lines of
those rules (the rules themselves: test_host_routes.py)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hikari_b200 as hk  # noqa: E402
from hikari_b200 import scenes  # noqa: E402
from hikari_b200.scenedesc import BSDF_DIFFUSE, BSDFDesc, CameraDesc, FilterDesc, MeshDesc, SceneDesc  # noqa: E402


def _closed_room(side):
    """A cube without openings, seen from inside: a path ends at its depth or in roulette alone."""
    sd = SceneDesc()
    c = [np.float32([x, y, z]) for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)]
    for q in ((0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)):
        p, i = scenes.quad(*(c[k] for k in q))
        n = np.cross(p[i[0][1]] - p[i[0][0]], p[i[0][2]] - p[i[0][0]])
        if np.dot(n, p.mean(0)) > 0:   # facing inwards
            i = i[:, ::-1].copy()
        sd.meshes.append(MeshDesc(p, i, BSDFDesc(type=BSDF_DIFFUSE, kd=[0.9, 0.9, 0.9])))
    lp, li = scenes.quad((-0.2, 0.99, -0.2), (0.2, 0.99, -0.2), (0.2, 0.99, 0.2), (-0.2, 0.99, 0.2))
    if np.cross(lp[li[0][1]] - lp[li[0][0]], lp[li[0][2]] - lp[li[0][0]])[1] > 0:
        li = li[:, ::-1].copy()
    sd.meshes.append(MeshDesc(lp, li, BSDFDesc(type=BSDF_DIFFUSE, kd=[0.5, 0.5, 0.5]), radiance=[4.0, 5.0, 6.0]))
    sd.camera = CameraDesc(side, side, scenes.look_at((0, 0, 0.9), (0, 0, 0), (0, 1, 0)), 60.0, 1e-4, 1e4)
    sd.filter = FilterDesc(2, 2.0, 0.5)
    return sd


def _launches(gs, which=0):
    n = C.c_int32()
    buf = np.zeros(1, np.uint32)
    hk.check(hk.lib().hk_wavefront_launch_log(gs.h, which, buf.ctypes.data, 1, C.byref(n)))
    return n.value


def test_render_of_more_passes_than_a_launch_of_the_loop_holds():
    """2^20 paths of 64 vertices in a pool of 2^10 slots: 2^16 iterations, a launch of the loop ends after 2^15.
    The film's weights say that every path was splatted once: up to 1024 terms a pixel (64 samples, 16 filter taps) in
    any order, 2^-24 each; the mean radiance may differ by what a few of the 2^26 rays that graze an edge change."""
    gs = hk.Scene.from_desc(_closed_room(128))
    gs.set_wavefront_config(dict(capacity=1024))
    films = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_AUTO):
        gs.set_image_form(form)
        film = torch.zeros(gs.film_shape(), device="cuda")
        gs.render(film, 64, 64, seed=3, rr_start=64)
        films.append(film.cpu().numpy().astype(np.float64))
    assert _launches(gs) > 1 << 15
    a, b = films
    assert np.allclose(a[..., 3], b[..., 3], rtol=1024 * 2.0 ** -24)
    assert abs(b[..., :3].mean() / a[..., :3].mean() - 1) < 1e-4


def test_negative_sample_offsets_and_image_indices_in_both_forms():
    """The same streams, so the same image up to the order of the film's additions (64 samples x 16 taps: 2^-24 each)."""
    gs = hk.Scene.from_desc(scenes.cornell_box(width=128, height=128))
    films = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_AUTO):
        gs.set_image_form(form)
        film = torch.zeros(gs.film_shape(), device="cuda")
        gs.render(film, 8, 4, seed=3, sample_offset=-5, image_index=-2)
        films.append(film.cpu().numpy().astype(np.float64))
    a, b = films
    assert np.allclose(a, b, rtol=1024 * 2.0 ** -24, atol=1e-6 * float(a.max()))


def test_first_render_beside_a_capture():
    """A stream is captured in the default mode while a scene renders for the first time on another stream, which makes
    its pool: the capture stays whole, and so does the image (64 samples x 16 taps a pixel, 2^-24 each)."""
    sd = scenes.cornell_box(width=256, height=256)
    x = torch.zeros(1024, device="cuda")
    films = [torch.zeros(hk.Scene.from_desc(sd).film_shape(), device="cuda") for _ in range(2)]
    gs, ref = hk.Scene.from_desc(sd), hk.Scene.from_desc(sd)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        gs.render(films[0], 2, 8, seed=3, stream=side)
    assert _launches(gs) > 0   # the wavefront
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1024
    ref.render(films[1], 2, 8, seed=3)
    a, b = (f.cpu().numpy() for f in films)
    assert np.allclose(a, b, rtol=1024 * 2.0 ** -24, atol=1e-6 * float(b.max()))


def test_counters_shared_by_renders_of_both_forms():
    """Renders of two scenes on two streams add to one counter array: small ones in the megakernel, whose warps add as
    they end, and large ones in the wavefront, which adds once per render.  Ray counts of a seed do not vary."""
    small, large = (hk.Scene.from_desc(scenes.cornell_box(width=128, height=128)), hk.Scene.from_desc(
        scenes.cornell_box(width=512, height=256)))
    films = [torch.zeros(s.film_shape(), device="cuda") for s in (small, large)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    one = [torch.zeros(5, dtype=torch.int64, device="cuda") for _ in range(2)]
    both = torch.zeros(5, dtype=torch.int64, device="cuda")
    for s, f, c in zip((small, large), films, one):
        s.render(f, 1, 8, seed=3, counters=c)
    torch.cuda.synchronize()
    n = (160, 40)
    for k in range(40):
        for j in range(4):
            small.render(films[0], 1, 8, seed=3, counters=both, stream=streams[0])
        large.render(films[1], 1, 8, seed=3, counters=both, stream=streams[1])
    torch.cuda.synchronize()
    assert _launches(large) > 0
    want = n[0] * one[0].cpu().numpy() + n[1] * one[1].cpu().numpy()
    assert tuple(both.cpu().numpy()[:3]) == tuple(want[:3])


# one path; a lane of every warp and one more path; the last count that is spread and the first in full warps; all resident
# lanes and more paths than they are, so that lanes take a second one; ragged tiles throughout
@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((592, 1), 1), ((593, 1), 1), ((128, 74), 1), ((9473, 1), 1), ((37, 29), 9),
                                      ((592, 64), 1), ((641, 67), 1), ((211, 101), 4)])
@pytest.mark.parametrize("scene", ["cornell_box", "cornell_smooth", "lights_scene"])
def test_megakernel_deals_every_path_once(scene, size, spp):
    """Against the wavefront: the same streams; the samples of 25 pixels, and the up to 64 terms of each, in any order."""
    kw = dict(textured=True, bitmap=True, bump=True, shading_normals=True) if scene == "lights_scene" else {}
    gs = hk.Scene.from_desc(getattr(scenes, scene)(width=size[0], height=size[1], **kw))
    out = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_WAVEFRONT):
        gs.set_image_form(form)
        out.append(gs.render_image(spp, 12, seed=5))
    (a, ca), (b, cb) = out
    assert tuple(ca[:3]) == tuple(cb[:3])
    terms = 25 * spp + 64
    assert np.allclose(a, b, rtol=terms * 2.0 ** -23, atol=terms * 2.0 ** -24 * float(np.abs(a).max()))


def _room(width, height):
    return scenes.cornell_box(width=width, height=height)


def _sky(width, height):
    return scenes.mesh_heavy("conductor", width=width, height=height, depth=12, level=3, env_res=(32, 16), seed=2)


def _textured_sky(width, height):
    return scenes.lights_scene(width=width, height=height, textured=True, bitmap=True, bump=True, shading_normals=True)


# as many paths as are resident (148 x 256 lanes); two more, in rounds of blocks of 128 threads; 131000, near the last of those;
# 2^17 and more, of 256 threads; several samples over ragged tiles
@pytest.mark.parametrize("size,spp", [((592, 64), 1), ((421, 90), 1), ((131, 1000), 1), ((512, 256), 1), ((257, 511), 1), ((37, 29), 123)])
@pytest.mark.parametrize("scene,depth,accel", [(_room, 6, hk.ACCEL_BVH8), (_room, 2, hk.ACCEL_BVH2), (_sky, 12, hk.ACCEL_BVH8),
                                               (_sky, 12, hk.ACCEL_BVH2), (_textured_sky, 12, hk.ACCEL_BVH8),
                                               (_textured_sky, 12, hk.ACCEL_BVH2)])
def test_rounds_deal_every_path_once(size, spp, scene, depth, accel):
    """Against the wavefront, as test_megakernel_deals_every_path_once."""
    gs = hk.Scene.from_desc(scene(*size))
    gs.set_accel(accel)
    out = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_WAVEFRONT):
        gs.set_image_form(form)
        out.append(gs.render_image(spp, depth, seed=5))
    (a, ca), (b, cb) = out
    assert tuple(ca[:3]) == tuple(cb[:3])
    terms = 25 * spp + 64
    assert np.allclose(a, b, rtol=terms * 2.0 ** -23, atol=terms * 2.0 ** -24 * float(np.abs(a).max()))
