"""The wavefront's shade kernels for one BSDF type, textured and perturbed,
and the megakernel's spread of few paths over its warps.

Both forms walk the same sample streams.  The megakernel evaluates every
material with the BSDF that looks its textures up at each use; a shade queue's
kernel looks them up once per vertex.  The arithmetic is the same, so the
images agree up to the order of the film's float additions (a few hundred
terms per pixel at 2^-24 each: 1e-5 relative, and 1e-6 of the largest value
where terms cancel) and the ray counts exactly."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hikari_b200 as hk  # noqa: E402
from hikari_b200 import scenes  # noqa: E402
from hikari_b200.scenedesc import (BSDF_BUMP_MAP, BSDF_NORMAL_MAP, BSDF_TWO_SIDED, TEX_CHECKERBOARD,  # noqa: E402
                                   BSDFDesc, TextureDesc)

TEXTURED = dict(scenes.textured_materials())


def _both(sd, spp):
    gs = hk.Scene.from_desc(sd)
    out = []
    for form in (hk.FORM_MEGAKERNEL, hk.FORM_WAVEFRONT):
        gs.set_image_form(form)
        img, ctr = gs.render_image(spp, 8, seed=11)
        out.append((np.asarray(img, np.float64), ctr))
    (a, ca), (b, cb) = out
    scale = float(np.abs(a).max())
    assert scale > 0
    assert tuple(ca[:3]) == tuple(cb[:3]), f"rays, shadow rays, dropped: {ca[:3]} vs {cb[:3]}"
    assert np.allclose(a, b, rtol=1e-5, atol=1e-6 * scale), f"max abs difference {np.abs(a - b).max():.3e} of {scale}"


@pytest.mark.parametrize("over", ["plain", "bump", "normal", "two_sided"])
@pytest.mark.parametrize("name", sorted(TEXTURED))
def test_textures_looked_up_once_per_vertex(name, over):
    """Spheres of one textured BSDF: its own queue, the queue of a bump or normal map over it, and two-sided (generic)."""
    b = TEXTURED[name]
    bumps = TextureDesc(kind=TEX_CHECKERBOARD, count=6, a=[0.01] * 3, b=[0.0] * 3)
    normals = TextureDesc(kind=TEX_CHECKERBOARD, count=6, a=[0.6, 0.5, 0.95], b=[0.45, 0.55, 0.95])
    if over == "bump":
        b = BSDFDesc(type=BSDF_BUMP_MAP, nested=b, textures={"kd": bumps})
    elif over == "normal":
        b = BSDFDesc(type=BSDF_NORMAL_MAP, nested=b, textures={"kd": normals})
    elif over == "two_sided":
        if "dielectric" in name:
            pytest.skip("twoSided refuses a transmissive BSDF")
        b = BSDFDesc(type=BSDF_TWO_SIDED, nested=b)
    sd = scenes.lights_scene(width=29, height=23, shading_normals=True, textured=True, bitmap=True)
    for m in sd.meshes[1:6]:
        m.bsdf = b
    _both(sd, 4)


# one path; under and over one path per scheduler's warp (592 of 148 SMs); the last sizes of partly and of fully filled warps
@pytest.mark.parametrize("size", [(1, 1), (24, 24), (25, 24), (135, 136), (138, 138)])
def test_few_paths_are_spread_over_the_warps(size):
    _both(scenes.lights_scene(width=size[0], height=size[1], shading_normals=True, textured=True), 1)
