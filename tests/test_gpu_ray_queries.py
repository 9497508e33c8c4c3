"""Ray queries at the edges of their split over warps, and rays that no camera makes."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hikari_b200 as hk  # noqa: E402
from hikari_b200 import scenes  # noqa: E402

CENTRE = torch.tensor([0.0, 1.0, 0.0])


@pytest.fixture(scope="module")
def scene():
    """A displaced sphere of 20480 triangles over a quad."""
    return hk.Scene.from_desc(scenes.mesh_heavy("plastic", width=32, height=32, depth=8, level=5, env_res=(64, 32), seed=1))


def _rays(n, seed):
    g = torch.Generator().manual_seed(seed)
    to = CENTRE + 2 * torch.rand(n, 3, generator=g) - 1
    fr = CENTRE + 3 * (2 * torch.rand(n, 3, generator=g) - 1)
    r = torch.empty(n, 8)
    r[:, :3], r[:, 3:6], r[:, 6], r[:, 7] = fr, to - fr, 1e-4, math.inf
    return r


def _trace(scene, rays, any_hit):
    return [x.cpu().numpy() for x in scene.trace(rays.cuda(), any_hit=any_hit)[:1 if any_hit else 4]]


# around one claim, one block of four warps, every warp with 32 rays (148 x 32 x 32) and with 128, the most
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 148 * 32 * 32 - 1, 148 * 32 * 32, 148 * 32 * 33 + 1,
                               148 * 32 * 128, 148 * 32 * 128 + 129])
@pytest.mark.parametrize("any_hit", [False, True])
def test_every_ray_is_answered(scene, n, any_hit):
    """A ray's answer does not depend on the rays beside it: the same rays backwards, bit for bit."""
    r = _rays(n, n)
    if any_hit:
        r[:, 7] = 1 - 1e-4
    got, back = _trace(scene, r, any_hit), _trace(scene, r.flip(0), any_hit)
    for a, b in zip(got, back):
        assert np.array_equal(a, b[::-1])
    miss = got[0] == (0 if any_hit else -1)
    assert n < 100 or (miss.any() and not miss.all())


def _odd(case, n=20000):
    r = _rays(n, 7)
    k = torch.arange(n)
    if case == "empty range":
        r[:, 6], r[:, 7] = 1.0, 0.5
    elif case == "in a plane":
        r[:, 3] = 0.0
    elif case == "along an axis":
        r[:, 3], r[:, 4] = 0.0, -0.0
    elif case == "no direction":
        r[:, 3:6] = 0.0
    elif case == "nan direction":
        r[k, 3 + k % 3] = math.nan
    elif case == "infinite direction":
        r[k, 3 + k % 3] = math.inf
    elif case == "nan origin":
        r[k, k % 3] = math.nan
    elif case == "infinite origin":
        r[k, k % 3] = -math.inf
    elif case == "nan range":
        r[k, 6 + k % 2] = math.nan
    return r


MISSES = ("empty range", "no direction", "nan direction", "infinite direction", "nan origin", "infinite origin", "nan range")


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("case", MISSES)
def test_rays_without_an_answer_miss(scene, case, any_hit):
    assert (_trace(scene, _odd(case), any_hit)[0] == (0 if any_hit else -1)).all()


@pytest.mark.parametrize("case", ["in a plane", "along an axis"])
def test_rays_along_axes(scene, case):
    """Zero components: the same occlusion in the binary tree, whose any-hit test is the same arithmetic."""
    r = _odd(case)
    wide = _trace(scene, r, True)[0]
    scene.set_accel(hk.ACCEL_BVH2)
    binary = _trace(scene, r, True)[0]
    scene.set_accel(hk.ACCEL_BVH8)
    assert np.array_equal(wide, binary) and (wide == 0).any() and (wide == 1).any()
