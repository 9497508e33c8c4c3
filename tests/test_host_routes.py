"""The library's host decisions -- form, pool, launches, streams, devices,
memory -- against a CUDA runtime of host memory (fake_cuda.cpp): its own host
sources, compiled with g++, over a fake that logs what would be launched."""
import concurrent.futures
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import hikari_b200 as hk
from hikari_b200 import build, scenes, serving

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = [os.path.join(build.CSRC, f) for f in build.SOURCES if f.endswith(".cpp")] + [os.path.join(HERE, "fake_cuda.cpp")]


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake_cuda")
    so = str(out / "libhikari_fake.so")

    def compile_one(src):
        obj = str(out / (os.path.basename(src) + ".o"))
        subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-pthread", "-I/usr/local/cuda/include", "-I" + build.CSRC, "-c",
                        src, "-o", obj], check=True)
        return obj

    with concurrent.futures.ThreadPoolExecutor() as pool:
        objs = list(pool.map(compile_one, SOURCES))
    # -Bsymbolic: the fake's entry points, also where a real runtime is loaded already
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic,--no-undefined", "-o", so] + objs + ["-lz", "-lpthread"], check=True)
    return so


class Fake:
    """The fake's controls."""

    def __init__(self, so):
        L = C.CDLL(so)
        L.fake_log.restype = C.c_char_p
        L.fake_live.restype = C.c_size_t
        L.fake_limit.argtypes = [C.c_size_t]
        L.fake_passes_left.restype = C.c_uint64
        L.fake_stream.restype = C.c_void_p
        self.L = L

    def log(self):
        """What was launched since the last call."""
        text = self.L.fake_log().decode().split("\n")[:-1]
        self.L.fake_clear()
        return text

    def forms(self):
        """The forms of the renders since the last call, one word per render."""
        return [x.split()[0] for x in self.log() if x.startswith(("mega", "begin"))]

    def live(self):
        return self.L.fake_live()


@pytest.fixture
def fake(fake_lib, monkeypatch):
    monkeypatch.setattr(hk, "LIB_PATH", fake_lib)
    monkeypatch.setattr(hk, "_lib", None)
    f = Fake(fake_lib)
    f.made = []
    f.log()
    yield f
    f.L.fake_limit(C.c_size_t(-1).value)
    f.L.fake_device(0)
    f.L.fake_other_capture(0)
    f.L.fake_user_capturing(0)
    f.L.fake_fail_instantiate(0)
    for s in f.made:   # while the fake is the library
        s.close()


def _scene(fake, width=64, height=64, lights=1):
    """A Cornell box; lights > 1: as many area lights."""
    sd = scenes.cornell_box(width=width, height=height)
    light = next(m for m in sd.meshes if m.radiance is not None)
    for k in range(lights - 1):
        sd.meshes.append(light)
    s = hk.Scene.from_desc(sd)
    fake.made.append(s)
    fake.log()
    return s


def _render(s, spp, depth=16, **kw):
    film = np.zeros(4, np.float32)   # the fake writes no film
    s.render(film, spp, depth, stream=0, **kw)


# 2^29 paths of depth 64; 2^25 of depth 1000; 2^19 of depth 64 in the least pool; the deepest that the path state holds
@pytest.mark.parametrize("width,spp,depth,capacity", [(256, 8192, 64, 0), (256, 16384, 64, 0), (1024, 32, 1000, 0),
                                                      (64, 128, 64, 1024), (256, 2, 65535, 0)])
def test_long_and_deep_renders_stay_on_the_wavefront(fake, width, spp, depth, capacity):
    s = _scene(fake, width, width)
    if capacity:
        s.set_wavefront_config(dict(capacity=capacity))
    _render(s, spp, depth)
    assert fake.forms() == ["begin"]
    # as many launches of the loop as the work can need if every path reaches its depth
    assert fake.L.fake_passes_left() == 0


def _devices(log):
    return [x.split()[x.split().index("device") + 1] for x in log if x.startswith("loop")]


def test_render_on_another_device_than_the_scenes(fake):
    """The megakernel, which runs where the caller is; the scene's pool stays on the scene's device."""
    s = _scene(fake, 512, 512)
    fake.L.fake_device(1)
    _render(s, 1)
    assert fake.forms() == ["mega"]
    fake.L.fake_device(0)
    _render(s, 1)
    log = fake.log()
    assert any(x.startswith("begin") for x in log) and _devices(log) == ["0"]


def test_batch_pools_belong_to_the_current_device(fake):
    s = _scene(fake)
    film = np.zeros(4, np.float32)
    for device in (1, 0, 0, 1):
        fake.L.fake_device(device)
        s.render_batch([film], 1, 8, stream=0)
        assert _devices(fake.log()) == [str(device)]


def _pool(s, fake, **kw):
    """Bytes that a batch's pool takes."""
    film, before = np.zeros(4, np.float32), fake.live()
    s.render_batch([film], 1, 8, stream=0, **kw)
    return fake.live() - before


# the second pool finds no memory beside the first: the first, idle, makes room
def test_a_fitted_pool_may_take_the_place_of_a_sized_one(fake):
    s = _scene(fake, 512, 512)
    film = np.zeros(4, np.float32)
    _pool(s, fake, capacity=1 << 20)
    fake.L.fake_limit(fake.live() + (1 << 20))
    s.render_batch([film], 1, 8, stream=0)
    assert [x for x in fake.log() if x.startswith("loop")][-1].endswith("capacity 262144")
    s.render_batch([film], 1, 8, stream=0, capacity=1 << 20)
    assert [x for x in fake.log() if x.startswith("loop")][-1].endswith("capacity 1048576")


def test_a_film_render_takes_the_place_of_a_sized_pool_once(fake):
    s = _scene(fake, 512, 512)
    _pool(s, fake, capacity=1 << 20)
    fake.L.fake_limit(fake.live() + (1 << 20))
    fake.log()
    _render(s, 1)
    _render(s, 1)
    log = fake.log()
    assert [x.split()[0] for x in log if x.startswith(("mega", "begin"))] == ["begin", "begin"]
    assert log.count("malloc-failed") == 1


def test_the_megakernel_form_gives_the_film_pool_back(fake):
    """A pool that a caller sized stays: hk_render_batch goes on using it."""
    s = _scene(fake, 512, 512)
    before = fake.live()
    _render(s, 1)
    assert fake.live() > before + (1 << 20)
    s.set_image_form(hk.FORM_MEGAKERNEL)
    assert fake.live() == before
    _render(s, 1)
    assert fake.live() == before
    s.set_image_form(hk.FORM_AUTO)
    sized = _pool(s, fake, capacity=1 << 20)
    s.set_image_form(hk.FORM_MEGAKERNEL)
    assert fake.live() == before + sized


def _image(s, spp):
    d = hk.render_desc(spp, 16)
    out = np.zeros((s.desc.camera.height, s.desc.camera.width, 3), np.float32)
    hk.check(hk.lib().hk_render_image(s.h, C.byref(d), out.ctypes.data, None, None))


def _store(s, **kw):
    c = hk.WavefrontConfig()
    for k, v in kw.items():
        setattr(c, k, v)
    hk.check(hk.lib().hk_scene_set_wavefront_config(s.h, C.byref(c)))


@pytest.mark.parametrize("field", ["threads_extend", "threads_shade"])
@pytest.mark.parametrize("threads", [100, 288])
def test_a_stored_configuration_that_the_pool_refuses(fake, field, threads):
    """hk_render, which does not need it, renders with the megakernel; hk_render_image too, except for the large images
    (2^22 paths of 256 x 256 pixels) that it has always refused then."""
    s = _scene(fake, 512, 512)
    _store(s, **{field: threads})
    _render(s, 1)
    _image(s, 15)
    assert fake.forms() == ["mega", "mega"]
    with pytest.raises(hk.HikariError):
        _image(s, 16)
    with pytest.raises(hk.HikariError):
        s.render_batch([np.zeros(4, np.float32)], 1, 8, stream=0, **{field: threads})


def test_a_stored_configuration_without_graphs(fake):
    """hk_render, which returns at once, has no loop without a graph; hk_render_image waits and launches kernel by kernel."""
    s = _scene(fake, 512, 512)
    _store(s, no_graph=1)
    _render(s, 16)
    assert fake.forms() == ["mega"]
    for spp in (1, 16):
        _image(s, spp)
        log = fake.log()
        assert "plain" in log and not any(x.startswith(("mega", "loop")) for x in log)
    s2 = _scene(fake, 64, 64)   # below 2^17 paths
    _store(s2, no_graph=1)
    _image(s2, 1)
    assert fake.forms() == ["mega"]


def test_whole_images_on_another_device(fake):
    """hk_render_image waits, so it may make a pool there."""
    s = _scene(fake, 512, 512)
    fake.L.fake_device(1)
    _image(s, 1)
    assert _devices(fake.log()) == ["1"]
    fake.L.fake_device(0)
    s = _scene(fake, 512, 512)
    _store(s, no_graph=1)
    fake.L.fake_limit(fake.live() + (8 << 20))   # the image's buffers, but no pool
    _image(s, 1)
    assert fake.forms() == ["mega"]


# 2^17 paths and more; 2^22 and more of 65536 pixels and more are refused, as they have always been
@pytest.mark.parametrize("width,height", [(16385, 8), (8, 16385)])
@pytest.mark.parametrize("no_graph", [0, 1])
def test_images_of_more_pixels_a_side_than_a_job_may_have(fake, width, height, no_graph):
    s = _scene(fake, width, height)
    if no_graph:
        _store(s, no_graph=1)
    _render(s, 1)
    _image(s, 31)   # below 2^22 paths
    assert fake.forms() == ["mega", "mega"]
    with pytest.raises(hk.HikariError):
        _image(s, 32)
    _render(s, 32)
    assert fake.forms() == ["mega"]
    s = _scene(fake, width - 1 if width > height else width, height - 1 if height > width else height)
    _render(s, 1)
    assert fake.forms() == ["begin"]


def test_negative_sample_offsets_and_image_indices(fake):
    """hk_render takes both as signed numbers of 64 bits, in either form."""
    s = _scene(fake, 512, 512)
    _render(s, 1, sample_offset=-5, image_index=-2)
    assert [x for x in fake.log() if x.startswith("begin")] == ["begin slots 262144 sample -5 image -2"]


def test_film_render_without_room_for_the_loops_graph(fake):
    s = _scene(fake, 512, 512)
    fake.L.fake_fail_instantiate(1)
    _render(s, 1)
    assert fake.forms() == ["mega"]
    fake.L.fake_fail_instantiate(0)
    _render(s, 1)
    assert fake.forms() == ["begin"]


def test_pools_are_made_beside_a_capture(fake):
    """A capture in the default mode forbids other threads, and its own thread on other streams, to allocate; hk_render
    did not allocate before it had a pool, so its allocations must not break a capture."""
    s = _scene(fake, 512, 512)
    fake.L.fake_other_capture(1)
    _render(s, 1)     # makes the pool and the loop's graph
    _render(s, 16)    # replaces the pool by a larger one
    assert fake.forms() == ["begin", "begin"]
    assert not fake.L.fake_capture_broken()


def _priorities(log):
    return [x.split()[2] for x in log if x.startswith("loop")]


def test_film_renders_keep_the_callers_priority(fake):
    """The pool's streams have the least and the greatest priority; a batch runs at the least, as it always has."""
    s = _scene(fake, 512, 512)
    film = np.zeros(4, np.float32)
    seen = []
    for priority in (0, -1, -5, 0):
        stream = fake.L.fake_stream(0, priority)
        s.render(film, 1, 8, stream=stream)
        seen += _priorities(fake.log())
    s.render(film, 1, 8, stream=fake.L.fake_stream(0, -5))
    fake.log()
    s.render_batch([film], 1, 8, stream=fake.L.fake_stream(0, -5))
    seen += _priorities(fake.log())
    assert seen == ["0", "-5", "-5", "0", "0"]


def _autotune(s):
    d, best, ms = hk.render_desc(1, 8), hk.WavefrontConfig(), C.c_float()
    hk.check(hk.lib().hk_wavefront_autotune(s.h, C.byref(d), C.byref(best), C.byref(ms)))
    return best.capacity


# lights x 2^22 slots: below 2^31, at it (2^21 fits), past it for every candidate (2^20 x 2048 = 2^31): the fitted pool
@pytest.mark.parametrize("lights,capacities", [(511, [1 << 20, 1 << 21, 1 << 22]), (512, [1 << 20, 1 << 21]), (1024, [1 << 20]),
                                               (2048, [1 << 16])])
def test_the_autotuner_tries_the_pools_that_fit(fake, lights, capacities):
    s = _scene(fake, 512, 512, lights)
    assert _autotune(s) == capacities[0]   # the fake's clock finds none faster than the first
    tried = []
    for x in fake.log():
        if x.startswith("loop"):
            c = int(x.split()[-1])
            if c not in tried:
                tried.append(c)
    assert tried == capacities


@pytest.mark.parametrize("lights", [4095, 4096, 9000])
def test_a_served_scene_of_many_lights(fake, lights):
    """2^19 slots x 4096 lights are 2^31 shadow records: the scene gets a smaller pool, the server goes on."""
    s = _scene(fake, 64, 64, lights)
    srv = serving.Server()
    try:
        jid, out = srv.submit(srv.add_scene(s), 1, 8, 0)
        srv.wait(jid, 60)
    finally:
        srv.close()
    slots = {int(x.split()[-1]) for x in fake.log() if x.startswith("pair")}
    assert slots == {1 << 19 if lights < 4096 else 1 << (18 if lights < 8192 else 17)}


# 148 x 4 warps: a lane each, 16 each, then full warps; more warps than are resident wait for none: 148 x 2 blocks of 4
@pytest.mark.parametrize("width,height,spp,lanes,grid", [(1, 1, 1, 1, 1), (592, 1, 1, 1, 148), (593, 1, 1, 2, 75), (592, 16, 1, 16, 148),
                                                         (9473, 1, 1, 32, 75), (64, 64, 4, 32, 128), (592, 64, 1, 32, 296),
                                                         (592, 128, 1, 32, 296)])
def test_few_paths_are_spread_over_one_warp_per_scheduler(fake, width, height, spp, lanes, grid):
    s = _scene(fake, width, height)
    _render(s, spp)
    assert fake.log() == [f"mega grid {grid} lanes {lanes}"]


def test_a_film_render_pins_no_host_memory(fake):
    """Its job and plan go to the device with a launch: pinned memory, most of what a pool costs to make, is the batch's."""
    s = _scene(fake, 512, 512)
    before = fake.L.fake_pinned()
    _render(s, 1)
    assert fake.forms() == ["begin"] and fake.L.fake_pinned() == before
    _pool(s, fake)
    assert fake.L.fake_pinned() == before + 1
    _render(s, 1)
    _pool(s, fake)
    assert fake.L.fake_pinned() == before + 1


def _sky(fake, width, height, material="conductor"):
    s = hk.Scene.from_desc(scenes.mesh_heavy(material, width=width, height=height, depth=8, level=1, env_res=(8, 4)))
    fake.made.append(s)
    fake.log()
    return s


# 148 x 256 lanes are resident: blocks of 128 threads, two an SM; of 256 threads, one an SM, where 2^17 paths start in rounds
def test_the_blocks_of_the_megakernel(fake):
    for make, depth, grids in ((_scene, 6, (296, 296, 148)), (_scene, 7, (296, 296, 296)), (_sky, 64, (296, 296, 148)),
                               (lambda *a: _sky(*a, "dielectric"), 7, (296, 296, 296))):
        for width, height, grid in ((592, 64, grids[0]), (511, 256, grids[1]), (512, 256, grids[2])):
            s = make(fake, width, height)
            s.set_image_form(hk.FORM_MEGAKERNEL)
            _render(s, 1, depth)
            assert fake.log() == [f"mega grid {grid} lanes 32"]


def _smooth(fake, width, height):
    s = hk.Scene.from_desc(scenes.cornell_smooth(width=width, height=height))
    fake.made.append(s)
    fake.log()
    return s


def _textures(fake, width, height):
    s = hk.Scene.from_desc(scenes.lights_scene(width=width, height=height, textured=True))
    fake.made.append(s)
    fake.log()
    return s


# paths x 2^-15: the last that the megakernel renders is a row less
@pytest.mark.parametrize("make,depth,line", [(_smooth, 3, 4), (_smooth, 4, 1), (_smooth, 16, 1), (_smooth, 17, 2), (_sky, 8, 4),
                                             (_sky, 9, 8), (_sky, 16, 8), (_sky, 17, 12), (_textures, 8, 4), (_textures, 9, 5),
                                             (_textures, 16, 5), (_textures, 17, 12), (_scene, 3, 8), (_scene, 4, 4), (_scene, 16, 4), (_scene, 17, 10),
                                             (_scene, 1024, 10), (_scene, 1025, 4)])
def test_the_line_between_the_forms(fake, make, depth, line):
    for height, form in ((32 * line - 1, "mega"), (32 * line, "begin")):
        s = make(fake, 1024, height)
        _render(s, 1, depth)
        _image(s, 1) if depth == 16 else None
        assert set(fake.forms()) == {form}
