"""Calls beside one another and at their limits."""
import ctypes as C

import numpy as np
import pytest

from oracle_lib import x2

pytestmark = pytest.mark.gpu
DEEP = 300  # beyond the wavefront's eight bits a path's depth


def closed_room(ctx, max_depth, width=32, height=24):
    """A closed room of one bright grey around the box's camera and light, no roulette: every path goes on to max_depth."""
    s = x2.SyntheticScene(0)
    d, cfg = s.desc, x2.Config.from_buffer_copy(s.config)
    corners = np.array([[x, y, z] for x in (-6, 6) for y in (-6, 6) for z in (-6, 6)], np.float32)
    quads = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    triangles = np.array([t for a, b, c, e in quads for t in ((a, b, c), (a, c, e))], np.uint32)
    first, material = np.array([0, 12], np.uint32), np.zeros(1, np.uint32)
    keep = [np.ascontiguousarray(corners.reshape(-1)), np.ascontiguousarray(triangles.reshape(-1)), first, material]
    d.vertex_count, d.triangle_count, d.mesh_count = 8, 12, 1
    d.vertices, d.triangles = keep[0].ctypes.data_as(C.POINTER(C.c_float)), keep[1].ctypes.data_as(C.POINTER(C.c_uint32))
    d.mesh_first, d.mesh_material = first.ctypes.data_as(C.POINTER(C.c_uint32)), material.ctypes.data_as(C.POINTER(C.c_uint32))
    for c in range(3):
        d.materials[0].diffuse[c] = 0.98
    cfg.width, cfg.height, cfg.rr_threshold = width, height, 0.0
    cfg.max_depth = cfg.max_diffuse_depth = cfg.max_glossy_depth = cfg.max_mirror_depth = max_depth
    return s, cfg, x2.Scene(ctx, d, cfg)


def one_thread(scene, pixels, indices):
    """integratePairs's samples: a counting call takes that kernel."""
    scene.count_traversal(True)
    out = scene.integrate(pixels, indices)
    scene.count_traversal(False)
    return out


@pytest.mark.parametrize("max_depth", [255, 256, DEEP])  # the deepest that the wavefront form takes, and beyond
def test_deep_paths_equal_one_thread_a_sample(ctx, max_depth):
    s, cfg, scene = closed_room(ctx, max_depth)
    rng = np.random.default_rng(1)
    pixels, indices = rng.integers(0, cfg.width * cfg.height, 200, dtype=np.uint32), np.arange(200, dtype=np.uint32)
    rgba, status = scene.integrate(pixels, indices)
    want, want_status = one_thread(scene, pixels, indices)
    scene.free()
    assert (want_status == x2.DONE).all() and (want[:, 3] == 1).all()
    assert np.array_equal(status, want_status)
    assert np.array_equal(rgba, want)


def test_unfinished_samples_are_not_handed_out(ctx):
    """Samples that the per-sample entry did not finish, in an early window of a long list or after an earlier call on the
    same buffers: an error, or the right samples, never something else as done."""
    import torch

    s, cfg, scene = closed_room(ctx, 4)
    n, some = (1 << 22) + 37, 100
    pixels = np.full(n, cfg.width * cfg.height, np.uint32)  # no such pixel: an error at once
    pixels[:some] = np.random.default_rng(2).integers(0, cfg.width * cfg.height, some, dtype=np.uint32)
    indices = np.arange(n, dtype=np.uint32)
    scene.integrate(pixels[:some], indices[:some])  # what an unfinished sample would find in its place
    deep = x2.Config.from_buffer_copy(cfg)
    deep.max_depth = deep.max_diffuse_depth = DEEP
    scene.set_config(deep)
    want, _ = one_thread(scene, pixels[:some], indices[:some])
    # The device entry.
    pairs = torch.tensor(np.stack([pixels[:some], indices[:some]], 1).astype(np.int64)).to(torch.int32).cuda()
    rgba, status = torch.zeros((some, 4), dtype=torch.float64, device="cuda"), torch.zeros(some, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    call = x2.library().x2_integrate_device
    assert call(scene.handle, pairs.data_ptr(), some, rgba.data_ptr(), status.data_ptr()) == x2.OK
    ctx.synchronize()
    done = (status == x2.DONE).cpu().numpy()
    assert np.array_equal(rgba.cpu().numpy()[done], want[done])
    assert (status[~torch.tensor(done)] == x2.ERROR).all()
    # The host entry, over two windows.
    try:
        got, got_status = scene.integrate(pixels, indices)
        assert np.array_equal(got[:some], want) and (got_status[:some] == x2.DONE).all()
        assert (got_status[some:] == x2.ERROR).all()
    except x2.X2Error as e:
        assert e.code == x2.EDEVICE
    scene.free()


def test_integrate_without_room_for_its_outputs(ctx):
    """The samples' outputs do not fit the device: the one-thread kernel, which needs none, takes the call."""
    import torch

    s, cfg, scene = closed_room(ctx, 4)
    n, small = 1 << 22, 1 << 20
    rng = np.random.default_rng(4)
    pairs = torch.tensor(np.stack([rng.integers(0, cfg.width * cfg.height, n), np.arange(n)], 1)).to(torch.int32).cuda()
    rgba, status = torch.zeros((n, 4), dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    call = x2.library().x2_integrate_device
    torch.cuda.synchronize()
    assert call(scene.handle, pairs.data_ptr(), small, rgba.data_ptr(), status.data_ptr()) == x2.OK
    ctx.synchronize()
    want = rgba[:small].clone()
    one_thread(scene, np.zeros(1, np.uint32), np.zeros(1, np.uint32))  # that kernel's local memory is there from here on
    rgba.zero_()
    held = []
    while (free := torch.cuda.mem_get_info()[0]) > 32 << 20:
        held.append(torch.empty(max(free - (24 << 20), 2 << 20) & ~((2 << 20) - 1), dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    try:
        rc = call(scene.handle, pairs.data_ptr(), n, rgba.data_ptr(), status.data_ptr())
        ctx.synchronize()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert rc == x2.OK
    assert (status == x2.DONE).all() and torch.equal(rgba[:small], want)
    scene.free()


@pytest.mark.parametrize("entry", ["integrate", "trace_rays"])
def test_long_lists_do_not_wait_for_other_streams(entry):
    """A list beyond the context's kept scratch, with another stream of the program at work: the call ends first. (A context
    of its own: one that has put by its most graphs destroys them first, which waits.)"""
    import torch

    own = x2.Context(0)
    s, cfg, scene = closed_room(own, 2)
    n = 1600000  # over 64 MB at 44 bytes
    rng = np.random.default_rng(5)
    if entry == "integrate":
        args = (rng.integers(0, cfg.width * cfg.height, n, dtype=np.uint32), np.arange(n, dtype=np.uint32))
    else:
        rays = np.zeros((n, 8), np.float32)
        rays[:, 3:6] = rng.normal(size=(n, 3))
        rays[:, 7] = 100.0
        args = (rays,)
    call = getattr(scene, entry)
    want = call(*args)
    few = [a[:300] for a in args]
    call(*few)
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(10)
        other.synchronize()
        torch.cuda._sleep(2000000000)  # about a second
        done = torch.cuda.Event()
        done.record()
    got = call(*args)
    waited = done.query()
    other.synchronize()
    own.close()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert not waited


def test_scenes_share_the_context_s_memory(ctx):
    """What per-sample calls and plain frames work in belongs to the context: more scenes hold no more of it."""
    import torch

    scenes = [x2.Scene(ctx, s.desc, s.config) for s in [x2.SyntheticScene(108) for _ in range(4)]]
    cfg = scenes[0].config
    pixels = np.random.default_rng(6).integers(0, cfg.width * cfg.height, 1 << 19, dtype=np.uint32)

    def use(scene):
        rgba, status = scene.integrate(pixels, np.arange(len(pixels), dtype=np.uint32))
        scene.frame_begin(1)
        scene.render_frame(0, 1)
        scene.wait()
        return rgba, scene.film()[0]

    first = use(scenes[0])
    before = torch.cuda.mem_get_info()[0]
    for scene in scenes[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(use(scene), first))
    after = torch.cuda.mem_get_info()[0]
    for scene in scenes:
        scene.free()
    assert before - after < 64 << 20  # films, chunk lists and counters


def test_build_memory(ctx):
    """The BVH build's peak in the device's pool, a triangle: no more than the 384 bytes of the build without the wide nodes'
    cost tables."""
    lib = C.CDLL("libcuda.so.1")
    pool, high, zero = C.c_void_p(), C.c_uint64(), C.c_uint64(0)
    assert lib.cuDeviceGetDefaultMemPool(C.byref(pool), ctx.device) == 0
    s = x2.SyntheticScene(11)
    x2.Scene(ctx, s.desc, s.config).free()
    ctx.synchronize()
    current = C.c_uint64()
    assert lib.cuMemPoolGetAttribute(pool, 7, C.byref(current)) == 0
    assert lib.cuMemPoolSetAttribute(pool, 8, C.byref(zero)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    x2.Scene(ctx, s.desc, s.config).free()
    assert lib.cuMemPoolGetAttribute(pool, 8, C.byref(high)) == 0
    each = (high.value - current.value) / s.desc.triangle_count
    print(f"build peak: {each:.1f} bytes a triangle")
    assert each < 385


def test_one_scene_every_call_in_turn(ctx):
    """Frames, samples, rays and adaptive frames on one scene, with the seed, the size, the samples and the launch shape
    changed between them, each as a scene that has done nothing else gives it."""
    s = x2.SyntheticScene(0)
    base = s.config

    def config(seed, width, height):
        cfg = x2.Config.from_buffer_copy(base)
        cfg.seed, cfg.width, cfg.height = seed, width, height
        return cfg

    rays = np.zeros((700, 8), np.float32)
    rays[:, 3:6] = np.random.default_rng(7).normal(size=(700, 3))
    rays[:, 7] = 50.0

    def frame(scene, plain, spp):
        scene.frame_begin(spp)
        (scene.render_frame if plain else scene.render_frame_wavefront)(0, spp)
        scene.wait()
        return scene.film()

    def adaptive(scene, cellular):
        result = scene.render_adaptive(4, 32, 0.01, cellular)
        return (result["passes"], result["samples"], *scene.film(odd=True))

    def samples(scene, n):
        r = np.random.default_rng(n)
        return scene.integrate(r.integers(0, scene.config.width * scene.config.height, n, dtype=np.uint32), np.arange(n, dtype=np.uint32))

    a, b, c = config(1, 90, 50), config(2, 90, 50), config(1, 40, 70)
    shape = {"paths": 2048, "light_split": 0}
    turns = [(a, {}, lambda x: frame(x, False, 3)), (a, {}, lambda x: frame(x, False, 3)), (a, {}, lambda x: samples(x, 1000)),
             (b, {}, lambda x: samples(x, 1000)), (b, {}, lambda x: frame(x, False, 3)), (b, {}, lambda x: frame(x, False, 2)),
             (a, {}, lambda x: adaptive(x, False)), (a, {}, lambda x: adaptive(x, False)), (a, {}, lambda x: samples(x, 30000)),
             (a, {}, lambda x: frame(x, False, 3)), (c, {}, lambda x: adaptive(x, True)), (a, {}, lambda x: adaptive(x, True)),
             (c, {}, lambda x: adaptive(x, True)), (c, shape, lambda x: frame(x, False, 3)), (c, shape, lambda x: samples(x, 30000)),
             (c, {}, lambda x: frame(x, True, 3)), (a, {}, lambda x: frame(x, True, 5)), (a, {}, lambda x: x.trace_rays(rays)),
             (a, {}, lambda x: frame(x, False, 3)), (a, {}, lambda x: samples(x, 1000))]
    scene = x2.Scene(ctx, s.desc, base)
    for k, (cfg, tune, turn) in enumerate(turns):
        scene.set_config(cfg)
        scene.wavefront_tune(**tune)
        got = turn(scene)
        alone = x2.Scene(ctx, s.desc, cfg)
        alone.wavefront_tune(**tune)
        want = turn(alone)
        alone.free()
        exact = k < 15 or k > 16  # the plain form adds a pixel's samples in the order they finish
        for g, w in zip(got, want):
            assert np.array_equal(g, w) if exact else np.allclose(g, w, rtol=1e-12, atol=1e-12), k
    scene.free()


def test_sample_lists_that_share_a_launch(ctx):
    """Lists of lengths about the steps that a launch's slots are rounded to, longer and shorter ones in turn: each list's own
    samples, whatever the last one left in its place."""
    s = x2.SyntheticScene(0)
    scene = x2.Scene(ctx, s.desc, s.config)
    rng = np.random.default_rng(8)
    lengths = [2048, 2000, 2047, 1, 1024, 1023, 1025, 1152, 1153, 2049, 2176, 2177, 2100, 2048, 5, 36864, 36865, 34000, 36864]
    lists = [(rng.integers(0, s.config.width * s.config.height, n, dtype=np.uint32), rng.integers(0, 1 << 16, n, dtype=np.uint32)) for n in lengths]
    got = [scene.integrate(*each) for each in lists]
    want, want_status = one_thread(scene, np.concatenate([p for p, _ in lists]), np.concatenate([i for _, i in lists]))
    scene.free()
    assert np.array_equal(np.concatenate([r for r, _ in got]), want)
    assert np.array_equal(np.concatenate([t for _, t in got]), want_status)
