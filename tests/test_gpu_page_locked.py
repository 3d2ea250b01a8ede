"""Caller rays where the library finds no page-locked host memory.

lux_test_fail_pinned (luxion_b200/csrc/host_common.h) makes the calling thread's requests for
page-locked blocks fail on the host and counts them."""
import ctypes as C

import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu

MANY = 1 << 20


def fail_pinned(calls):
    f = lx.lib().lux_test_fail_pinned
    f.restype, f.argtypes = C.c_int, [C.c_int]
    return f(calls)


@pytest.fixture(scope="module")
def renderer():
    s = lx.random_scene(seed=3, total_tris=30_000, num_instances=12, min_tris=500, max_tris=6000, num_textures=4,
                        texture_size=64, env_width=0, env_height=0, width=64, height=64)
    r = lx.Renderer(s, default_options())
    yield r
    r.close()


def some_rays(n, seed=1):
    g = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = g.uniform((-12, 0.2, -12), (12, 8, 12), (n, 3))
    d = g.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3] = g.uniform(1.0, 40.0, n)
    return rays


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_static_call_asks_for_no_page_locked_memory(renderer, mode):
    rays = some_rays(5000)
    want = renderer.trace_rays_static(rays, mode, 1)
    fail_pinned(MANY)
    try:
        got = renderer.trace_rays_static(rays, mode, 1)
    finally:
        left = fail_pinned(0)
    assert np.array_equal(got, want)
    assert left == MANY


def test_static_call_of_a_context_made_without_page_locked_memory(renderer):
    rays = some_rays(5000)
    want = renderer.trace_rays_static(rays, 0, 1)
    s = lx.random_scene(seed=3, total_tris=30_000, num_instances=12, min_tris=500, max_tris=6000, num_textures=4,
                        texture_size=64, env_width=0, env_height=0, width=64, height=64)
    resident = lx.ResidentScene(s, default_options())
    fail_pinned(MANY)
    try:
        r = lx.Renderer(resident, default_options(), camera=s.desc.camera)
        got = r.trace_rays_static(rays, 0, 1)
    finally:
        fail_pinned(0)
    assert np.array_equal(got, want)
    r.close()


@pytest.mark.parametrize("n", [1, 5000])
def test_call_without_page_locked_memory_for_the_error_word(renderer, n):
    rays = some_rays(n)
    want = renderer.trace_rays_static(rays, 0, 1)
    fail_pinned(MANY)
    try:
        got = renderer.trace_rays(rays, 0, 1)
    finally:
        left = fail_pinned(0)
    assert np.array_equal(got, want)
    assert left < MANY


def page_locked(shape, dtype):
    import torch
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


@pytest.mark.parametrize("n", [131_071, 131_072, 209_715, 209_716])
@pytest.mark.parametrize("rays_locked,hits_locked", [(True, True), (True, False), (False, True)])
def test_page_locked_buffers_are_not_staged(renderer, n, rays_locked, hits_locked):
    # the library asks for one block for the error word, and for one per buffer that it stages:
    # pageable ones of 4 MB (131,072 rays, 209,716 hits) and more
    import torch
    rays = some_rays(n)
    want = renderer.trace_rays(rays, 0, 1)
    hits = np.zeros((n, 5), np.uint32)
    if rays_locked:
        src, rays = rays, page_locked((n, 8), torch.float32)
        rays[:] = src
    if hits_locked:
        hits = page_locked((n, 5), torch.int32).view(np.uint32)
    fail_pinned(MANY)
    try:
        rc = lx.lib().lux_trace_rays(renderer._h, lx.ptr(rays), n, 0, 1, lx.ptr(hits, C.c_uint32))
    finally:
        asked = MANY - fail_pinned(0)
    assert rc == 0 and np.array_equal(hits, want)
    assert asked == 1 + (not rays_locked and n >= 131_072) + (not hits_locked and n >= 209_716)


class NoThreads:
    """No thread can be started meanwhile: the default stack is larger than the address space."""

    def __enter__(self):
        self.libc, self.old, new = C.CDLL(None), C.create_string_buffer(256), C.create_string_buffer(256)
        assert self.libc.pthread_getattr_default_np(self.old) == 0
        assert self.libc.pthread_attr_init(new) == 0
        assert self.libc.pthread_attr_setstacksize(new, C.c_size_t(1 << 47)) == 0
        assert self.libc.pthread_setattr_default_np(new) == 0

    def __exit__(self, *exc):
        assert self.libc.pthread_setattr_default_np(self.old) == 0


@pytest.mark.parametrize("staging", [True, False], ids=["staging", "no-staging"])
@pytest.mark.parametrize("threads", [True, False], ids=["threads", "no-threads"])
@pytest.mark.parametrize("n", [131_073, 262_145])
def test_large_batches_without_threads_or_staging(renderer, n, threads, staging):
    rays = some_rays(n)
    step = 50_021
    want = np.concatenate([renderer.trace_rays_static(rays[i:i + step], 0, 1) for i in range(0, n, step)])
    renderer.trace_rays(rays, 0, 1)
    fail_pinned(0 if staging else MANY)
    try:
        if threads:
            got = renderer.trace_rays(rays, 0, 1)
        else:
            with NoThreads():
                got = renderer.trace_rays(rays, 0, 1)
    finally:
        fail_pinned(0)
    assert np.array_equal(got, want)
