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
