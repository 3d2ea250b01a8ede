"""The ray sort's output: the queue in the order of a stable sort by the rays' Morton keys
(lux_morton_sort against numpy's stable argsort of lux_morton_keys).

Sizes at the ends of a warp and of a tile of 4096 items, and more tiles than the launch has blocks;
keys spread over the scene, few different ones, all equal, and all of rays that miss the scene's box
(0xFFFFFFFF); and several bounces in a row, as the counter sets alternate between them."""
import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu

BIG = 592 * 4096 + 77


@pytest.fixture(scope="module")
def renderer():
    s = lx.random_scene(seed=5, total_tris=20_000, num_instances=8, min_tris=500, max_tris=8000, num_textures=2,
                        texture_size=64, env_width=64, env_height=32, width=1280, height=960, trace_depth=6)
    r = lx.Renderer(s, default_options(ray_sorting=1, spp_per_wave=2))
    yield r
    r.close()


def rays_of(kind, n, seed):
    g = np.random.default_rng(seed)
    m = {"spread": n, "few": 5, "equal": 1, "miss": n}[kind]
    r = np.zeros((m, 8), np.float32)
    r[:, 0:3] = g.uniform((-12, 0.2, -12), (12, 8, 12), (m, 3))
    d = g.normal(size=(m, 3))
    if kind == "miss":
        r[:, 1] += 1e4
        d[:, 1] = np.abs(d[:, 1])
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return r if m == n else r[g.integers(0, m, n)]


@pytest.mark.parametrize("n", [1, 31, 33, 4095, 4096, 4097, 100_003, BIG])
@pytest.mark.parametrize("kind", ["spread", "few", "equal", "miss"])
@pytest.mark.parametrize("bounce", [0, 1, 4])
def test_order_is_the_stable_sort_by_key(renderer, n, kind, bounce):
    rays = rays_of(kind, n, n + bounce)
    plain = renderer.morton_keys(rays)
    want = np.argsort(plain, kind="stable")
    keys, order = renderer.morton_sort(rays, bounce)
    assert np.array_equal(order, want)
    assert np.array_equal(keys, plain[want])
    if kind == "miss":
        assert np.all(plain == 0xFFFFFFFF)
    elif kind == "spread" and n > 1000:
        assert np.unique(plain).size > n // 20


def test_arguments(renderer):
    rays = rays_of("spread", 10, 1)
    assert renderer.morton_sort(rays[:0])[1].size == 0
    with pytest.raises(lx.LuxError) as e:
        renderer.morton_sort(rays, 64)
    assert e.value.code == -1
    with pytest.raises(lx.LuxError) as e:
        renderer.morton_sort(rays_of("spread", 1280 * 960 * 2 + 1, 1))
    assert e.value.code == -1
    r = lx.Renderer(lx.cornell36(32, 32), default_options())
    with pytest.raises(lx.LuxError) as e:
        r.morton_sort(rays)
    assert e.value.code == -7
    r.close()
