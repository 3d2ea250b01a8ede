"""The whole-path kernel against the wavefront.

A timed call (enable_timing) runs every bounce as separate launches; an untimed one hands waves of
few paths, and the last bounces of larger ones, to the whole-path kernel. Both compute every path
alike, so images, counts and statistics are equal bit for bit. Sizes: one path, a warp and one more,
fewer paths than the kernel's grid has warps and lanes, several paths per lane, the largest wave
that runs whole and one above it (which hands over, or, in the closed white furnace where no path
ends, does not), and several waves in flight.
"""
import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200 import _ffi
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu

NEE = {"none": {}, "dmis": dict(direct_light_sampling=1), "emis": dict(env_importance_sampling=1)}


def random_scene(width, height, depth, masked=False):
    s = lx.random_scene(seed=9, total_tris=30_000, num_instances=12, min_tris=500, max_tris=6000, num_emissive=3,
                        num_textures=4, texture_size=64, env_width=64, env_height=32, width=width, height=height,
                        trace_depth=depth)
    if masked:  # every other material decides its hits by texture alpha: masked, then blended
        for k in range(0, s.desc.num_materials, 2):
            m = s.desc.materials[k]
            m.albedo_tex, m.alpha_cutoff = 3, 0.5
            m.alpha_mode = _ffi.ALPHA_MASK if k % 4 else _ffi.ALPHA_BLEND
            m.albedo_tt.rotation, m.albedo_tt.scale[0], m.albedo_tt.offset[1] = 0.3, 1.7, 0.21
    return s


def both_ways(scene, first, spp, **kw):
    out = []
    for timed in (True, False):
        r = lx.Renderer(scene, default_options(**kw))
        r.enable_timing(timed)
        r.render(first, spp)
        st = r.stats()
        out.append((r.image_sum().view(np.uint32), np.array(r.wave_counts(16)),
                    [st[k] for k in ("rays_radiance", "rays_shadow", "path_bounces", "samples")]))
        r.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


@pytest.mark.parametrize("nee", list(NEE))
@pytest.mark.parametrize("layout", [_ffi.BVH_SINGLE_LEVEL, _ffi.BVH_TWO_LEVEL], ids=["single", "two"])
@pytest.mark.parametrize("width,height,spp,depth", [(1, 1, 1, 1), (33, 1, 1, 7), (61, 37, 1, 12), (256, 250, 1, 3),
                                                    (300, 220, 4, 5), (700, 450, 1, 6)])
def test_whole_paths_equal_wavefront(nee, layout, width, height, spp, depth):
    both_ways(random_scene(width, height, depth), 5, spp, bvh_layout=layout, **NEE[nee])


def test_alpha_tested_paths():
    both_ways(random_scene(160, 120, 8, masked=True), 2, 2, env_importance_sampling=1)


@pytest.mark.parametrize("height", [444, 445])
def test_largest_whole_wave(height):
    # 640 * 444 = 284160 paths: five per lane of a grid of 3 blocks on 148 SMs
    both_ways(random_scene(640, height, 4), 1, 1, env_importance_sampling=1)


def test_closed_white_scene_stays_a_wavefront():
    both_ways(lx.furnace(700, 500, subdiv=8, metallic=0.0, roughness=1.0, ior=1.0), 1, 1, trace_depth=9)


def test_waves_in_flight():
    both_ways(random_scene(320, 200, 9), 1, 7, env_importance_sampling=1, spp_per_wave=2)


def test_compensated_and_split_calls():
    s = random_scene(97, 41, 6)
    kw = dict(direct_light_sampling=1, precision=_ffi.PRECISION_COMPENSATED)
    both_ways(s, 3, 3, **kw)
    a, b = lx.Renderer(s, default_options(**kw)), lx.Renderer(s, default_options(**kw))
    a.render(3, 3)
    for i in range(3):
        b.render_iter(3 + i)
    assert np.array_equal(a.image_sum().view(np.uint32), b.image_sum().view(np.uint32))
    a.close()
    b.close()
