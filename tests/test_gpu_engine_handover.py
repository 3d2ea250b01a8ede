"""Jobs submitted while an earlier wave of the job engine is still in flight although the
whole-path kernel has finished it.

The scene is a closed white room, whose paths almost all reach bounce 3, where the engine hands a
wave over when no work waits. The steps: wave A runs bounces 0 to 2; nothing waits, so A is finished
from bounce 3 on; B is submitted and runs bounces 0 to 2 beside A; the next hand-over covers A,
already finished, and B. A third wave follows in the same way. Each image and the total of traced
rays equal the single-job renders' bit for bit. Sizes: a few hundred paths, and 100,000, which is
more than one path and less than two per lane of the whole-path grid (56,832 lanes on 148 SMs).
"""
import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200 import _ffi
from luxion_b200._ffi import default_options
from luxion_b200.scene_builder import SceneBuilder, look_at_camera

pytestmark = pytest.mark.gpu

DEPTH = 12
LANES = 56_832
NEE = {"none": {}, "dmis": dict(direct_light_sampling=1), "emis": dict(env_importance_sampling=1)}


def room(width, height):
    sb = SceneBuilder(width, height, trace_depth=DEPTH)
    v = np.array([[x, y, z] for x in (-2, 2) for y in (-2, 2) for z in (-2, 2)], np.float32)
    tris = []
    for a in range(3):
        for s in (-2, 2):
            q = [i for i in range(8) if v[i, a] == s]
            q = [q[0], q[1], q[3], q[2]]
            for t in ([q[0], q[1], q[2]], [q[0], q[2], q[3]]):
                n = np.cross(v[t[1]] - v[t[0]], v[t[2]] - v[t[0]])
                tris.append(t if n[a] * s < 0 else [t[0], t[2], t[1]])  # facing the inside
    sb.add_instance(sb.add_mesh(v, tris), sb.add_material(color=(1.0, 1.0, 1.0), ior=1.0))
    lamp = np.array([[-0.1, 1.9, -0.1], [0.1, 1.9, -0.1], [0.1, 1.9, 0.1], [-0.1, 1.9, 0.1]], np.float32)
    sb.add_instance(sb.add_mesh(lamp, [[0, 1, 2], [0, 2, 3]]),
                    sb.add_material(emission_color=(1.0, 0.9, 0.8), emission_strength=20.0))
    sb.set_env(np.ones((8, 16, 4), np.float32))
    sb.camera = look_at_camera(width, height, (0.3, -0.2, 1.5), (0, 0, 0), 70.0)
    return sb


@pytest.mark.parametrize("layout", [_ffi.BVH_SINGLE_LEVEL, _ffi.BVH_TWO_LEVEL], ids=["single", "two"])
@pytest.mark.parametrize("nee", list(NEE))
@pytest.mark.parametrize("width,height", [(20, 15), (400, 250)])
def test_wave_beside_a_finished_one(width, height, nee, layout):
    scene = room(width, height)
    opt = dict(bvh_layout=layout, **NEE[nee])
    first = (1, 2, 9)
    r = lx.Renderer(scene, default_options(trace_depth=DEPTH, **opt))
    want, rays = [], 0
    for it in first:
        r.reset()
        r.render(it, 1)
        want.append(r.image_sum())
        st = r.stats()
        rays += st["rays_radiance"] + st["rays_shadow"]
        if width * height > LANES:
            assert LANES < r.wave_counts(DEPTH)[0][3] < 2 * LANES
    r.close()

    E = lx.Engine([scene], default_options(**opt), max_paths=width * height)
    ids = []
    for it in first:
        ids.append(E.submit(0, 1, trace_depth=DEPTH, first_iter=it))
        E.step()
        E.step()
    E.run()
    total = E.stats()["rays"]
    got = [E.image(i) for i in ids]
    E.close()
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert total == rays
