"""Primitives of many pixels: at the edges of what a lane, a warp and a part of
a primitive draws, many of them in one warp, mixed with small and culled ones,
and pictures that most of them fill. Every pixel equals the sequential CPU
restatement's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dust,sizes", [(3, [64.0]), (61, [8.0, 8.9, 9.1]), (200, [60.0, 63.9, 64.1, 66.0]),
                                        (40, [0.5, 30.0, 64.0, 65.0, 500.0]), (300, [400.0])])
@pytest.mark.parametrize("width,height", [(331, 203), (64, 65)])
def test_large_primitives_bit_exact(native, oracle, dust, sizes, width, height):
    from astro_gb300 import ic
    from astro_gb300.render import reference_camera

    L = native.layouts
    pm, vr, ct = ic.reference_scene(2, 3, dust, seed=dust)
    rng = np.random.default_rng(dust)
    vr["radius"][5:] = rng.choice(sizes, dust)
    vr["radius"][:5] = [1.0, 2e4, 3e5, 9e5, 5e6]
    cam = reference_camera(width, height, position=(5e4, -5e4, 1.4e6))
    with native.Simulation(native.default_params(L.PRESET_REFERENCE), max_n=len(pm) + 7) as sim:
        sim.upload(pm, vr, ct, n_tree=5)
        sim.lighting_pass(2)
        lit = sim.read_colors()
        for _ in range(2):  # the first picture outgrows the fragment buffer
            rgba, depth = sim.splat(cam, width, height)
            want_rgba, want_depth = oracle.splat(pm, vr, lit, cam, width, height)
            assert np.array_equal(depth, want_depth) and np.array_equal(rgba, want_rgba)
