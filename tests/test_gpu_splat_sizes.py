"""Primitives around the size where the splat's emission goes from one lane to
the whole warp, mixed in one warp, partly off-screen and culled, and particle
counts at the edges of the fragment keys' index bits. Every pixel equals the
sequential CPU restatement's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


@pytest.mark.parametrize("dust", [0, 1, 27, 51, 1019, 1020, 4000])
@pytest.mark.parametrize("width,height", [(1, 1), (97, 61)])
def test_sizes_bit_exact(ag, oracle, dust, width, height):
    from astro_gb300 import ic
    from astro_gb300.render import reference_camera

    L = ag.layouts
    pm, vr, ct = ic.reference_scene(2, 3, dust, seed=dust + 3)
    rng = np.random.default_rng(dust)
    # Points of 0.4 to 14 pixels: boxes of 1 to over 200 cells, on both sides of 64.
    vr["radius"][5:] = rng.choice([0.4, 2.0, 5.9, 6.0, 6.1, 7.0, 7.9, 8.0, 14.0], dust)
    vr["radius"][2:5] = [1.0, 2e4, 3e5]
    cam = reference_camera(width, height, position=(1e5, -5e4, 1.2e6))
    with ag.Simulation(ag.default_params(L.PRESET_REFERENCE), max_n=len(pm)) as sim:
        sim.upload(pm, vr, ct, n_tree=5)
        sim.lighting_pass(2)
        lit = sim.read_colors()
        rgba, depth = sim.splat(cam, width, height)
    want_rgba, want_depth = oracle.splat(pm, vr, lit, cam, width, height)
    assert np.array_equal(depth, want_depth) and np.array_equal(rgba, want_rgba)
