"""The layer pass at the edges of its tiles (512, 1,024 or 2,048 keys, by the
count), and the counters that the sort (PHYSICAL) or the encode (REFERENCE)
zeroes for the build and the traversal behind it: stage calls that repeat a
build, drop a sort or mix with whole steps. Trees, accelerations and states are
equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


@pytest.mark.parametrize("n", [2, 511, 512, 513, 131071, 131072, 131073, 1048575, 1048576, 1048577])
def test_tile_edges_bit_exact(ag, oracle, n):
    from astro_gb300 import ic
    from test_gpu_parity import assert_tree_equal, run_gpu

    L = ag.layouts
    p = ag.default_params(L.PRESET_PHYSICAL, lbits=13 if n % 2 else 9,
                          flags=L.FLAG_IEEE_EXACT | L.FLAG_OPEN_DELTA, bucket=8)
    pm, vr = ic.uniform_cube(n, seed=n)
    out = run_gpu(ag, p, pm, vr, dt=1e-3, steps=2)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=2)
    assert_tree_equal(out, ref)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]


@pytest.mark.parametrize("preset,n", [("phys", 20000), ("phys", 140000), ("ref", 3000)])
@pytest.mark.parametrize("no_graph", [False, True])
def test_stage_calls_between_steps(ag, preset, n, no_graph):
    from astro_gb300 import ic

    L = ag.layouts
    p = ag.default_params(L.PRESET_PHYSICAL if preset == "phys" else L.PRESET_REFERENCE)
    if no_graph:
        p.flags |= L.FLAG_NO_GRAPH
    pm, vr = ic.disk_bulge(n, seed=3)

    def stages(sim, builds=1):
        sim.generate_morton_codes()
        sim.sort()
        for _ in range(builds):
            sim.build_tree()
        sim.barnes_hut()
        stats = sim.read_stats(), sim.read_far_stats()
        sim.update_spheres(1e-3)
        return stats

    with ag.Simulation(p, max_n=200000) as sim:
        sim.upload(pm, vr)
        sim.draw(1e-3, 1)
        first = sim.read_stats(), sim.read_far_stats()
        sim.draw(1e-3, 4)
        want = sim.download()
        last = sim.read_stats(), sim.read_far_stats()
    with ag.Simulation(p, max_n=200000) as sim:
        sim.upload(*ic.plummer(150001, seed=1))
        sim.draw(1e-3, 2)
        sim.generate_morton_codes()
        sim.sort()  # left by the next upload, which has another layout
        sim.upload(pm, vr)
        assert stages(sim) == first
        sim.draw(1e-3, 1)
        stages(sim, builds=3)
        sim.draw(1e-3, 1)
        assert stages(sim, builds=2) == last
        got = sim.download()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        sim.generate_morton_codes()
        sim.sort()  # left by the next upload, which has the same layout
        sim.upload(pm, vr)
        sim.draw(1e-3, 5)
        got = sim.download()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
