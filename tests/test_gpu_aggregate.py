"""The bottom-up aggregation where its paths meet: layers with and without
work lists, single-child chains that cross from one to the other and into the
climbing launch, one leaf or one system only, and layouts that change under a
context (the work lists and arrival counts share storage). Node records,
groups (through the interaction counts) and accelerations equal the CPU
restatement's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


def _params(ag, form, lbits, quad=True, group_size=24):
    L = ag.layouts
    flags = L.FLAG_IEEE_EXACT | L.FLAG_OPEN_DELTA | (L.FLAG_QUADRUPOLE if quad else 0)
    return ag.default_params(L.PRESET_PHYSICAL, lbits=lbits, form=form, flags=flags, bucket=8,
                             group_size=group_size)


@pytest.mark.parametrize("n,lbits,quad", [(1, 1, True), (3, 21, True), (32767, 9, False), (32769, 9, True),
                                          (70001, 21, True), (1048577, 11, True), (1100003, 8, False)])
@pytest.mark.parametrize("form", [0, 1])
def test_paths_bit_exact(ag, oracle, n, lbits, quad, form):
    from astro_gb300 import ic
    from test_gpu_parity import assert_tree_equal, run_gpu

    p = _params(ag, form, lbits, quad)
    pm, vr = ic.uniform_cube(n, seed=n) if n % 2 else ic.plummer(n, seed=n)
    out = run_gpu(ag, p, pm, vr, dt=1e-3, steps=2)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=2)
    assert_tree_equal(out, ref)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]


@pytest.mark.parametrize("form", [0, 1])
def test_layouts_change_under_a_context(ag, oracle, form):
    from astro_gb300 import ic

    p = _params(ag, form, 12)
    with ag.Simulation(p, max_n=1100000, max_systems=4) as sim:
        for n in (1100000, 40000, 1, 1099999, 33000):
            pm, vr = ic.disk_bulge(n, seed=n) if n > 1 else ic.plummer(1, seed=1)
            sim.upload(pm, vr)
            sim.draw(1e-3, 2)
            got, _ = sim.download()
            acc = sim.read_accel()
            if n > 100000:
                continue
            pm_o, vr_o = pm.copy(), vr.copy()
            ref = oracle.phys_run(p, pm_o, vr_o, dt=1e-3, steps=2)
            assert np.array_equal(acc, ref["acc4"])
            assert np.array_equal(got["position"], pm_o["position"])
