"""The native autotuner tries a knob where its values run different kernels:
no walk_frontier, block_warps with the per-particle walk only, sort variants
above the one-launch sort and each shape once."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,per_particle", [(3000, False), (3000, True), (70000, False)])
def test_trials_differ_in_what_runs(native, n, per_particle):
    from astro_gb300 import ic

    L = native.layouts
    pm, vr = ic.plummer(n, seed=4)
    flags = L.FLAG_OPEN_DELTA | (L.FLAG_PER_PARTICLE if per_particle else L.FLAG_QUADRUPOLE)
    p = native.default_params(L.PRESET_PHYSICAL, lbits=8, softening=0.01, flags=flags)
    with native.Simulation(p, max_n=n) as sim:
        sim.upload(pm, vr)
        res = sim.autotune(samples=64, keep=L.TUNE_KEEP_LBITS | L.TUNE_KEEP_GROUP_SIZE | L.TUNE_KEEP_ACCURACY)
    tried = {k: {t["knobs"][k] for t in res["trials"]} for k in ("walk_frontier", "block_warps", "sort_variant")}
    assert tried["walk_frontier"] == {0}
    assert tried["block_warps"] == ({4, 8} if per_particle else {4})
    assert tried["sort_variant"] == ({0} if n <= 65536 else set(range(8)))
