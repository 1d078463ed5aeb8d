"""As many systems as make the top layer a launch of its own, and just fewer:
systems of one particle, no larger than a group, and larger. Records, groups (through the interaction
counts) and accelerations equal the CPU restatement's bit for bit; so do deep
trees whose layers lie around that size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(native, oracle, pm, vr, sizes, lbits, form, steps=2):
    from test_gpu_parity import assert_tree_equal, run_gpu

    L = native.layouts
    p = native.default_params(L.PRESET_PHYSICAL, lbits=lbits, form=form, bucket=2, group_size=8,
                              flags=L.FLAG_IEEE_EXACT | L.FLAG_OPEN_DELTA | L.FLAG_QUADRUPOLE)
    out = run_gpu(native, p, pm, vr, dt=1e-3, steps=steps, sizes=sizes)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=steps, sizes=sizes)
    assert_tree_equal(out, ref)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]


@pytest.mark.parametrize("nsys,most,lbits", [(18431, 12, 3), (18432, 12, 3), (24576, 1, 1), (33000, 20, 2),
                                             (65536, 3, 5)])
@pytest.mark.parametrize("form", [0, 1])
def test_top_layer_of_many_systems(native, oracle, nsys, most, lbits, form):
    from astro_gb300 import ic

    sizes = [1 + k * 7919 % most for k in range(nsys)]
    pm, vr = ic.uniform_cube(sum(sizes), seed=nsys)
    _run(native, oracle, pm, vr, sizes, lbits, form)


@pytest.mark.parametrize("n,lbits", [(18431, 21), (18432, 21), (24577, 9), (30001, 14), (32767, 21)])
@pytest.mark.parametrize("form", [0, 1])
def test_deep_trees_around_the_line(native, oracle, n, lbits, form):
    from astro_gb300 import ic

    pm, vr = ic.uniform_cube(n, seed=n)
    _run(native, oracle, pm, vr, None, lbits, form)
