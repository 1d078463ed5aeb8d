"""The last layers of the tree, which one block of the cluster makes alone while
the others write the groups: trees whose layers hold just under and just over
that block's nodes, chains above one node, and many systems at the root layer.
Records, groups (through the interaction counts) and accelerations equal the CPU
restatement's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lbits,nsys", [(2, 21, 1), (65, 2, 1), (513, 3, 1), (900, 2, 1), (4000, 4, 1), (33000, 5, 1),
                                          (600, 4, 63), (600, 4, 64), (600, 4, 65), (3000, 5, 300)])
@pytest.mark.parametrize("form", [0, 1])
def test_last_layers_bit_exact(native, oracle, n, lbits, nsys, form):
    from astro_gb300 import ic
    from test_gpu_parity import assert_tree_equal, run_gpu

    L = native.layouts
    sizes = [n // nsys + (1 if k < n % nsys else 0) for k in range(nsys)]
    parts = [ic.uniform_cube(s, seed=5 + k) for k, s in enumerate(sizes)]
    pm = np.concatenate([a for a, _ in parts])
    vr = np.concatenate([b for _, b in parts])
    p = native.default_params(L.PRESET_PHYSICAL, lbits=lbits, form=form, bucket=4, group_size=8,
                              flags=L.FLAG_IEEE_EXACT | L.FLAG_OPEN_DELTA | L.FLAG_QUADRUPOLE)
    out = run_gpu(native, p, pm, vr, dt=1e-3, steps=3, sizes=sizes)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=3, sizes=sizes)
    assert_tree_equal(out, ref)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]
