"""The group walk where every buffer of a warp runs over window after window: far
nodes, cells, leaf ranges and the next frontier, with every number of items left
behind the block that is written. Lists and counts equal the CPU restatement's
(exact form: the accelerations bit by bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plummer", "cube"])
@pytest.mark.parametrize("theta,far,bucket,group_size", [(0.25, 0.15, 1, 8), (0.3, 0.3, 2, 32), (0.25, 0.0, 1, 64)])
def test_overflowing_buffers_bit_exact(native, oracle, kind, theta, far, bucket, group_size):
    from astro_gb300 import ic
    from test_gpu_parity import run_gpu

    L = native.layouts
    p = native.default_params(L.PRESET_PHYSICAL, lbits=8, theta=theta, far_ratio=far, bucket=bucket,
                              group_size=group_size, flags=L.FLAG_IEEE_EXACT | L.FLAG_QUADRUPOLE | L.FLAG_OPEN_DELTA)
    pm, vr = ic.plummer(6000, seed=13) if kind == "plummer" else ic.uniform_cube(6000, seed=13)
    out = run_gpu(native, p, pm, vr, dt=1e-3, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=1)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]
    # Many blocks of each list a walk: a particle meets that many sources.
    assert out["interactions"] > 500 * len(pm)
