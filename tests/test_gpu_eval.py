"""The group evaluation where its shape changes: groups at the edges of the
particles a lane holds and of the parts the lists are split into, lists at
the edges of a staged block, and softening lengths on both sides of the
packed form's bound. Compared with the CPU restatement at the fast form's
tolerance (|da| <= 2e-5 |a| + 1e-6 of the median); counts must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


def _check(ag, oracle, p, pm, vr):
    from test_gpu_parity import acc_close, run_gpu

    out = run_gpu(ag, p, pm, vr, dt=1e-3, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=1)
    ok, rel = acc_close(out["acc4"], ref["acc4"])
    assert ok.all(), f"{(~ok).sum()} particles outside tolerance, worst {rel.max():.3e}"
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]


@pytest.mark.parametrize("group_size", [1, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("form", [0, 1])
def test_group_size_edges(ag, oracle, group_size, form):
    from astro_gb300 import ic

    L = ag.layouts
    flags = L.FLAG_OPEN_DELTA | (L.FLAG_QUADRUPOLE if group_size % 2 == 0 else 0)
    p = ag.default_params(L.PRESET_PHYSICAL, lbits=9, form=form, group_size=group_size,
                          far_ratio=0.25 if group_size % 8 else 0.0, bucket=8, softening=0.005,
                          flags=flags)
    pm, vr = ic.disk_bulge(12000, seed=31 + group_size)
    _check(ag, oracle, p, pm, vr)


@pytest.mark.parametrize("n,lbits", [(1, 3), (2, 1), (33, 1), (64, 1), (127, 1), (129, 1), (5000, 2),
                                     (9001, 3)])
@pytest.mark.parametrize("form", [0, 1])
def test_list_edges(ag, oracle, n, lbits, form):
    """Few, large leaves: one range longer than a staged tile, tiles that end
    inside a range, chunks of every size left over."""
    from astro_gb300 import ic

    L = ag.layouts
    p = ag.default_params(L.PRESET_PHYSICAL, lbits=lbits, form=form, group_size=64, far_ratio=0.5,
                          bucket=0, softening=0.01, open_delta_weight=0.5)
    pm, vr = ic.uniform_cube(n, seed=n)
    _check(ag, oracle, p, pm, vr)


@pytest.mark.parametrize("eps", [0.0, 1e-15, 9.0e-13, 9.2e-13])
def test_small_softening(ag, oracle, eps):
    """eps^2 below 2^-80 takes the general loops, which skip a particle's own
    entry; just above it the packed loops add exactly zero for it."""
    from astro_gb300 import ic

    L = ag.layouts
    p = ag.default_params(L.PRESET_PHYSICAL, lbits=7, group_size=40, softening=eps, far_ratio=0.2)
    pm, vr = ic.plummer(3000, seed=8)
    _check(ag, oracle, p, pm, vr)


@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("far", [0.0, 0.3])
@pytest.mark.parametrize("n,lbits,theta", [(1, 4, 0.7), (40, 2, 0.7), (6000, 10, 0.7), (3000, 5, 0.2)])
def test_walk_variants_bit_exact(ag, oracle, delta, far, n, lbits, theta):
    """The walk's four variants, with frontiers below and above the 32 runs
    that stay on chip and lists that end inside and at a block: counts and
    (in the exact form, which sums in list order) accelerations are equal."""
    from astro_gb300 import ic
    from test_gpu_parity import run_gpu

    L = ag.layouts
    flags = L.FLAG_IEEE_EXACT | L.FLAG_QUADRUPOLE | (L.FLAG_OPEN_DELTA if delta else 0)
    p = ag.default_params(L.PRESET_PHYSICAL, lbits=lbits, theta=theta, far_ratio=far, flags=flags,
                          bucket=4, group_size=24)
    pm, vr = ic.plummer(n, seed=77)
    out = run_gpu(ag, p, pm, vr, dt=1e-3, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=1)
    assert np.array_equal(out["acc4"], ref["acc4"])
    assert out["interactions"] == ref["interactions"] and out["node_visits"] == ref["node_visits"]
