"""The REFERENCE walk's two kernels: trees that fit the shared layout and
trees that do not, depths on both sides of the tables that step over layers
every particle opens, accepted nodes near and far, and particles of every
type in the tree. Forces, counts and the moved state equal the CPU
restatement's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


def _counts(p, nodes, root, pm, codes, types, n_tree):
    """(interactions, visits) of the reference's walk over all particles, node
    by node with the particles that reach it (FP32, the reference's order)."""
    f = np.float32
    pos, n = pm["position"], len(pm)
    own = np.full(n, 0xFFFFFFFFFFFFFFFF, np.uint64)
    own[:n_tree] = np.where(types[:n_tree] != 2, codes, own[:n_tree])
    inter = visits = 0
    stack = [(root, np.ones(n, bool))]
    while stack:
        k, mask = stack.pop()
        nd = nodes[k]
        visits += int(mask.sum())
        d = nd["centerOfMass"] - pos
        d2 = ((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) + f(p.softening)
        d2 = np.maximum(d2, f(1e-6))
        dist = np.maximum(np.sqrt(d2), f(1e-6))
        if nd["layer"] == 0:
            inter += int((mask & (own != nd["mortonCode"]) & (d2 > f(p.leaf_min_dist2))).sum())
            continue
        far = f(2.0 ** (21 + int(nd["layer"]))) / dist < f(p.theta)
        inter += int((mask & far).sum())
        below = mask & ~far
        if below.any():
            stack += [(int(c), below) for c in nd["children"] if c != 0xFFFFFFFF]
    return inter, visits


@pytest.mark.parametrize("stars,planets,dust", [(1, 0, 0), (1, 1, 31), (5, 200, 3000), (3, 60, 1025),
                                                (5, 330, 511), (5, 900, 700)])
@pytest.mark.parametrize("lbits,theta,spread", [(6, 0.7, 1.0), (6, 0.7, 40.0), (1, 0.5, 1.0), (9, 0.3, 15.0),
                                                (12, 1.5, 100.0)])
def test_small_and_large_trees_bit_exact(ag, oracle, stars, planets, dust, lbits, theta, spread):
    from astro_gb300 import ic

    L = ag.layouts
    n_tree = stars + planets
    pm, vr, ct = ic.reference_scene(stars, planets, dust, seed=stars + planets + dust)
    # Spread past the range of the quantiser and the nodes' nominal sizes, so
    # that nodes of several layers are accepted.
    pm["position"] *= np.float32(spread)
    if n_tree > 3:
        pm["position"][2] = pm["position"][1]  # two bodies in one leaf
        ct["type"][3] = 2                      # dust inside the tree
    p = ag.default_params(L.PRESET_REFERENCE, lbits=lbits, theta=theta)
    with ag.Simulation(p, max_n=len(pm)) as sim:
        sim.upload(pm, vr, ct, n_tree=n_tree)
        sim.draw(1.0 / 60.0, 1)
        acc = sim.read_accel()
        stats = sim.read_stats()
        codes, _, _ = sim.read_keys()
        nodes = sim.read_nodes()
        root = int(sim.tree_info()[1][-1])
        got, gotv = sim.download()
    pm_o, vr_o = pm.copy(), vr.copy()
    ref = oracle.ref_run(p, pm_o, vr_o, ct, n_tree=n_tree, dt=1.0 / 60.0, steps=1, split_passes=64)
    assert np.array_equal(acc, ref["acc4"])
    assert stats == _counts(p, nodes, root, pm, codes, ct["type"], n_tree)
    assert np.array_equal(got["position"], pm_o["position"])
    assert np.array_equal(gotv["velocity"], vr_o["velocity"])
