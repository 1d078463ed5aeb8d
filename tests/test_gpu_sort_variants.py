"""Every sort_variant a context accepts, at a count that the pass kernels sort
(fewer pairs are sorted in one launch, whatever the variant): equal to a stable
sort of the codes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", range(13))
def test_variants_match_stable_argsort(native, variant):
    from astro_gb300 import ic

    L = native.layouts
    pm, vr = ic.plummer(100003, seed=5)
    with native.Simulation(native.default_params(L.PRESET_PHYSICAL, lbits=11, sort_variant=variant),
                           max_n=len(pm)) as sim:
        sim.upload(pm, vr)
        sim.generate_morton_codes()
        sim.sort()
        codes, sorted_codes, index = sim.read_keys()
    order = np.argsort(codes, kind="stable")
    assert np.array_equal(sorted_codes, codes[order])
    assert np.array_equal(index, order.astype(np.uint32))
