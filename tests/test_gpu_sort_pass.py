"""The radix sort's pass kernels at the sizes where the default changes its tile
and at tile edges, more tiles than resident blocks, and a count that is known
on the device only: equal to a stable sort."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65537, 69632, 69633, 524287, 524288, 528385, 1300001, 8388607, 8388608, 8391681])
@pytest.mark.parametrize("bits", [63, 13])
def test_default_pass_matches_stable_sort(native, n, bits):
    import torch

    from astro_gb300.radix_sort import RadixSort

    gen = torch.Generator(device="cuda").manual_seed(n)
    room = n + 5000
    keys = torch.randint(0, (1 << bits) - 1, (room,), device="cuda", generator=gen, dtype=torch.int64)
    index = torch.arange(room, device="cuda", dtype=torch.int32)
    keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
    count = torch.tensor([n], device="cuda", dtype=torch.int32)
    sorter = RadixSort(room, bits)
    sorter.sort(keys, index, keys_out, index_out, room, count)
    torch.cuda.synchronize()
    want, order = torch.sort(keys[:n], stable=True)
    assert torch.equal(keys_out[:n], want)
    assert torch.equal(index_out[:n].long(), order)
    assert bool((keys_out[n:] == -1).all()) and bool((index_out[n:] == -1).all())
