"""Sorts of one block: radix passes in shared memory at the edges of their
items, threads and passes, and the bitonic network beside them; equal to a
stable sort, with the values given or the places, the count on the host or the
device."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 256, 257, 1000, 1023, 1024, 1025, 2047, 2048, 2049, 2051, 4095, 4096])
@pytest.mark.parametrize("bits", [1, 8, 9, 40, 41, 64])
def test_block_sorts_match_stable_sort(native, n, bits):
    import torch

    from astro_gb300.radix_sort import RadixSort

    gen = torch.Generator(device="cuda").manual_seed(64 * n + bits)
    keys = torch.randint(0, (1 << min(bits, 63)) - 1 + (bits < 2), (4096,), device="cuda", generator=gen,
                         dtype=torch.int64)
    index = torch.randint(0, 1 << 31, (4096,), device="cuda", generator=gen).int()
    for room, count in ((n, None), (min(4096, n + 37), torch.tensor([n], device="cuda", dtype=torch.int32))):
        keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
        RadixSort(4096, bits).sort(keys, index, keys_out, index_out, room, count)
        torch.cuda.synchronize()
        want, order = torch.sort(keys[:n], stable=True)
        assert torch.equal(keys_out[:n], want)
        assert torch.equal(index_out[:n], index[order])
        assert bool((keys_out[n:] == -1).all()) and bool((index_out[n:] == -1).all())
