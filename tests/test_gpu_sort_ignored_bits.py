"""Large sorts of keys that hold something above key_bits: those bits take no
part, whichever way the passes are scheduled, and come out with their keys.
Equal to a stable sort of the low bits. The schedule in the sorter's scratch
says which way was taken (counter word 10: the number of digits, and from bit 8
the top digits sorted by; word 14: the ordering of neighbours gave up)."""
import pytest

pytestmark = pytest.mark.gpu

N = 2 * 1024 * 1024 + 77


def _sorted_as(torch, keys, key_bits, top, gave_up):
    from astro_gb300.radix_sort import RadixSort

    n = keys.numel()
    index = torch.arange(n, device="cuda", dtype=torch.int32)
    keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
    sorter = RadixSort(n, key_bits)
    sorter.sort(keys, index, keys_out, index_out, n)
    low = keys if key_bits == 64 else keys & ((1 << key_bits) - 1)
    order = torch.sort(low, stable=True).indices
    assert torch.equal(index_out.long(), order)
    assert torch.equal(keys_out, keys[order])
    words = sorter.temp[: 4 * 16].view(torch.int32).tolist()
    assert words[10] >> 8 == top and bool(words[14]) == gave_up


# 40 bits have too few digits for the top ones alone, 41 too few bits in them.
@pytest.mark.parametrize("key_bits,top", [(40, 0), (41, 0), (48, 3), (56, 3), (63, 3)])
def test_bits_above_key_bits_take_no_part(native, key_bits, top):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(key_bits)
    keys = torch.randint(-(1 << 63), (1 << 63) - 1, (N,), device="cuda", generator=gen, dtype=torch.int64)
    _sorted_as(torch, keys, key_bits, top, False)


@pytest.mark.parametrize("length,gave_up", [(120, False), (5000, True)])
def test_runs_under_other_high_bits(native, length, gave_up):
    """Keys that agree in the sorted digits and differ above key_bits are one
    run: ordered among neighbours where it is short, by all digits where not."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(length)
    keys = torch.randint(-(1 << 63), (1 << 63) - 1, (N,), device="cuda", generator=gen, dtype=torch.int64)
    at = torch.randperm(N, device="cuda", generator=gen)[:length]
    keys[at] = (keys[at] >> 48 << 48) + 0x123456000000 + torch.arange(length, 0, -1, device="cuda")
    _sorted_as(torch, keys, 48, 3, gave_up)


def test_repeats_under_other_high_bits_do_not_qualify(native):
    """Few distinct low parts: the top digits do not tell the keys apart, whatever
    lies above."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(3)
    keys = torch.randint(-(1 << 63), (1 << 63) - 1, (N,), device="cuda", generator=gen, dtype=torch.int64)
    few = torch.randint(0, 1 << 48, (3000,), device="cuda", generator=gen, dtype=torch.int64)
    pick = torch.randint(0, 3000, (N,), device="cuda", generator=gen)
    _sorted_as(torch, (keys >> 48 << 48) + few[pick], 48, 0, False)
