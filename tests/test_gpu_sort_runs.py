"""Large sorts by the top digits where many keys share them: runs at the edges
of what is ordered among neighbours, of what a block sorts and of a warp's part,
runs at both ends of the array, many runs, and equal keys in them. Equal to a
stable sort; the schedule in the sorter's scratch says which way was taken
(counter word 10: from bit 8 the top digits sorted by; word 14: 1 long runs, 2
all digits after all; word 15: the long runs listed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2 * 1024 * 1024 + 1234


def _sampled(n):
    """Places that the sort looks at to judge the keys (4,096 of them)."""
    h = (np.arange(1, 4097, dtype=np.uint64) * 0x9E3779B1) & 0xFFFFFFFF
    h = ((h ^ (h >> 15)) * 0x85EBCA77) & 0xFFFFFFFF
    return ((h ^ (h >> 13)) * n) >> 32


def _keys(torch, key_bits, lengths, seed, prefix=None, low_values=None):
    """Uniform keys, and runs of keys that share the top digits at places that
    are not sampled; what is below the digits repeats within low_values."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(top, *shape):
        return torch.randint(0, top, shape, device="cuda", generator=gen, dtype=torch.int64)

    keys = rand((1 << min(key_bits, 63)) - 1, N)
    shift = 8 * ((key_bits + 7) // 8 - 3)
    free = torch.ones(N, dtype=torch.bool, device="cuda")
    free[torch.from_numpy(_sampled(N).astype(np.int64)).cuda()] = False
    places = torch.nonzero(free).flatten()
    places = places[torch.randperm(len(places), device="cuda", generator=gen)]
    taken = 0
    for k, length in enumerate(lengths):
        at = places[taken: taken + length]
        taken += length
        high = (prefix if prefix is not None else 0x10000 + 517 * k) << shift
        # Nobody else has this prefix.
        keys = torch.where(keys >> shift == high >> shift, keys ^ (1 << shift), keys)
        keys[at] = high + rand(low_values or (1 << shift) - 1, length)
    return keys


def _check(torch, keys, key_bits, flags, listed):
    from astro_gb300.radix_sort import RadixSort

    index = torch.arange(N, device="cuda", dtype=torch.int32)
    keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
    sorter = RadixSort(N, key_bits)
    for _ in range(2):  # the scratch is left as the first sort left it
        keys_out.fill_(-1)
        sorter.sort(keys, index, keys_out, index_out, N)
        want, order = torch.sort(keys, stable=True)
        assert torch.equal(keys_out, want)
        assert torch.equal(index_out.long(), order)
    words = sorter.temp[: 4 * 16].view(torch.int32).tolist()
    assert words[10] >> 8 == 3 and words[14] == flags
    if flags == 1:
        assert words[15] == listed


@pytest.mark.parametrize("length", [128, 129, 255, 256, 257, 1023, 1024, 1025, 2048, 2049, 5000, 32767, 32768, 32769,
                                    50000])
@pytest.mark.parametrize("key_bits", [48, 63, 64])
def test_run_lengths(native, length, key_bits):
    import torch

    keys = _keys(torch, key_bits, [length], seed=length)
    _check(torch, keys, key_bits, 0 if length <= 128 else (1 if length <= 32768 else 2), 1)


@pytest.mark.parametrize("prefix", [0, (1 << 24) - 2])
@pytest.mark.parametrize("length", [129, 4000])
def test_runs_at_the_ends(native, prefix, length):
    import torch

    _check(torch, _keys(torch, 48, [length], 5, prefix=prefix), 48, 1, 1)


def test_many_runs_with_equal_keys(native):
    import torch

    lengths = [100 + 3 * k for k in range(700)]
    keys = _keys(torch, 56, lengths, 11, low_values=7)
    _check(torch, keys, 56, 1, sum(n > 128 for n in lengths))


def test_two_long_runs_one_too_long(native):
    import torch

    _check(torch, _keys(torch, 48, [700, 40000, 900], 12), 48, 1 | 2, None)
