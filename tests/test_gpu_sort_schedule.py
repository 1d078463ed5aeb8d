"""Large sorts whose passes the device schedules: digits that all keys share are
left out, the top digits alone are sorted and the rest ordered among neighbours,
and all digits are sorted where a run of equal top digits is too long for that.
Every case equals a stable sort."""
import pytest

pytestmark = pytest.mark.gpu

N = 2 * 1024 * 1024 + 12345


def _keys(torch, kind, n, gen):
    k = torch.randint(0, (1 << 63) - 1, (n,), device="cuda", generator=gen, dtype=torch.int64)
    if kind.startswith("run"):  # equal top digits, the rest counting down
        length = int(kind[3:])
        at = torch.randperm(n, device="cuda", generator=gen)[:length]
        k[at] = (0x2345678912345678 & ~0xFFFFFF) + torch.arange(length, 0, -1, device="cuda")
    elif kind == "short":  # many short runs, some of equal keys
        k = (k >> 43 << 43) + (k & 3)
    elif kind == "equal":
        k.fill_(0x123456789ABCDEF)
    elif kind == "low36":
        k &= (1 << 36) - 1
    elif kind == "high":
        k &= ~0xFFFFFFFF
    elif kind == "clusters":
        k = (k & 0x0003000000FFFFFF) | 0x1234000000000000
    elif kind == "sorted":
        k = torch.sort(k).values
    elif kind == "extremes":
        k[: n // 2] |= 0x7FFFFF0000000000
        k[0], k[n - 1] = 0, (1 << 63) - 1
    return k


@pytest.mark.parametrize("kind", ["uniform", "run127", "run128", "run129", "run130", "run5000", "short", "equal",
                                  "low36", "high", "clusters", "sorted", "extremes"])
@pytest.mark.parametrize("key_bits,device_count", [(63, False), (64, True)])
def test_schedules_match_stable_sort(native, kind, key_bits, device_count):
    import torch

    from astro_gb300.radix_sort import RadixSort

    gen = torch.Generator(device="cuda").manual_seed(7)
    n, room = N, N + (777 if device_count else 0)
    keys = _keys(torch, kind, room, gen)
    before = keys.clone()
    index = torch.arange(room, device="cuda", dtype=torch.int32)
    keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
    count = torch.tensor([n], device="cuda", dtype=torch.int32) if device_count else None
    sorter = RadixSort(room, key_bits)
    for _ in range(2):  # the scratch is left as the first sort left it
        keys_out.fill_(-1)
        sorter.sort(keys, index, keys_out, index_out, room, count)
        torch.cuda.synchronize()
        want, order = torch.sort(keys[:n], stable=True)
        assert torch.equal(keys_out[:n], want)
        assert torch.equal(index_out[:n].long(), order)
        assert bool((keys_out[n:] == -1).all())
    assert torch.equal(keys, before)
